"""A geometry that mcl_set_geometry refuses leaves the engine as it was: the sweeps that follow take the decisions of
the geometry in force (the simple schedule's kernel, which reads the device's point types), on every replica."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu

DIMS = (20, 14, 12)
SURF = [("homeotropic", 1.5, 0, 0), ("rp", 0.5, 40, 10)]


def geometry(seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(DIMS))
    pt = rng.choice([0, 1, 2, 3], size=n, p=[0.3, 0.5, 0.1, 0.1]).astype(np.int32)
    nrm = rng.normal(size=(n, 3))
    return pt, (nrm / np.linalg.norm(nrm, axis=1)[:, None]).astype(np.float32)


def refused(seed):
    pt, nrm = geometry(seed)
    bad = pt.copy()
    bad[-3] = 9  # past almost every site
    yield bad, nrm
    yield np.zeros_like(pt), nrm  # no site left


def run(schedule, steps):
    e = M.Engine(M.Model("ll", surfaces=SURF),
                 [M.Replica(*DIMS, "custom", (1, 0, 1), T=0.6, seed=5 + r) for r in range(2)], schedule)
    steps(e)
    for r in range(2):
        e.random_directors(r, 3 + r)
    e.sweeps(2)
    e.sweeps(2, measure=True)
    out = [(e.download(r), e.series(r), e.measure(r)) for r in range(2)]
    e.close()
    return out


def valid_then_refused(e):
    for r in range(2):
        e.set_geometry(r, *geometry(1 + r))
    e.sweeps(1)
    for g in refused(8):
        with pytest.raises(M.McLicsError):
            e.set_geometry(0, *g)
    e.set_geometry(1, *geometry(4))  # what is swept is listed again


def refused_then_valid(e):
    for g in refused(9):
        with pytest.raises(M.McLicsError):
            e.set_geometry(0, *g)
    e.set_geometry(1, *geometry(2))
    e.set_geometry(0, *geometry(6))
    with pytest.raises(M.McLicsError):
        e.set_geometry(0, *next(refused(7)))


@pytest.mark.parametrize("steps", [valid_then_refused, refused_then_valid])
def test_a_refused_geometry_changes_nothing(steps):
    for a, b in zip(run(M.SCHED_CHECKER2, steps), run(M.SCHED_CHECKER2_SIMPLE, steps)):
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[1]["acceptance"], b[1]["acceptance"])
        assert a[2]["n_valid"] == b[2]["n_valid"]
        np.testing.assert_allclose(a[1]["energy"], b[1]["energy"], rtol=2e-6, atol=2e-6)


def test_directors_are_still_checked_against_the_geometry_in_force():
    """Upload skips empty sites only: a refused geometry must not mark sites as empty."""
    e = M.Engine(M.Model("ll", surfaces=SURF), [M.Replica(*DIMS, "custom", (0, 0, 0), T=0.6)])
    pt, nrm = geometry(1)
    pt[:] = 1
    e.set_geometry(0, pt, nrm)
    bad = np.zeros_like(pt)
    with pytest.raises(M.McLicsError):
        e.set_geometry(0, bad, nrm)
    with pytest.raises(M.McLicsError):
        e.upload(0, np.zeros(3 * pt.size, np.float32))
    e.close()
