"""The sweep over site lists of sphere and custom lattices against the kernel with one thread per cell of the box
(the simple schedule): the same decisions bit for bit, observables within the grouping of the bond sums. Empty sites
inside and at the edges, isolated sites, several surfaces, periodic and free axes, odd extents, several replicas, a
geometry set again between sweeps."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu

SURF = [("homeotropic", 1.5, 0, 0), ("rp", 0.5, 40, 10)]
MODELS = {
    "ll": dict(potential="ll"),
    "ll_dipole": dict(potential="ll", field_dir=(1, 0, 0.3), elecA=0.2, elecP=0.4),
    "ghrl_field": dict(potential="ghrl", k=(1.0, 0.5, 1.5), field_dir=(0, 1, 0), elecA=0.3),
    "ghrl": dict(potential="ghrl", k=(1.0, 0.5, 1.5)),
    "chiral": dict(potential="ghrl", k=(1.48, 1, 2.28, 12.0)),
    "pear": dict(potential="pear", A=1.5, B1=0.09, C=0.3),
}
LATTICES = [((21, 21, 21), "sphere", (0, 0, 0)), ((24, 24, 24), "sphere", (0, 0, 0)), ((33, 30, 20), "custom", (0, 1, 0)),
            ((40, 30, 20), "custom", (1, 0, 1)), ((2, 2, 2), "custom", (1, 1, 1)), ((1, 5, 1), "custom", (0, 0, 0))]


def geometry(dims, seed, empty=0.2):
    rng = np.random.default_rng(seed)
    n = int(np.prod(dims))
    pt = rng.choice([0, 1, 2, 3], size=n, p=[empty, 0.6 - empty / 2, 0.2 - empty / 4, 0.2 - empty / 4]).astype(np.int32)
    pt[n // 2] = 1
    nrm = rng.normal(size=(n, 3))
    return pt, (nrm / np.linalg.norm(nrm, axis=1)[:, None]).astype(np.float32)


def pair(name, lattice, T, replicas=1):
    dims, geo, per = lattice
    out = []
    for sched in (M.SCHED_CHECKER2, M.SCHED_CHECKER2_SIMPLE):
        e = M.Engine(M.Model(surfaces=SURF, **MODELS[name]),
                     [M.Replica(*dims, geo, per, T=T, elecE=1.2, seed=99 + r) for r in range(replicas)], sched)
        for r in range(replicas):
            if geo == "custom":
                e.set_geometry(r, *geometry(dims, 3 + r))
            e.random_directors(r, 5 + r)
        e.set_sweep_counter(2 ** 32 - 2)
        out.append(e)
    return out


def compare(a, b):
    for r in range(a.n):
        np.testing.assert_array_equal(a.download(r), b.download(r))
        assert a.ang_var(r) == b.ang_var(r)
        sa, sb = a.series(r), b.series(r)
        np.testing.assert_array_equal(sa["acceptance"], sb["acceptance"])
        # FP32 bond sums: each bond from one end instead of both
        np.testing.assert_allclose(sa["energy"], sb["energy"], rtol=2e-6, atol=2e-6)
        np.testing.assert_allclose(sa["q"], sb["q"], rtol=0, atol=1e-12)
        np.testing.assert_allclose(sa["nsum"], sb["nsum"], rtol=1e-12, atol=1e-9)


@pytest.mark.parametrize("lattice", LATTICES, ids=lambda s: "%dx%dx%d-%s" % (*s[0], s[1]))
@pytest.mark.parametrize("name", sorted(MODELS))
def test_lists_take_the_same_decisions(name, lattice):
    for T in (0.6, 0.0):
        a, b = pair(name, lattice, T, 2)
        for e in (a, b):
            e.sweeps(3)
            e.sweeps(4, measure=True)
        compare(a, b)
        if lattice[1] == "custom":
            for e in (a, b):  # another geometry: other lists
                e.set_geometry(1, *geometry(lattice[0], 77, 0.4))
                e.random_directors(1, 8)
                e.clear_series()
                e.sweeps(2, measure=True)
            compare(a, b)
        a.close()
        b.close()


def test_recorded_decisions_are_those_of_the_lists():
    a, b = pair("ll", LATTICES[0], 0.6)
    a.record_decisions()
    a.sweeps(2)
    b.sweeps(2)
    np.testing.assert_array_equal(a.download(0), b.download(0))
    a.record_decisions(False)
    a.sweeps(2, measure=True)
    b.sweeps(2, measure=True)
    compare(a, b)
    a.close()
    b.close()
