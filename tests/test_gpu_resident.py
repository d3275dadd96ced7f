"""The resident sweep (small lattices in the shared memory of a thread-block cluster) against the colour passes: the
same draws, the same arithmetic, so directors, acceptances and amplitudes are the same bits; observables differ by the
grouping of their FP32 sums. Shapes at the edges of its task map: odd and tiny extents, free and periodic axes, one
plane, more replicas than clusters, uneven replicas, every kernel combination of the models, calls of one and of many
sweeps, and one-step calls from a captured graph."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu

SURF = [("homeotropic", 1.5, 0, 0), ("rp", 0.5, 40, 10)]
GSURF = [("rp_ghrl", 1.0, 90, 30), ("fg_ghrl", 0.8, 0, 0)]
MODELS = {
    "ll": dict(potential="ll"),
    "ll_field": dict(potential="ll", field_dir=(1, 0, 0.3), elecA=0.2),
    "ll_dipole": dict(potential="ll", field_dir=(1, 0, 0.3), elecA=0.2, elecP=0.4),
    "ghrl": dict(potential="ghrl", k=(1.0, 0.5, 1.5)),
    "ghrl_field": dict(potential="ghrl", k=(1.0, 0.5, 1.5), field_dir=(0, 1, 0), elecA=0.3),
    "ghrl_dipole": dict(potential="ghrl", k=(1.0, 0.5, 1.5), field_dir=(0, 1, 0), elecP=0.2),
    "chiral": dict(potential="ghrl", k=(1.48, 1, 2.28, 12.0)),
    "chiral_field": dict(potential="ghrl", k=(1.48, 1, 2.28, 12.0), field_dir=(0, 1, 0), elecA=0.1),
    "chiral_dipole": dict(potential="ghrl", k=(1.48, 1, 2.28, 12.0), field_dir=(0, 1, 0), elecP=0.2),
    "pear": dict(potential="pear", A=1.5, B1=0.09, C=0.3),
    "pear_field": dict(potential="pear", A=1.5, B1=0.09, C=0.3, field_dir=(0.3, 0, 1), elecP=0.7, elecA=0.1),
}
SHAPES = [
    (32, 32, 32, "bulk", (1, 1, 1)), (2, 2, 2, "bulk", (1, 1, 1)), (6, 4, 4, "bulk", (1, 0, 1)),
    (30, 18, 26, "bulk", (0, 0, 0)), (29, 10, 9, "bulk", (0, 0, 0)), (1, 1, 1, "bulk", (0, 0, 0)),
    (5, 1, 3, "bulk", (0, 0, 0)), (66, 12, 10, "bulk", (1, 1, 1)), (17, 16, 15, "bulk", (0, 1, 0)),
    (28, 20, 17, "slab", (1, 1, 0)), (16, 16, 1, "slab", (1, 1, 0)), (50, 34, 5, "slab", (0, 1, 0)),
]


def model(name, geometry):
    surfaces = (GSURF if "chiral" in name else SURF) if geometry == "slab" else []
    return M.Model(surfaces=surfaces, **MODELS[name])


def engines(m, reps):
    """The engine's own choice, and the colour passes by a plan; random directors, equal seeds."""
    out = []
    for plan in (None, (4, 3)):
        e = M.Engine(m, reps)
        if plan:
            e.set_plan(*plan)
        for r in range(e.n):
            e.random_directors(r, 5 + r)
        e.set_sweep_counter(2 ** 32 - 3)  # the upper half of the counter changes on the way
        out.append(e)
    return out


def launches(e, n, measure):
    a = e.profile_read()[2]
    e.sweeps(n, measure)
    return e.profile_read()[2] - a


def compare(a, b):
    for r in range(a.n):
        np.testing.assert_array_equal(a.download(r), b.download(r))
        assert a.ang_var(r) == b.ang_var(r)
        sa, sb = a.series(r), b.series(r)
        for k in ("acceptance", "ang_var", "sweep", "n_valid"):
            np.testing.assert_array_equal(sa[k], sb[k], err_msg=k)
        # FP32 partial sums in another grouping: the tolerances of the tiled kernels' comparison
        np.testing.assert_allclose(sa["energy"], sb["energy"], rtol=2e-6, atol=2e-6)
        np.testing.assert_allclose(sa["q"], sb["q"], rtol=0, atol=4e-7)
        np.testing.assert_allclose(sa["S"], sb["S"], rtol=0, atol=2e-6)
    assert a.sweep_counter() == b.sweep_counter() and a.series_length() == b.series_length()


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%dx%d-%s-%s" % (*s[:4], "".join(map(str, s[4]))))
@pytest.mark.parametrize("name", sorted(MODELS))
def test_resident_equals_colour_passes(name, shape):
    nx, ny, nz, geo, per = shape
    for T in (0.9, 0.0):
        a, b = engines(model(name, geo), [M.Replica(nx, ny, nz, geo, per, T=T, elecE=1.2, seed=99)])
        assert launches(a, 3, False) == 1  # one launch for the call: the resident kernel runs
        b.sweeps(3)
        for n, measure in ((4, True), (1, False), (1, True)):
            a.sweeps(n, measure)
            b.sweeps(n, measure)
        compare(a, b)
        a.close()
        b.close()


@pytest.mark.parametrize("sizes", [[(16, 16, 16), (20, 20, 20), (32, 32, 32), (10, 12, 14)], [(24, 24, 24)] * 40],
                         ids=["uneven", "more-than-clusters"])
def test_resident_batches(sizes):
    reps = [M.Replica(*s, T=0.4 + 0.05 * i, seed=9 + i) for i, s in enumerate(sizes)]
    a, b = engines(model("ll", "bulk"), reps)
    assert launches(a, 5, False) == 1
    b.sweeps(5)
    a.sweeps(6, True)
    b.sweeps(6, True)
    compare(a, b)
    a.close()
    b.close()


def test_resident_steps_from_a_graph_and_without_adaptation():
    a, b = engines(model("ll", "bulk"), [M.Replica(32, 32, 32, T=1.0, seed=3)])
    T = np.array([1.05], np.float32)
    for e in (a, b):
        e.set_graphs(True)
        rec = [e.sweeps_io(1, T) for _ in range(3)]
        e.set_adaptation(False)
        rec += [e.sweeps_io(1, T), e.sweeps_io(4, T)]
        e.last = np.concatenate(rec)
    np.testing.assert_array_equal(a.last["acceptance"], b.last["acceptance"])
    np.testing.assert_array_equal(a.last["ang_var"], b.last["ang_var"])
    np.testing.assert_allclose(a.last["energy"], b.last["energy"], rtol=2e-6, atol=0)
    np.testing.assert_allclose(a.last["S"], b.last["S"], rtol=0, atol=2e-6)
    compare(a, b)
    a.close()
    b.close()


def test_a_plan_and_the_wait_hook_bring_the_colour_passes_back():
    e = M.Engine(model("ll", "bulk"), [M.Replica(32, 32, 32, T=1.0, seed=3)])
    assert launches(e, 2, False) == 1
    e.debug_wait_limit(20_000_000, withhold_first_load=True)
    with pytest.raises(M.McLicsError):
        e.sweeps(1)
        e.synchronize()
    e.debug_wait_limit(2_000_000_000, withhold_first_load=False)
    assert launches(e, 2, False) == 1
    e.set_plan(2, 0)
    assert launches(e, 2, False) == 6
    t = e.autotune(20)
    assert t["ms_per_sweep"] <= t["ms_default"]
    e.close()
