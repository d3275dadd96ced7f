"""The tile plan an engine chooses by itself (configuration and planes per segment by expected time) on lattices too
large for the resident sweep: whatever it picks, the directors are those of a plan asked for."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu

MODELS = {
    "ll": lambda s: M.Model("ll", surfaces=s),
    "ghrl": lambda s: M.Model("ghrl", k=(1.0, 0.5, 1.5), surfaces=s),
    "chiral": lambda s: M.Model("ghrl", k=(1.48, 1, 2.28, 12.0), field_dir=(0, 0, 1), elecA=0.1, surfaces=s),
    "pear": lambda s: M.Model("pear", field_dir=(0, 0, 1), elecP=1.0, surfaces=s),
}
SHAPES = [((64, 64, 64), "bulk", (1, 1, 1), 1), ((130, 70, 50), "slab", (1, 1, 0), 1), ((101, 75, 50), "bulk", (0, 0, 0), 1),
          ((200, 300, 3), "slab", (1, 1, 0), 1), ((34, 250, 40), "bulk", (1, 1, 1), 2), ((300, 40, 2), "bulk", (1, 1, 1), 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "%dx%dx%d-%s" % (*s[0], s[1]))
@pytest.mark.parametrize("name", sorted(MODELS))
def test_default_plan_takes_the_same_decisions(name, shape):
    dims, geo, per, n = shape
    m = MODELS[name]([("homeotropic", 1.0, 0, 0)] * 2 if geo == "slab" else [])
    out = []
    for plan in (None, (2, 8), (3, 5)):
        e = M.Engine(m, [M.Replica(*dims, geo, per, T=0.7, seed=7 + r) for r in range(n)])
        p = e.plan()
        assert p["tile_config"] in (2, 3, 4) and 1 <= p["planes_per_segment"] <= dims[2]
        if plan:
            e.set_plan(*plan)
        for r in range(n):
            e.random_directors(r, 3 + r)
        e.sweeps(2)
        e.sweeps(3, measure=True)
        out.append(([e.download(r) for r in range(n)], [e.series(r) for r in range(n)]))
        e.close()
    for dirs, series in out[1:]:
        for r in range(n):
            np.testing.assert_array_equal(dirs[r], out[0][0][r])
            np.testing.assert_array_equal(series[r]["acceptance"], out[0][1][r]["acceptance"])
            np.testing.assert_allclose(series[r]["energy"], out[0][1][r]["energy"], rtol=2e-6, atol=2e-6)
