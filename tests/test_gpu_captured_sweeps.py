"""Sweeps of a custom lattice captured into a caller's graph: accepted also right after a geometry was set, when the site
lists of the sweep are not built yet (nothing in a capture may wait for the device), and a replay sweeps the geometry in
force, also one set after the capture."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DIMS = (18, 15, 10)


def geometry(seed, empty):
    rng = np.random.default_rng(seed)
    n = int(np.prod(DIMS))
    pt = rng.choice([0, 1, 2], size=n, p=[empty, 0.8 - empty, 0.2]).astype(np.int32)
    nrm = rng.normal(size=(n, 3))
    return pt, (nrm / np.linalg.norm(nrm, axis=1)[:, None]).astype(np.float32)


@pytest.mark.parametrize("listed", [False, True], ids=["before-the-lists", "with-lists"])
def test_captured_sweeps_follow_the_geometry(listed):
    model = M.Model("ll", surfaces=[("homeotropic", 1.5, 0, 0)])
    a, b = (M.Engine(model, [M.Replica(*DIMS, "custom", (0, 0, 0), T=0.6, seed=5)]) for _ in range(2))

    def both(f):
        for e in (a, b):
            f(e)

    def same():
        np.testing.assert_array_equal(a.download(0), b.download(0))
        assert a.sweep_counter() == b.sweep_counter()

    both(lambda e: e.set_geometry(0, *geometry(4, 0.5)))
    both(lambda e: e.random_directors(0, 3))
    if listed:
        both(lambda e: e.sweeps(1))
    s = torch.cuda.Stream()
    a.set_stream(s.cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        a.sweeps(3)
    g.replay()
    torch.cuda.synchronize()
    b.sweeps(3)
    same()
    both(lambda e: e.sweeps(2))
    same()
    both(lambda e: e.set_geometry(0, *geometry(8, 0.2)))  # more sites than before
    both(lambda e: e.random_directors(0, 6))
    both(lambda e: e.sweeps(1))
    with torch.cuda.stream(s):
        g.replay()
    torch.cuda.synchronize()
    b.sweeps(3)
    same()
    a.set_stream(0)
    both(lambda e: e.close())
