"""Graphs of sweeps on colour-pass plans against direct launches, bit for bit: calls around the length of a graph, with
and without measurement, one sweep on an idle and on a busy stream, across a series that moves, a switched adaptation,
another plan, temperatures and a cleared series; and that graphs were replayed at all, where they should be."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SURF = [("homeotropic", 1.5, 0, 0), ("rp", 0.5, 40, 10)]
CASES = {
    "ll-bulk": (dict(potential="ll"), [(36, 22, 26), (16, 16, 16), (50, 34, 12)], "bulk", (1, 1, 1), (2, 7)),
    "ghrl-slab": (dict(potential="ghrl", k=(1.0, 0.5, 1.5), surfaces=SURF), [(66, 34, 20)], "slab", (1, 1, 0), (4, 5)),
    "pear-slab": (dict(potential="pear", A=1.5, B1=0.09, C=0.3, surfaces=SURF), [(34, 30, 17), (20, 16, 9)], "slab",
                  (1, 0, 0), (3, 6)),
    "ll-dipole": (dict(potential="ll", field_dir=(1, 0, 0.3), elecA=0.2, elecP=0.4), [(40, 18, 14)], "bulk", (0, 1, 1),
                  (4, 3)),
}


def engine(case, graphs):
    model, sizes, geo, per, plan = CASES[case]
    e = M.Engine(M.Model(**model), [M.Replica(*s, geo, per, T=0.8, seed=3 + r) for r, s in enumerate(sizes)])
    e.set_plan(*plan)
    for r in range(e.n):
        e.random_directors(r, 9 + r)
    e.set_sweep_counter(2 ** 32 - 20)
    e.set_graphs(graphs)
    return e


def same(a, b):
    assert a.sweep_counter() == b.sweep_counter() and a.series_length() == b.series_length()
    for r in range(a.n):
        np.testing.assert_array_equal(a.download(r), b.download(r))
        assert a.ang_var(r) == b.ang_var(r)
        assert a.series(r).tobytes() == b.series(r).tobytes()


@pytest.mark.parametrize("case", sorted(CASES))
def test_graphs_of_any_length_of_call(case):
    a, b = engine(case, False), engine(case, True)

    def both(n, measure, replays):
        before = b.debug_graph_replays()
        for e in (a, b):
            e.sweeps(n, measure)
        assert b.debug_graph_replays() - before == replays, n
        assert a.debug_graph_replays() == 0

    for n in (8, 9, 17, 29, 7, 3):
        for measure in (False, True):
            both(n, measure, n // 8)
    same(a, b)
    both(37, True, 4)  # more records than before: the series has moved
    same(a, b)
    for e in (a, b):
        e.set_adaptation(False)
    both(16, True, 2)
    same(a, b)
    for e in (a, b):
        e.set_adaptation(True)
        e.set_temperature(0.5)
        e.clear_series()
    both(11, True, 1)
    same(a, b)
    for e in (a, b):
        e.set_plan(2, 4)
    both(24, False, 3)
    both(10, True, 1)
    same(a, b)
    for measure in (False, True):
        b.synchronize()
        both(1, measure, 1)  # an idle stream
    same(a, b)
    for e in (a, b):
        for k in range(6):
            e.sweeps(1, k % 2 == 0)  # as the stream happens to be
    same(a, b)
    a.close()
    b.close()


def test_one_sweep_graphs_leave_a_capture_alone():
    a, b = engine("ll-bulk", True), engine("ll-bulk", False)
    s = torch.cuda.Stream()
    a.set_stream(s.cuda_stream)
    a.sweeps(1)
    a.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        a.sweeps(1)
    with torch.cuda.stream(s):
        g.replay()
    torch.cuda.synchronize()
    b.sweeps(2)
    same(a, b)
    a.set_stream(0)
    a.close()
    b.close()
