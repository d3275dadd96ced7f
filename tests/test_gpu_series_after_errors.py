"""A call that fails after some of its sweeps were queued: the records those left in the series are whole (S and the
director belong to the record's Q), through mcl_sweeps and mcl_sweeps_io. The failure is a series that cannot grow."""
import numpy as np
import pytest

from helpers import M
from oracle import learned as L

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("io", [False, True], ids=["sweeps", "sweeps_io"])
def test_records_of_a_failed_call_are_solved(io):
    n = 4096  # replicas: 622 KB per row of the series, which starts with 64 rows (40 MB)
    e = M.Engine(M.Model("ll"), [M.Replica(4, 4, 4, T=0.8, seed=1 + r) for r in range(n)])
    for r in range(n):
        e.random_directors(r, r)
    e.set_proposal(L.init_params(3).astype(np.float32))
    e.set_proposal_mix(2)
    e.sweeps_io(2)  # both kernels, their buffers and the series
    e.sweeps(2, measure=True)
    e.synchronize()
    torch.cuda.empty_cache()
    hold = []
    for piece in (1 << 30, 1 << 26, 1 << 24):  # less than the 80 MB of the next series stays free
        while torch.cuda.mem_get_info()[0] > 2 * piece + (16 << 20):
            hold.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
    assert torch.cuda.mem_get_info()[0] < 70 << 20
    with pytest.raises(M.McLicsError):
        e.sweeps_io(80) if io else e.sweeps(80, measure=True)
    del hold
    torch.cuda.empty_cache()
    assert e.series_length() == 64
    for r in (0, n // 2, n - 1):
        s = e.series(r)
        q = s["q"]
        m = np.stack([np.stack([q[:, 0], q[:, 1], q[:, 2]], 1), np.stack([q[:, 1], q[:, 3], q[:, 4]], 1),
                      np.stack([q[:, 2], q[:, 4], q[:, 5]], 1)], 1)
        w, v = np.linalg.eigh(m)
        np.testing.assert_allclose(s["S"], w[:, 2], rtol=0, atol=1e-12)
        np.testing.assert_allclose(np.abs((s["director"] * v[:, :, 2]).sum(1)), 1, rtol=0, atol=1e-9)
    e.sweeps(2, measure=True)  # the engine stays usable
    assert e.series_length() == 66
    e.close()
