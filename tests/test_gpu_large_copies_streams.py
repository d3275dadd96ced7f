"""Large downloads on streams other than the engine's own, the per-thread default stream among them (whose handle names
another stream in every host thread): what arrives is the state after the sweeps queued before. More engines at once
than there are pinned rings, rings given back in between, and pinned destinations."""
import threading

import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DIMS = [(128, 128, 90), (150, 131, 149)]  # 17.7 MB and 35.1 MB, no multiples of a chunk
PER_THREAD = 2  # cudaStreamPerThread


def engine(dims, seed=1):
    e = M.Engine(M.Model("ll"), [M.Replica(*dims, "bulk", (0, 0, 0), T=0.7, seed=seed)])
    e.random_directors(0, seed)
    return e


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("which", ["per-thread", "caller"])
def test_downloads_follow_the_sweeps_on_the_engines_stream(which, dims):
    a, b = engine(dims), engine(dims)
    s = torch.cuda.Stream()
    a.set_stream(PER_THREAD if which == "per-thread" else s.cuda_stream)
    for _ in range(4):
        a.sweeps(20)  # still running when the download is asked for
        got = a.download(0)
        b.sweeps(20)
        b.synchronize()
        np.testing.assert_array_equal(got, b.download(0))
    a.sweeps(10)
    b.sweeps(10)
    np.testing.assert_array_equal(a.local_order(0), b.local_order(0))
    a.set_stream(0)
    a.close()
    b.close()


def test_more_engines_than_rings_and_rings_given_back():
    wrong = []

    def work(seed):
        e, t = engine(DIMS[1], seed), engine(DIMS[1], seed)
        for k in range(4):
            e.sweeps(3)
            t.sweeps(3)
            if not np.array_equal(e.download(0), t.download(0)):
                wrong.append(seed)
            if seed == 3:
                M.trim()
        e.close()
        t.close()

    threads = [threading.Thread(target=work, args=(s,)) for s in range(3, 8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    M.trim()
    M.trim()


def test_pinned_and_kept_destinations():
    e = engine(DIMS[1])
    ref = e.download(0)
    for out in (torch.empty(ref.size, dtype=torch.float32).pin_memory().numpy(), np.ones(ref.size, np.float32)):
        for _ in range(2):
            M.check(M.lib().mcl_download_directors(e._h, 0, out.ctypes.data))
            np.testing.assert_array_equal(out, ref)
            out[:] = 0
    e.close()
