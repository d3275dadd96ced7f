"""Downloads and local order parameters large enough for the pinned ring (16 MiB and more): every chunk lands where it
belongs, in arrays whose size is no multiple of a chunk, again and again, and from two threads with an engine each."""
import threading

import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu


def field(n, seed):
    v = np.random.default_rng(seed).normal(size=(n, 3)).astype(np.float32)
    return (v / np.linalg.norm(v, axis=1)[:, None]).reshape(-1)


@pytest.mark.parametrize("dims", [(128, 128, 86), (150, 131, 149), (256, 256, 70)])
def test_large_downloads_return_what_was_uploaded(dims):
    e = M.Engine(M.Model("ll"), [M.Replica(*dims, "bulk", (0, 0, 0), T=1.0, seed=1)])
    for seed in (1, 2):
        ni = field(e.sites(0), seed)
        assert ni.nbytes >= 16 << 20
        e.upload(0, ni)
        np.testing.assert_array_equal(e.download(0), ni)
    big, small = e.local_order(0), M.Engine(M.Model("ll"), [M.Replica(*dims[:2], 4, "bulk", (0, 0, 0), T=1.0)])
    small.upload(0, ni[:3 * dims[0] * dims[1] * 4])
    n = dims[0] * dims[1] * 3  # the first three planes do not see beyond the fourth
    np.testing.assert_array_equal(big[:n], small.local_order(0)[:n])
    e.close()
    small.close()


def test_large_downloads_in_two_threads():
    dims, wrong = (150, 131, 149), []

    def work(seed):
        e = M.Engine(M.Model("ll"), [M.Replica(*dims, "bulk", (0, 0, 0), T=1.0, seed=1)])
        ni = field(e.sites(0), seed)
        e.upload(0, ni)
        for _ in range(4):
            if not np.array_equal(e.download(0), ni):
                wrong.append(seed)
        e.close()

    threads = [threading.Thread(target=work, args=(s,)) for s in (3, 4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
