"""Order between torch's stream, which gathers a batch and allocates the sample buffers, and the library's own streams,
which train on and fill them: a trainer step or an extraction may start only after torch's stream has been waited for
since the last work was queued on it. On the CPU, with a torch and a library that only keep the order of the calls."""
import sys
import types

import numpy as np
import pytest

from helpers import M
from mclics_b200 import learned


class Tensor:
    def __init__(self, log, shape):
        self.log, self.shape = log, shape

    def __getitem__(self, i):
        self.log.append("queue")
        return self

    def contiguous(self):
        return self

    def data_ptr(self):
        return 8


@pytest.fixture
def log(monkeypatch):
    log = []
    torch = types.ModuleType("torch")
    torch.float32 = "float32"
    torch.Generator = lambda device: types.SimpleNamespace(manual_seed=lambda s: None)

    def queued(n, **kw):
        log.append("queue")
        return Tensor(log, (n,) if isinstance(n, int) else n)

    torch.randperm = torch.empty = queued
    torch.cuda = types.SimpleNamespace(
        current_stream=lambda *a: types.SimpleNamespace(synchronize=lambda: log.append("wait")))
    monkeypatch.setitem(sys.modules, "torch", torch)

    class Trainer:
        def __init__(self, params, batch):
            pass

        def step(self, *a):
            log.append("use")
            return 0.0

        def params(self):
            return np.zeros(3)

        def close(self):
            pass

    monkeypatch.setattr(M, "Trainer", Trainer)
    return log


def check(log, uses):
    assert log.count("use") == uses
    waited = False
    for what in log:
        if what == "use":
            assert waited
        else:
            waited = what == "wait"


def test_a_step_waits_for_its_batch(log):
    feat, dirs = Tensor(log, (64, 8)), Tensor(log, (64, 3))
    learned.train(feat, dirs, epochs=2, batch=16, params=np.zeros(M.N_MLP_PARAMS, np.float32))
    check(log, 8)


def test_samples_go_to_buffers_that_torch_has_done_with(log):
    engine = types.SimpleNamespace(n=2, sweeps=lambda n: None, extract_samples=lambda *a: log.append("use"))
    learned.collect(engine, snapshots=2, gap=1, per_snapshot=5)
    # a slice of a buffer queues nothing in torch: only the allocation counts
    check([w for i, w in enumerate(log) if w != "queue" or i < 2], 4)
