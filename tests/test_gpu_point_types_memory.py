"""Site lists that the host has no memory for: the sweep goes on without them, with the same decisions. In a process of
its own whose address space is limited for that one call."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import resource
import numpy as np
from helpers import M

DIMS = (256, 256, 208)  # 109 MB of lists, in arrays that grow
n = int(np.prod(DIMS))
pt = np.ones(n, np.int32)
pt[::7] = 2
nrm = np.zeros((n, 3), np.float32)
nrm[:, 2] = 1
engines = []
for schedule in (M.SCHED_CHECKER2_SIMPLE, M.SCHED_CHECKER2):
    e = M.Engine(M.Model("ll", surfaces=[("homeotropic", 1.5, 0, 0)]),
                 [M.Replica(*DIMS, "custom", (1, 1, 1), T=0.6, seed=5)], schedule)
    e.set_geometry(0, pt, nrm)
    e.random_directors(0, 3)
    engines.append(e)
a, b = engines
a.sweeps(2, measure=True)  # loads the kernels that both use
a.synchronize()
pages = int(open("/proc/self/statm").read().split()[0])
old = resource.getrlimit(resource.RLIMIT_AS)
resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + (48 << 20), old[1]))
b.sweeps(2, measure=True)
b.synchronize()
resource.setrlimit(resource.RLIMIT_AS, old)
assert np.array_equal(a.download(0), b.download(0))
# per sweep two colours, the observables (part of the list sweep where there are lists) and the finalisation
assert b.profile_read()[2] == 2 * 4 + 1
print("same")
"""


def test_the_sweep_goes_on_without_lists_it_has_no_memory_for():
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=here, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=here))
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr
