"""mcl_autotune while the ghost cells of periodic axes are out of date (after sweeps that do not keep them, such as
recorded ones): the sweeps after it read the present directors across the boundaries."""
import numpy as np
import pytest

from helpers import M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(24, 20, 16), (70, 66, 40)])
def test_tuning_after_recorded_sweeps(dims):
    out = []
    for tune in (True, False):
        e = M.Engine(M.Model("ll"), [M.Replica(*dims, T=0.8, seed=3)])
        e.random_directors(0, 4)
        e.record_decisions()
        e.sweeps(2)
        e.record_decisions(False)
        if tune:
            e.autotune(2)
        e.sweeps(3, measure=True)
        out.append((e.download(0), e.ang_var(0), e.sweep_counter()))
        e.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1:] == out[1][1:]
