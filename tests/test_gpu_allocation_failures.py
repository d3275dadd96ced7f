"""A device allocation that fails is reported by the call that needed it, and by no later one."""
import pytest

from helpers import M

pytestmark = pytest.mark.gpu


def test_a_failed_allocation_is_reported_once():
    e = M.Engine(M.Model("ll"), [M.Replica(8, 8, 8, T=0.8)])
    with pytest.raises(M.McLicsError):
        e.reserve_series(2_000_000_000)  # 304 GB
    e.sweeps(2, measure=True)  # the first launch after it
    assert e.series_length() == 2
    with pytest.raises(M.McLicsError):
        e.reserve_series(2_000_000_000)
    other = M.Engine(M.Model("ll"), [M.Replica(8, 8, 8, T=0.8)])
    other.sweeps(1)
    other.close()
    e.close()
