"""Waits that give up, on a GPU and without a fault: the state behind them is set
on the host (galaxy_bh_wait_probe)."""
import pytest

from galaxy_b200 import _lib
from galaxy_b200.nbody_gpu import NbodyGpu

pytestmark = pytest.mark.gpu


def test_a_step_behind_a_wait_that_gave_up_stops():
    """The sort's codes may be out of order then, and kernels that go by them would
    read out of place: they have to leave the cells alone and find nothing to sum."""
    gpu = NbodyGpu("0")
    status = _lib.load().galaxy_bh_wait_probe(gpu.handle, 1_000_000)
    assert (status, "timed out" in _lib.last_error()) == (_lib.BH_TIMEOUT, True), _lib.last_error()
