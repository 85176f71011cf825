"""Waits that give up, on a GPU and without a fault: the state behind them is set
on the host (galaxy_bh_wait_probe)."""
import pytest

from galaxy_b200 import _lib, scenarios
from galaxy_b200.nbody_gpu import Config, NbodyGpu, ParallelTreeRuntime, bodies_to_state

pytestmark = pytest.mark.gpu


def test_a_step_behind_a_wait_that_gave_up_stops():
    """The sort's codes may be out of order then, and kernels that go by them would
    read out of place: they have to leave the cells alone and find nothing to sum."""
    gpu = NbodyGpu("0")
    status = _lib.load().galaxy_bh_wait_probe(gpu.handle, 1_000_000)
    assert (status, "timed out" in _lib.last_error()) == (_lib.BH_TIMEOUT, True), _lib.last_error()


def test_both_waits_of_the_sort_give_up_and_the_device_stays_usable():
    """The look-back waits for the tiles of a group and for groups of 32 tiles: each
    gives up on a predecessor that never publishes, and a simulation of two groups,
    which waits both ways, then repeats itself bit for bit."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    cfg = Config(theta=0.7, softening_kpc=0.01, g=1.0, bucket=2)
    rec = bodies_to_state(scenarios.make("cold_disc", 140001, 3, eps=0.01))

    def evolve():
        ev, _ = gpu.create_evolving_state_records(rec)
        tree = rt.create_tree(gpu, ev, cfg)
        rt.rebuild(gpu, ev, tree, cfg)
        rt.force(gpu, ev, tree, cfg)
        rt.step(gpu, ev, tree, cfg, 1e-3, 2)
        return gpu.read_evolving_state_records(ev)[0].tobytes()

    before = evolve()
    assert _lib.load().galaxy_bh_wait_probe(gpu.handle, 1_000_000) == _lib.BH_TIMEOUT
    assert "over tiles, over tile groups" in _lib.last_error()
    assert evolve() == before
