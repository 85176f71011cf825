"""Stage times of a rebuild."""
import ctypes as C

import numpy as np
import pytest

from galaxy_b200 import _lib, scenarios
from galaxy_b200.nbody_gpu import Config, NbodyGpu, ParallelTreeRuntime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 4096, 16385, 65536, 65537])
def test_every_stage_has_its_own_time(n):
    """A leaf size of 1,000 has the chain counts (topology) look at up to 1,000
    neighbours of each position, many times the sort's work, which does not depend on
    it: the time appears as topology, whether one launch does all stages (up to
    65,536 bodies) or each has its own.  (1,000 bodies are one leaf: no neighbours.)"""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    times = []
    for bucket in (1, 1000):
        cfg = Config(theta=0.5, softening_kpc=0.01, g=1.0, bucket=bucket)
        ev, _ = gpu.create_evolving_state(scenarios.make("cold_disc", n, 5, eps=0.01))
        tree = rt.create_tree(gpu, ev, cfg)
        t = [rt.rebuild(gpu, ev, tree, cfg) for _ in range(9)]
        times.append(np.median([[x.bounds_seconds, x.morton_seconds, x.radix_seconds,
                                 x.topology_seconds] for x in t], axis=0))
    (_, _, sort1, chains1), (bounds, codes, sort, chains) = times
    assert min(bounds, codes) > 0.0
    assert n <= 1000 or (chains > 4.0 * chains1 and chains > sort)
    assert sort < 2.0 * sort1


@pytest.mark.parametrize("bucket", [1, 7])
def test_a_rebuild_without_times_builds_the_same_tree(bucket):
    """Callers that ask for no times get another form of the small sort: the same
    bits, at the edges of its blocks and clusters."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    cfg = Config(theta=0.5, softening_kpc=0.01, g=1.0, bucket=bucket)
    for n in (2, 33, 1024, 1025, 2049, 4096, 4097, 8193, 16385, 32769, 65535, 65536):
        ev, _ = gpu.create_evolving_state(scenarios.make("exponential_disc", n, n, eps=0.01))
        tree = rt.create_tree(gpu, ev, cfg)
        rt.rebuild(gpu, ev, tree, cfg)
        timed = rt.read_evidence(gpu, tree)
        rt.rebuild(gpu, ev, tree, Config(theta=0.5, softening_kpc=0.01, g=1.0, bucket=bucket + 2))
        assert rt.read_evidence(gpu, tree).cells.tobytes() != timed.cells.tobytes() or n < 8
        _lib.check(_lib.load().galaxy_bh_tree_rebuild(gpu.handle, ev.handle, tree.handle,
                                                      C.byref(cfg.to_c()), None))
        plain = rt.read_evidence(gpu, tree)
        for a, b in ((timed.entries, plain.entries), (timed.bodies, plain.bodies),
                     (timed.cells, plain.cells)):
            assert a.tobytes() == b.tobytes(), n
