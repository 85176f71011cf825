"""Device memory that a call takes for its own length is given back."""
import pytest
import torch

from galaxy_b200 import scenarios
from galaxy_b200.nbody_gpu import Config, NbodyGpu, ParallelTreeRuntime

pytestmark = pytest.mark.gpu


def test_a_large_export_keeps_no_memory():
    """The evidence of 3,000,000 bodies takes about 480 MB on the device: the handle
    keeps at most 256 MB of what single calls took."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    cfg = Config(theta=0.5, softening_kpc=0.005, g=1.0, bucket=1)
    ev, _ = gpu.create_evolving_state(scenarios.make("cold_disc", 3_000_000, 3, eps=0.005))
    tree = rt.create_tree(gpu, ev, cfg)
    rt.rebuild(gpu, ev, tree, cfg)
    rt.force(gpu, ev, tree, cfg)
    free = torch.cuda.mem_get_info()[0]
    evidence = rt.read_evidence(gpu, tree)
    assert evidence.cells.nbytes + evidence.bodies.nbytes + evidence.entries.nbytes > 400 << 20
    # (and 32 MB for the granularity that the driver maps memory in)
    assert free - torch.cuda.mem_get_info()[0] <= (256 + 32) << 20
