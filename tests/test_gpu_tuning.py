"""The launch-shape knobs reach the kernels."""
import json

import pytest
import torch

from galaxy_b200 import scenarios
from galaxy_b200.nbody_gpu import Config, NbodyGpu, ParallelTreeRuntime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.01, 1e-20, 0.0])
def test_traverse_warps_with_any_softening(tmp_path, eps):
    """2, 4 or 8 warps a traversal block, also where the softening squared is zero or
    subnormal (another form of the kernel), with the same bits."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    cfg = Config(theta=0.5, softening_kpc=eps, g=1.0, bucket=1, force_stats=False)
    ev, _ = gpu.create_evolving_state(scenarios.exponential_disc(3000, 5))
    tree = rt.create_tree(gpu, ev, cfg)
    rt.rebuild(gpu, ev, tree, cfg)
    rt.force(gpu, ev, tree, cfg)
    want = gpu.read_evolving_accelerations_f32(ev)[0].tobytes()
    for warps in (2, 4, 8):
        rt.tune(tree, traverse_warps=warps)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            rt.force(gpu, ev, tree, cfg)
        trace = str(tmp_path / f"{warps}.json")
        prof.export_chrome_trace(trace)
        blocks = [e["args"]["block"][0] for e in json.load(open(trace))["traceEvents"]
                  if "k_traverse<" in e.get("name", "") and "block" in e.get("args", {})]
        assert blocks == [32 * warps]
        assert gpu.read_evolving_accelerations_f32(ev)[0].tobytes() == want
