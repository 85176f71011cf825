"""Opening decisions where squared distances come near the end of f32."""
import numpy as np
import pytest

from galaxy_b200 import scenarios
from galaxy_b200.nbody_gpu import (Config, NbodyGpu, ParallelTreeRuntime, bodies_to_state,
                                   state_to_bodies)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crit", [9.99999999e18, 1.1e19, 1.6e19])
def test_decisions_equal_the_reference_near_the_end_of_f32(oracle, crit):
    """Distances of up to 2e19 have squares of up to 4e38, the end of f32 is 3.4e38,
    and the critical distance (width / theta) of the root's children is `crit`: the
    same cells are visited, approximated and summed as in the reference's f64."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    bodies = np.array(scenarios.make("cold_disc", 3000, 4, eps=0.01))
    bodies[:, :2] *= 1e19
    bodies[:, 2:4] = 0.0
    b32 = state_to_bodies(bodies_to_state(bodies))
    span = float(max(np.ptp(b32[:, 0]), np.ptp(b32[:, 1])))
    cfg = Config(theta=(span * 0.500000000001 + 1e-12) / crit, softening_kpc=1e10, g=1.0, bucket=1)
    ev, _ = gpu.create_evolving_state(bodies)
    tree = rt.create_tree(gpu, ev, cfg)
    rt.rebuild(gpu, ev, tree, cfg)
    rt.force(gpu, ev, tree, cfg)
    got = rt.force_stats(gpu, tree)
    oc = oracle.Config(theta=cfg.theta, softening=cfg.softening_kpc, g=cfg.g, bucket=1, max_depth=48)
    want = oracle.flat_accelerations(b32, oracle.build_flat_tree(b32, oc), oc)[1]
    for key in ("visited_nodes", "approximated_cells", "direct_terms"):
        assert got[key] == want[key], key


@pytest.mark.parametrize("theta", [1e-20, 1e-38, 1e-39, 1e-44])
def test_tiny_angles_open_every_cell_without_the_f64_test(theta):
    """A critical distance far beyond every body's, also beyond f32, opens each cell as
    theta = 0 does, and no decision is left to f64."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    bodies = scenarios.exponential_disc(2000, 5)
    ev, _ = gpu.create_evolving_state(bodies)
    got = []
    for angle in (0.0, theta):
        cfg = Config(theta=angle, softening_kpc=0.01, g=1.0, bucket=1)
        tree = rt.create_tree(gpu, ev, cfg)
        rt.rebuild(gpu, ev, tree, cfg)
        rt.force(gpu, ev, tree, cfg)
        got.append((rt.force_stats(gpu, tree), gpu.read_evolving_accelerations_f32(ev)[0].tobytes()))
    assert got[0][0]["exact_mac_fallbacks"] == 0
    assert got[0] == got[1]
