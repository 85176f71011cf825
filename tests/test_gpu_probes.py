"""FP64 direct probes over many slices of the sources."""
import numpy as np
import pytest

from galaxy_b200 import scenarios
from galaxy_b200.nbody_gpu import Config, NbodyGpu, bodies_to_state, state_to_bodies

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1 << 22) + 1, 9_200_003])
def test_few_probes_of_many_bodies(n):
    """Few probes are summed in up to 4,440 slices of the sources (2,049 and 4,440
    here), added with their roundings kept: at most 8 terms a thread in turn, a tree of
    8 levels and a few roundings for the slices, against numpy's sum in pairs (16 in
    turn, 17 levels).  With 8 roundings a term on either side the difference is below
    128 2^-53 of the terms' magnitudes."""
    gpu, eps = NbodyGpu("0"), 0.01
    bodies = scenarios.make("cold_disc", n, 5, eps=eps)
    records = bodies_to_state(bodies)
    b32 = state_to_bodies(records)
    ev, _ = gpu.create_evolving_state_records(records)
    probes = np.array([0, n // 2, n - 1], np.uint32)
    got = gpu.direct_probes(ev, Config(theta=0.5, softening_kpc=eps, g=1.0), probes)
    for probe, a in zip(probes, got):
        d = b32[:, :2] - b32[probe, :2]
        r2 = d[:, 0] ** 2 + d[:, 1] ** 2 + eps * eps
        terms = d * (b32[:, 4] / (r2 * np.sqrt(r2)))[:, None]
        want = np.array([terms[:, 0].copy().sum(), terms[:, 1].copy().sum()])
        assert (np.abs(a - want) <= 128 * 2.0 ** -53 * np.abs(terms).sum(0)).all()
