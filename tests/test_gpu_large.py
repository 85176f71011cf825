"""Copies and batches of large simulations."""
import numpy as np
import pytest
import torch

from galaxy_b200 import _lib, scenarios
from galaxy_b200.batch import Batch
from galaxy_b200.nbody_gpu import Config, NbodyGpu, ParallelTreeRuntime

pytestmark = pytest.mark.gpu


def test_copies_of_mixed_sizes_and_pinned_arrays_on_one_handle():
    """Arrays of 16 MB and more go through the handle's pinned slots, smaller and
    pinned ones do not: one after the other, in both directions, each whole."""
    gpu, lib, rng = NbodyGpu("0"), _lib.load(), np.random.default_rng(3)
    states = []
    for n in (700_001, 300, (1 << 20) + 3, 524_288):
        rec = rng.uniform(0.5, 2.0, (n, 8)).astype(np.float32)
        states.append((gpu.create_evolving_state_records(rec.view(_lib.EVOLVE_STATE_DTYPE)[:, 0])[0],
                       rec))
    pinned = torch.empty(((1 << 20) + 3, 8), dtype=torch.float32, pin_memory=True).numpy()
    for order in ((0, 2, 1, 3), (3, 0, 1, 2)):
        for k in order:
            ev, rec = states[k]
            got = gpu.read_evolving_state_records(ev)[0]
            assert np.array_equal(got.view(np.uint32).ravel(), rec.view(np.uint32).ravel())
            pinned[:len(rec)] = rec[::-1]  # a pinned upload, read back pinned
            _lib.check(lib.galaxy_bh_write_state(gpu.handle, ev.handle, _lib.ptr(pinned), len(rec)))
            pinned[:] = 0.0
            _lib.check(lib.galaxy_bh_read_state(gpu.handle, ev.handle, _lib.ptr(pinned), len(rec),
                                                None))
            assert np.array_equal(pinned[:len(rec)], rec[::-1])
            rec = np.ascontiguousarray(rec * np.float32(1.5))  # and a pageable one
            _lib.check(lib.galaxy_bh_write_state(gpu.handle, ev.handle, _lib.ptr(rec), len(rec)))
            states[k] = (ev, rec)


def test_batch_with_outer_cuts_every_256_blocks():
    """Above 8,192 blocks of the aggregates (2,097,152 positions in all) an outer cut is
    every 256 of them instead of every 128, for the small members too: each has the
    forces it has alone, bit for bit."""
    gpu = NbodyGpu("0")
    rt = ParallelTreeRuntime(gpu)
    cfg = Config(theta=0.9, softening_kpc=0.01, g=1.0, bucket=3, force_stats=False)
    members, alone = [], []
    for k, n in enumerate((40_001, 2_000_003, 5, 70_000, 32_769)):
        bodies = scenarios.make(("exponential_disc", "cold_disc")[k % 2], n, k, eps=0.01)
        ev, _ = gpu.create_evolving_state(bodies)
        tree = rt.create_tree(gpu, ev, cfg)
        rt.rebuild(gpu, ev, tree, cfg)
        rt.force(gpu, ev, tree, cfg)
        alone.append(gpu.read_evolving_accelerations_f32(ev)[0].view(np.uint32))
        tree.close()
        ev.close()
        members.append(gpu.create_evolving_state(bodies)[0])
    Batch(gpu, members, [cfg] * len(members)).solve()
    for ev, want in zip(members, alone):
        assert np.array_equal(gpu.read_evolving_accelerations_f32(ev)[0].view(np.uint32), want)
