"""The engine's host side (bh_engine.cu) on a CPU: compiled as C++ against a fake
CUDA runtime (fake_cuda.cpp), so that failing calls, error words and threads can
be tried without a GPU."""
import ctypes as C
import os
import subprocess
import threading

import numpy as np
import pytest

from galaxy_b200 import _lib, build
from galaxy_b200.nbody_gpu import Config

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libhost.so")
    include = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    # (-Bsymbolic: its own runtime, whatever other one the process has loaded)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-pthread",
                    "-Wl,-Bsymbolic", "-I" + include,
                    "-x", "c++", os.path.join(build.CSRC, "bh_engine.cu"),
                    os.path.join(HERE, "fake_cuda.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    for name, (res, args) in _lib.SIGNATURES.items():
        if hasattr(lib, name):
            fn = getattr(lib, name)
            fn.restype, fn.argtypes = res, args
    lib.fake_pin.argtypes, lib.fake_unpin.argtypes = [C.c_void_p, C.c_size_t], [C.c_void_p]
    return lib


@pytest.fixture
def device(fake):
    fake.fake_reset()
    dev = C.c_void_p()
    assert fake.galaxy_bh_device_open(0, C.byref(dev)) == _lib.BH_OK
    yield dev
    fake.fake_reset()
    fake.galaxy_bh_device_close(dev)


def new_state(fake, dev, records):
    st = C.c_void_p()
    assert fake.galaxy_bh_state_create(dev, _lib.ptr(records), len(records), C.byref(st),
                                       None) == _lib.BH_OK
    return st


def test_two_threads_on_one_handle_read_their_own_states(fake, device):
    """Large pageable arrays go through the handle's pinned slots: two threads
    that read two states at once through one handle each get their own."""
    n = (16 << 20) // 32 + 5
    records = [np.zeros((n, 8), np.float32) for _ in range(2)]
    for k, r in enumerate(records):
        r[:] = 1.0 + k + np.arange(n, dtype=np.float32)[:, None] / n
    states = [new_state(fake, device, r) for r in records]
    wrong = [0, 0]

    def read(k):
        out = np.empty_like(records[k])
        for _ in range(6):
            assert fake.galaxy_bh_read_state(device, states[k], _lib.ptr(out), n, None) == 0
            wrong[k] += not np.array_equal(out, records[k])

    threads = [threading.Thread(target=read, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for st in states:
        fake.galaxy_bh_state_destroy(st)
    assert wrong == [0, 0]


def test_a_failed_rebuild_or_step_leaves_no_tree_to_use(fake, device):
    """After a rebuild or a step that ended in an error the cells are not those of
    the sums and codes beside them: nothing walks them until a rebuild succeeds."""
    records = np.ones((100, 8), np.float32)
    st, tree, cfg = new_state(fake, device, records), C.c_void_p(), C.byref(Config().to_c())
    assert fake.galaxy_bh_tree_create(device, st, cfg, C.byref(tree)) == _lib.BH_OK
    accel = np.zeros((100, 2))

    def uses():
        return [fake.galaxy_bh_force(device, st, tree, cfg, None),
                fake.galaxy_bh_force_f64(device, st, tree, cfg, _lib.ptr(accel), None, None),
                fake.galaxy_bh_read_tree_evidence(device, tree, None, None, None, 0, None, 0, None),
                fake.galaxy_bh_step(device, st, tree, cfg, 1e-3, 1)]

    for fail in (lambda: fake.galaxy_bh_tree_rebuild(device, st, tree, cfg, None),
                 lambda: fake.galaxy_bh_step(device, st, tree, cfg, 1e-3, 1)):
        assert fake.galaxy_bh_tree_rebuild(device, st, tree, cfg, None) == _lib.BH_OK
        assert uses() == [_lib.BH_OK] * 4
        fake.fake_rebuild_error(1)  # the sort's wait gave up
        assert fail() == _lib.BH_TIMEOUT
        fake.fake_rebuild_error(0)
        assert uses() == [_lib.BH_INVALID_ARG] * 4
    fake.galaxy_bh_tree_destroy(tree)
    fake.galaxy_bh_state_destroy(st)


@pytest.mark.parametrize("bits,status", [(8, _lib.BH_CAPACITY_OVERFLOW), (16, _lib.BH_INVALID_ARG)])
def test_a_refused_packed_tree_leaves_the_output_alone(fake, device, bits, status):
    """A walk that meets its stack's end or an index out of range gives no result."""
    n = 40
    settings = np.zeros(1, _lib.BH_SETTINGS_DTYPE)
    settings["info"][0, 0] = n
    bodies, entries = np.zeros(n, _lib.GPU_BODY_DTYPE), np.zeros(n, _lib.GPU_ENTRY_DTYPE)
    cells, out = np.zeros(3, _lib.GPU_CELL_DTYPE), np.full((n, 4), 7.0, np.float32)

    def traverse():
        return fake.galaxy_bh_traverse_packed(device, _lib.ptr(settings), _lib.ptr(bodies), n,
                                              _lib.ptr(entries), _lib.ptr(cells), len(cells),
                                              _lib.ptr(out), None)

    fake.fake_packed_error(bits)
    assert traverse() == status
    assert (out == 7.0).all()
    fake.fake_packed_error(0)
    assert traverse() == _lib.BH_OK
    assert (out == 0.0).all()


@pytest.mark.parametrize("name", ["packed", "into", "evidence", "f64", "probes"])
def test_a_call_that_fails_leaves_no_transfer_behind(fake, device, name):
    """Whichever CUDA call fails in one that takes device memory for its own length,
    it returns with nothing queued that still reads or writes the caller's pinned
    arrays."""
    n, cfg = 64, Config().to_c()
    st, tree, p = new_state(fake, device, np.ones((n, 8), np.float32)), C.c_void_p(), _lib.ptr
    assert fake.galaxy_bh_tree_create(device, st, C.byref(cfg), C.byref(tree)) == _lib.BH_OK
    assert fake.galaxy_bh_tree_rebuild(device, st, tree, C.byref(cfg), None) == _lib.BH_OK
    settings = np.zeros(1, _lib.BH_SETTINGS_DTYPE)
    settings["info"][0, 0] = n
    bodies, entries = np.zeros(n, _lib.GPU_BODY_DTYPE), np.zeros(n, _lib.GPU_ENTRY_DTYPE)
    cells, accel = np.zeros(n, _lib.GPU_CELL_DTYPE), np.zeros((n, 4), np.float32)
    f64, abs_sum, probes = np.zeros((n, 2)), np.zeros(n), np.arange(n, dtype=np.uint32)
    call = {
        "packed": lambda: fake.galaxy_bh_traverse_packed(
            device, p(settings), p(bodies), n, p(entries), p(cells), n, p(accel), None),
        "into": lambda: fake.galaxy_bh_force_into(
            device, st, p(settings), p(bodies), p(entries), p(cells), n, None),
        "evidence": lambda: fake.galaxy_bh_read_tree_evidence(
            device, tree, None, p(entries), p(bodies), n, p(cells), n, None),
        "f64": lambda: fake.galaxy_bh_force_f64(device, st, tree, C.byref(cfg), p(f64),
                                                p(abs_sum), None),
        "probes": lambda: fake.galaxy_bh_direct_probes(device, st, C.byref(cfg), p(probes), n,
                                                       p(f64)),
    }[name]
    arrays = [settings, bodies, entries, cells, accel, f64, abs_sum, probes]
    for a in arrays:
        fake.fake_pin(a.ctypes.data, a.nbytes)
    assert (call(), fake.fake_transfers()) == (_lib.BH_OK, 0)
    seen = []  # status and transfers left, by the call that failed
    fake.fake_fail_after(0)
    while True:
        got = (call(), fake.fake_transfers())
        if not fake.fake_failed():  # there are no more
            break
        seen.append(got)
        fake.fake_fail_after(len(seen))
    for a in arrays:
        fake.fake_unpin(a.ctypes.data)
    fake.galaxy_bh_tree_destroy(tree)
    fake.galaxy_bh_state_destroy(st)
    assert got == (_lib.BH_OK, 0)
    assert len(seen) >= 3 and seen == [(_lib.BH_CUDA_ERROR, 0)] * len(seen)
