"""Copies between pageable arrays and the device: sizes around the staged path's chunks and ring, several threads at once."""
import subprocess
import sys
import threading

import numpy as np
import pytest

from dvm_b200 import _capi

pytestmark = pytest.mark.gpu

PART, CHUNK, RING = 64 * 1024, 1024 * 1024, 8 * 1024 * 1024


@pytest.fixture(autouse=True)
def ring():
    """The ring is set up once enough has been copied without it."""
    lib = _capi.load()
    assert lib.dvm_rt_set_device(0) == 0
    src = np.zeros(4 * RING + 1, np.uint8)
    d = lib.dvm_rt_malloc(src.size)
    assert lib.dvm_rt_memcpy_h2d(d, src.ctypes.data, src.size, None) == 0 and lib.dvm_rt_sync(None) == 0 and lib.dvm_rt_free(d) == 0


def _round_trip(lib, n, seed):
    src = np.random.default_rng(seed).integers(0, 256, n, dtype=np.uint8)
    dst = np.zeros(n + 1, np.uint8)
    d = lib.dvm_rt_malloc(n)
    for _ in range(2):
        assert lib.dvm_rt_memcpy_h2d(d, src.ctypes.data, n, None) == 0
        # (the source may be reused as soon as the call returns)
        keep = src.copy()
        src[:] = 0
        assert lib.dvm_rt_memcpy_d2h(dst[1:].ctypes.data, d, n, None) == 0   # (an odd host address)
        assert lib.dvm_rt_sync(None) == 0
        src[:] = keep
        assert np.array_equal(dst[1:], src)
        dst[:] = 0
    assert lib.dvm_rt_free(d) == 0


@pytest.mark.parametrize("n", [1, 32 * 1024 - 1, 32 * 1024, PART - 1, PART, PART + 1, 4 * PART + 3, CHUNK - 1, CHUNK, CHUNK + 1, RING - 5, RING, RING + 1, 3 * RING + 12345])
def test_sizes(n):
    lib = _capi.load()
    assert lib.dvm_rt_set_device(0) == 0
    _round_trip(lib, n, n)


def test_threads():
    lib = _capi.load()
    errors = []

    def work(i):
        try:
            assert lib.dvm_rt_set_device(0) == 0
            for j in range(4):
                _round_trip(lib, 700_000 + 300_000 * i + j, 10 * i + j)
        except Exception as e:   # (an assertion in a thread must fail the test)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_copies_beside_a_stream_capture():
    """A thread that copies does not break the capture of another one, and is not broken by it."""
    import torch
    import dvm_b200 as dvm
    lib = _capi.load()
    assert lib.dvm_rt_set_device(0) == 0
    x, y = torch.arange(4096.0, device="cuda"), torch.zeros(4096, device="cuda")
    k = dvm.PyKernel("vector")
    a = k.load([4096], dvm.float32)
    s = k.store(k.add(a, 1.0))
    for op, t in ((a, x), (s, y)):
        k.bind_device(op, t.data_ptr(), t.numel() * 4)
    k.codegen()
    k.launch(torch.cuda.current_stream().cuda_stream)
    n = 4 * CHUNK + 77
    src, dst = np.random.default_rng(9).integers(0, 256, n, dtype=np.uint8), np.zeros(n, np.uint8)
    dev, own = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.cuda.Stream()
    torch.cuda.synchronize()
    rcs = []

    def copy():
        assert lib.dvm_rt_set_device(0) == 0
        for _ in range(3):
            rcs.append(lib.dvm_rt_memcpy_h2d(dev.data_ptr(), src.ctypes.data, n, own.cuda_stream))
            rcs.append(lib.dvm_rt_memcpy_d2h(dst.ctypes.data, dev.data_ptr(), n, own.cuda_stream))

    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):   # (the default mode: unsafe calls of any thread are refused)
        k.launch(stream.cuda_stream)
        t = threading.Thread(target=copy)
        t.start()
        t.join()
    own.synchronize()
    assert rcs == [0] * 6 and np.array_equal(src, dst)
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, x + 1.0)


def test_system_without_threads():
    """Where no worker thread can be created the copy takes the driver's path; the caller, behind a C entry, sees no exception."""
    code = """
import resource
import numpy as np
from dvm_b200 import _capi
lib = _capi.load()
n = 40 << 20
src = np.arange(n, dtype=np.uint8)
assert lib.dvm_rt_set_device(0) == 0
d = lib.dvm_rt_malloc(n)
assert lib.dvm_rt_memcpy_h2d(d, src.ctypes.data, 64, None) == 0 and lib.dvm_rt_sync(None) == 0
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (1 << 20), resource.RLIM_INFINITY))   # (less than a thread's stack)
rc = lib.dvm_rt_memcpy_h2d(d, src.ctypes.data, n, None)
resource.setrlimit(resource.RLIMIT_AS, (resource.RLIM_INFINITY, resource.RLIM_INFINITY))
assert rc in (0, 2), rc   # (the driver may need memory of its own: an error, no abort)
print("DONE")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "DONE" in r.stdout, (r.returncode, r.stderr[-2000:])


def test_copies_before_the_ring_is_worth_it():
    """In a process of its own: arrays copied by the driver's path, then the one that has the ring set up, then through it."""
    code = """
import numpy as np
from dvm_b200 import _capi
lib = _capi.load()
assert lib.dvm_rt_set_device(0) == 0
for i, n in enumerate([40_000, 4_000_001, 9_000_000, 3_000_000, 5_000_000, 64 * 1024, 20_000_003]):
    src, dst = np.random.default_rng(i).integers(0, 256, n, dtype=np.uint8), np.zeros(n, np.uint8)
    d = lib.dvm_rt_malloc(n)
    assert lib.dvm_rt_memcpy_h2d(d, src.ctypes.data, n, None) == 0 and lib.dvm_rt_memcpy_d2h(dst.ctypes.data, d, n, None) == 0
    assert lib.dvm_rt_sync(None) == 0 and lib.dvm_rt_free(d) == 0
    assert np.array_equal(src, dst), n
print("DONE")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "DONE" in r.stdout, (r.returncode, r.stderr[-2000:])
