"""Copies between pageable arrays and the device: sizes around the staged path's chunks and ring, several threads at once."""
import threading

import numpy as np
import pytest

from dvm_b200 import _capi

pytestmark = pytest.mark.gpu

PART, CHUNK, RING = 64 * 1024, 1024 * 1024, 8 * 1024 * 1024


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
