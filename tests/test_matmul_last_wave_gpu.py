"""MatMul in tiles of CTA pairs whose last wave is not full: its tiles are worked on as halves of 128 columns."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# 148 SMs hold 74 pairs: 80 tiles (the last columns in the first half, and in the second), 75 (one tile in two halves), 85, 111
# (the most that fit as halves) and 112 (none); fewer tiles than half a wave are in test_matmul_tiles_gpu.py
SIZES = [(1024, 5003, 200), (1024, 4888, 72), (768, 6400, 64), (1100, 4304, 136), (768, 9472, 64), (1792, 4096, 64)]


def test_last_wave():
    code = ("import sys; sys.path.insert(0, '.')\nfrom tests.test_matmul_tiles_gpu import FORMS, _check\n"
            "for i, (m, n, k) in enumerate(%r):\n    for form in FORMS: _check(m, n, k, form, i)\n" % (SIZES,))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, DVM_B200_MM_PLAN="0,1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
