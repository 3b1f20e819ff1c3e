"""MatMul tilings: every kernel variant at the edges of its tiles - few rows, a cut contraction, rows at any even address."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BF = 2

# rows, columns, depth: tile edges (64 / 128 columns, 128 rows, 64 of depth), remainders, single rows, odd widths and depths
SIZES = [(1, 64, 64), (1, 8, 8), (33, 72, 64), (97, 136, 200), (128, 128, 128), (129, 257, 65), (102, 600, 472), (64, 63, 1), (7, 1000, 1031),
         (300, 513, 511), (16, 2056, 1024), (260, 130, 72)]
FORMS = ["gelu", "plain", "trans_a", "trans_b", "interpreted"]


def _check(m, n, k, form, seed):
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(seed)
    bf = lambda x: Tester.convert_from_bf16(Tester.convert_to_bf16(x))
    a = bf(rng.standard_normal((m, k)).astype(np.float32))
    b = bf(rng.standard_normal((k, n)).astype(np.float32) * (1.0 / np.sqrt(k)))
    bias = bf(rng.standard_normal((n,)).astype(np.float32))
    t = Tester("mix")
    la = t.load(np.ascontiguousarray(a.T) if form == "trans_a" else a, "bfloat16")
    lb = t.load(np.ascontiguousarray(b.T) if form == "trans_b" else b, "bfloat16")
    want = a.astype(np.float64) @ b.astype(np.float64)
    if form == "gelu":
        c = t.matmul(la, lb, False, False, t.load(bias, "bfloat16"))
        s = t.store(t.cast(W.gelu_tanh(t, t.cast(c, 3)), BF))
        x = want + bias
        want = x / (1 + np.exp(-2 * np.sqrt(2 / np.pi) * (x + 0.044715 * x ** 3)))
    elif form == "interpreted":   # a post-fusion program the kernels have no form of their own for, fp32 result
        c = t.matmul(la, lb, False, False)
        s = t.store(t.mul(t.cast(c, 3), t.load(bias.reshape(1, n))))
        want = want * bias
    else:
        s = t.store(t.matmul(la, lb, form == "trans_a", form == "trans_b"))
    t.run()
    got = Tester.convert_from_bf16(t.output(s)) if s.dtype() == BF else t.output(s)
    # one rounding of the product to bf16 (2^-9 of it), one of the result, and fp32 sums of k terms of size about 1 / sqrt(k)
    bound = 2.0 ** -8 * (np.abs(want) + 1.0) * (2.0 if form in ("gelu", "interpreted") else 1.0)
    if form == "interpreted":
        bound = bound * np.maximum(np.abs(bias), 1.0)
    assert np.all(np.abs(got - want) <= bound), (m, n, k, form, float(np.max(np.abs(got - want) - bound)))


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m,n,k", SIZES)
def test_sizes(m, n, k, form):
    _check(m, n, k, form, m + 7 * n + 13 * k)


@pytest.mark.parametrize("plan", ["0,1", "64,1", "64,2", "64,8", "128,1", "128,4"])
def test_every_tiling(plan):
    """The same sizes through one forced tiling (the switch is read once per process)."""
    code = ("import sys; sys.path.insert(0, '.')\nfrom tests.test_matmul_tiles_gpu import SIZES, FORMS, _check\n"
            "for i, (m, n, k) in enumerate(SIZES):\n    for form in FORMS: _check(m, n, k, form, i)\n")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, DVM_B200_MM_PLAN=plan), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
