"""Attention of more query rows than one wave of CTAs holds: a CTA computes several units, one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("batch,heads,sq,skv", [(1, 2, 300, 1), (4, 40, 130, 100), (10, 31, 17, 129), (25, 13, 128, 257), (2, 80, 511, 300)])
def test_units(batch, heads, sq, skv, d, dtype):
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    code = {"bfloat16": 2, "float16": 1}[dtype]
    rng = np.random.default_rng(batch + heads + 3 * sq + 7 * skv + d)
    def rounded(x):
        x = x.astype(np.float32)
        return Tester.convert_from_bf16(Tester.convert_to_bf16(x)) if dtype == "bfloat16" else x.astype(np.float16).astype(np.float32)
    q, k, v = (rounded(rng.standard_normal((batch, heads, s, d))) for s in (sq, skv, skv))
    k[0, 0, skv // 2] = rounded(k[0, 0, skv // 2] * 6.0)   # a late, large score: the running maximum moves
    t = Tester("split")
    ops = [t.load(x, dtype) for x in (q, k, v)]
    st = t.store(W.attention(t, *ops, 1.0 / np.sqrt(d), code))
    t.run()
    got = t.output(st)
    got = Tester.convert_from_bf16(got) if dtype == "bfloat16" else got.astype(np.float32)
    unit = 2.0 ** -8 if dtype == "bfloat16" else 2.0 ** -11
    s = q @ np.swapaxes(k, -1, -2) / np.sqrt(np.float32(d))
    p = np.exp(s - s.max(-1, keepdims=True))
    want = p @ v / p.sum(-1, keepdims=True)
    # a score of size |s| is rounded twice (relative error of p: 2 |s| unit), p and the result once each; the fp32 of this
    # oracle adds far less than one of these
    bound = unit * (2.0 * np.abs(s).max(-1, keepdims=True) + 2.0) * np.abs(v).max()
    assert np.all(np.abs(got - want) <= bound), float((np.abs(got - want) - bound).max())
