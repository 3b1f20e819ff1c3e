"""Attention of a few query rows against a key/value cache: every split of the keys over warps and CTAs, and its edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("batch,heads,sq,skv", [(1, 1, 1, 1), (1, 2, 3, 15), (2, 2, 1, 17), (1, 3, 16, 64), (1, 4, 8, 129), (1, 1, 9, 2047),
                                                (2, 8, 1, 515), (1, 2, 2, 4111), (5, 30, 1, 200), (20, 32, 1, 1100)])
def test_decode(batch, heads, sq, skv, d, dtype):
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    code = {"bfloat16": 2, "float16": 1}[dtype]
    rng = np.random.default_rng(batch + heads + 3 * sq + 7 * skv + d)
    def data(s):
        x = rng.standard_normal((batch, heads, s, d)).astype(np.float32)
        return Tester.convert_from_bf16(Tester.convert_to_bf16(x)) if dtype == "bfloat16" else x.astype(np.float16).astype(np.float32)
    q, k, v = data(sq), data(skv), data(skv)
    k[0, 0, skv // 2] *= 6.0   # a late, large score: the running maximum moves
    t = Tester("split")
    ops = [t.load(x, dtype) for x in (q, k, v)]
    st = t.store(W.attention(t, *ops, 1.0 / np.sqrt(d), code))
    t.run()
    got = t.output(st)
    got = Tester.convert_from_bf16(got) if dtype == "bfloat16" else got.astype(np.float32)
    unit = 2.0 ** -8 if dtype == "bfloat16" else 2.0 ** -11
    kd = (Tester.convert_from_bf16(Tester.convert_to_bf16(k)) if dtype == "bfloat16" else k.astype(np.float16)).astype(np.float64)
    s = q.astype(np.float64) @ np.swapaxes(kd, -1, -2) / np.sqrt(d)
    p = np.exp(s - s.max(-1, keepdims=True))
    want = p @ v.astype(np.float64) / p.sum(-1, keepdims=True)
    # a score of size |s| is rounded twice (relative error of p: 2 |s| unit), p and the result once each
    bound = unit * (2.0 * np.abs(s).max(-1, keepdims=True) + 2.0) * np.abs(v).max()
    assert np.all(np.abs(got - want) <= bound), float((np.abs(got - want) - bound).max())
