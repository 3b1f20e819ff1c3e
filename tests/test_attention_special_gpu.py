"""Attention with scores that overflow to -inf and with NaN: in the first keys of a warp, of a key tile, of all of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (the 256-row kernel works on 128 keys at a time; a decode warp on 16 or 32 of its share of the keys)
SHAPES = [(1, 64, 128), (4, 700, 64), (16, 700, 128), (1, 8192, 64), (40, 300, 64), (130, 700, 128), (300, 500, 64)]


def _attention(q, k, v, scale, scale_first):
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    t = Tester("split")
    ops = [t.load(x) for x in (q, k, v)]
    if scale_first:
        st = t.store(W.attention(t, *ops, scale, 1))
    else:
        s = t.mul(t.cast(t.matmul(ops[0], ops[1], False, True), 3), scale)
        e = t.exp(t.sub(s, t.max(s, (-1,), True)))
        st = t.store(t.matmul(t.cast(t.div(e, t.sum(e, (-1,), True)), 1), ops[2], False, False))
    t.run()
    return t.output(st).astype(np.float64)


@pytest.mark.parametrize("scale_first", [True, False])
@pytest.mark.parametrize("sq,skv,d", SHAPES)
@pytest.mark.parametrize("where", ["first", "all_but_last", "every_other_block", "all"])
def test_scores_of_minus_infinity(sq, skv, d, where, scale_first):
    rng = np.random.default_rng(sq + skv + d)
    q = np.abs(rng.standard_normal((2, 1, sq, d))).astype(np.float16) + np.float16(1)
    k, v = (rng.standard_normal((2, 1, skv, d)).astype(np.float16) for _ in range(2))
    hidden = np.zeros(skv, bool)
    hidden[{"first": slice(0, skv // 2), "all_but_last": slice(0, skv - 1), "every_other_block": slice(0, 0), "all": slice(None)}[where]] = True
    if where == "every_other_block":
        hidden[:] = np.arange(skv) // 16 % 2 == 0
    k[0, 0, hidden] = -60000.0   # (the score, -60000 d and less, is -inf in fp16)
    with np.errstate(all="ignore"):
        s = (q.astype(np.float64) @ np.swapaxes(k.astype(np.float64), -1, -2))
        s = np.where(s < -65520.0, -np.inf, s) / np.sqrt(d)
        p = np.exp(s - s.max(-1, keepdims=True))
        want = p @ v.astype(np.float64) / p.sum(-1, keepdims=True)
    got = _attention(q, k, v, 1.0 / np.sqrt(d), scale_first)
    assert np.array_equal(np.isnan(got), np.isnan(want))   # (where every score is -inf the graph's own result is NaN)
    ok = ~np.isnan(want)
    # a score of size |s| is rounded twice (relative error of p: 2 |s| unit), p and the result once each
    largest = np.where(np.isfinite(s), np.abs(s), 0.0).max()
    assert np.all(np.abs(got[ok] - want[ok]) <= 2.0 ** -11 * (2.0 * largest + 2.0) * float(np.abs(v).max()))


@pytest.mark.parametrize("scale_first", [True, False])
@pytest.mark.parametrize("sq,skv,d", SHAPES)
@pytest.mark.parametrize("count", [1, 16, 128])
def test_nan_reaches_the_result(sq, skv, d, count, scale_first):
    """A NaN score makes its row's sum, and so every element of the row's result, NaN - also where it is all that a warp sees."""
    rng = np.random.default_rng(sq + skv + d)
    q, k, v = (rng.standard_normal((2, 1, s, d)).astype(np.float16) for s in (sq, skv, skv))
    at = skv // 2 // 16 * 16
    k[1, 0, at:at + count] = np.nan
    got = _attention(q, k, v, 1.0 / np.sqrt(d), scale_first)
    assert np.all(np.isnan(got[1])) and not np.any(np.isnan(got[0]))
