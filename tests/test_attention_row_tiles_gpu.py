"""Prefill attention around its tiles: warps of 16 rows, halves of 64 keys, score buffers used in turn; a maximum that rises with every
key tile in some rows only, so that accumulators are rescaled while P V of the tile before is in flight; scales of either sign behind
the cast."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one row tile per CTA and two (more than 148 tiles of 128 rows), rows and keys one off the edges of 16, 64 and 128
@pytest.mark.parametrize("batch,sq,skv", [(1, 17, 63), (1, 31, 64), (2, 33, 65), (1, 113, 127), (1, 128, 385), (1, 129, 640), (80, 143, 191), (75, 256, 513)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("scale,scale_first", [(0.125, True), (0.125, False), (-0.125, False), (0.0, False)])
def test_rising_maxima(batch, sq, skv, d, scale, scale_first):
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(batch + sq + skv + d)
    # whole numbers and a scale of 1 / 8: every score is exact in fp16, before and after the scale
    q, k = (rng.integers(-1, 2, (batch, 1, s, d)).astype(np.float16) for s in (sq, skv))
    v = rng.standard_normal((batch, 1, skv, d)).astype(np.float16)
    # rows 5 of every 16 see scores that grow by more than 8 from key tile to key tile
    q[:, :, 5::16, 0] = np.float16(8.0 * (1.0 if scale >= 0 else -1.0))
    k[:, :, :, 0] = (np.arange(skv) // 64 * 9.0).astype(np.float16)
    t = Tester("split")
    ops = [t.load(x) for x in (q, k, v)]
    if scale_first:
        st = t.store(W.attention(t, *ops, scale, 1))
    else:
        s = t.mul(t.cast(t.matmul(ops[0], ops[1], False, True), 3), scale)
        e = t.exp(t.sub(s, t.max(s, (-1,), True)))
        st = t.store(t.matmul(t.cast(t.div(e, t.sum(e, (-1,), True)), 1), ops[2], False, False))
    t.run()
    got = t.output(st).astype(np.float64)
    s = q.astype(np.float64) @ np.swapaxes(k.astype(np.float64), -1, -2) * scale
    p = np.exp(s - s.max(-1, keepdims=True))
    want = p @ v.astype(np.float64) / p.sum(-1, keepdims=True)
    # every p is rounded once (below 2 ** -14 to a multiple of 2 ** -24; the largest of a row is at least 1) and the result once
    l, size = p.sum(-1, keepdims=True), np.abs(v.astype(np.float64))
    bound = 2.0 ** -11 * (p @ size / l + np.abs(want)) * 1.01 + 2.0 ** -25 * size.sum(-2, keepdims=True) / l + 2.0 ** -25
    assert np.all(np.abs(got - want) <= bound), float((np.abs(got - want) - bound).max())


# one row tile per CTA and two
@pytest.mark.parametrize("sq", [128, 149 * 128])
def test_row_sums_of_many_keys(sq):
    """2 ** 19 keys, all but the first with the same weight: a running fp32 sum that takes them one by one rounds in the same direction
    every time, by up to 2 ** 16 / 2 units of 2 ** -24 over the lanes; sums per key tile leave 4096 such additions."""
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    keys, d = 1 << 19, 64
    score = np.tile(0.25 + 0.1171875 * np.arange(64), sq // 64)   # of the first key; 0 for the others
    q, k, v = np.zeros((1, 1, sq, d), np.float16), np.zeros((1, 1, keys, d), np.float16), np.zeros((1, 1, keys, d), np.float16)
    q[0, 0, :, 0] = 8.0 * score
    k[0, 0, 0, 0], v[0, 0, 0] = 1.0, 32768.0   # (only the first key has values: the result is 32768 over the row's sum)
    t = Tester("split")
    st = t.store(W.attention(t, *[t.load(x) for x in (q, k, v)], 0.125, 1))
    t.run()
    want = (32768.0 / (1.0 + (keys - 1) * np.exp(-score)))[None, None, :, None]
    # the result's rounding, and 4096 additions of half a unit each
    off = np.abs(t.output(st).astype(np.float64) / want - 1.0)
    assert np.all(off <= 2.0 ** -11 + 4096 * 2.0 ** -25), float(off.max() * 2.0 ** 11)
