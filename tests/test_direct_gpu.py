"""Direct kernel (short reduce-free programs): lengths around its tiles and granules, every operand kind; chained launches."""
import numpy as np
import pytest

from .util import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float16, np.int32])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 511, 1023, 1024, 1027, 4099, 300001])
def test_lengths(n, dtype):
    rng = np.random.default_rng(n)
    x, y = ((rng.integers(-50, 50, (n,))).astype(dtype) for _ in range(2))
    (dev,), (ref,), _ = run_both(lambda k, a, b: k.add(k.mul(a, b), k.maximum(a, b)), [x, y])
    assert np.array_equal(dev, ref)   # whole numbers: every step is exact


@pytest.mark.parametrize("n", [7, 1025])
def test_operand_kinds(n):
    """Selects, compares, casts, values with several uses, four inputs, two results."""
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(n)
    a, b, c, d = (rng.standard_normal((n,)).astype(np.float32) for _ in range(4))
    t = Tester("vector")
    la, lb, lc, ld = (t.load(v) for v in (a, b, c, d))
    s = t.add(la, lb)
    m = t.greater(s, 0.0)
    r = t.select(m, t.mul(s, lc), t.sub(ld, s))
    st = [t.store(r), t.store(t.cast(r, 4)), t.store(t.cast(m, 4))]
    t.run()
    sv = a + b
    want = np.where(sv > 0, sv * c, d - sv)
    assert np.array_equal(t.output(st[0]), want)
    assert np.array_equal(t.output(st[1]), want.astype(np.int32))
    assert np.array_equal(t.output(st[2]), (sv > 0).astype(np.int32))


def test_chained_launches_see_each_others_results():
    """Kernels back to back on one stream, each reading what the one before wrote: direct, row and interpreter launches in
    turn, without a synchronisation between them."""
    import torch
    import dvm_b200 as dvm
    x = torch.zeros((200, 1024), device="cuda")
    y = torch.zeros_like(x)
    s = torch.zeros((200, 1), device="cuda")
    stream = torch.cuda.Stream()

    def kernel(build, binds):
        k = dvm.PyKernel("vector")
        ops = build(k)
        for op, t in zip(ops, binds):
            k.bind_device(op, t.data_ptr(), t.numel() * 4)
        k.codegen()
        return k

    def plus_one(k):
        a = k.load([200, 1024], dvm.float32)
        return [a, k.store(k.add(a, 1.0))]

    def times_with_mean(k):   # y - mean(y) + mean(y) = y, with the mean stored
        a = k.load([200, 1024], dvm.float32)
        m = k.mul(k.sum(a, (1,), True), 1.0 / 1024)
        return [a, k.store(k.add(k.sub(a, m), m)), k.store(m)]

    def row_max(k):           # (a maximum runs on the interpreter)
        a = k.load([200, 1024], dvm.float32)
        m = k.max(a, (1,), True)
        return [a, k.store(k.add(k.sub(a, m), m)), k.store(m)]

    ks = [kernel(plus_one, (x, y)), kernel(times_with_mean, (y, x, s)), kernel(plus_one, (x, y)), kernel(row_max, (y, x, s))]
    rounds = 100
    torch.cuda.synchronize()
    for _ in range(rounds):
        for k in ks:
            k.launch(stream.cuda_stream)
    torch.cuda.synchronize()
    assert torch.equal(x, torch.full_like(x, 2.0 * rounds))   # (whole numbers below 2^24 in every partial sum)
