"""Vector stages whose ring holds a tensor that ends inside a 16-byte unit, behind four valid elements of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,code", [("bfloat16", 2), ("float16", 1), ("float32", 3)])
@pytest.mark.parametrize("rows,cols", [(3, 1870), (7, 1871), (2, 4093), (5, 1868), (3, 1866), (1, 14), (2, 20)])
def test_broadcast_row_behind_a_reduction(rows, cols, dtype, code):
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(rows + cols)
    def rounded(x):
        x = x.astype(np.float32)
        if dtype == "bfloat16":
            return Tester.convert_from_bf16(Tester.convert_to_bf16(x))
        return x.astype(np.float16).astype(np.float32) if dtype == "float16" else x
    x, w = rounded(rng.uniform(0.5, 2.0, (rows, cols))), rounded(rng.uniform(0.5, 2.0, (1, cols)))
    t = Tester("vector")
    f = lambda v: t.cast(v, 3) if code != 3 else v
    lx, lw = f(t.load(x, dtype)), f(t.load(w, dtype))
    m = t.max(lx, (-1,), True)
    y = t.mul(t.sub(lx, m), lw)
    st = t.store(t.cast(y, code) if code != 3 else y)
    t.run()
    got = t.output(st)
    got = Tester.convert_from_bf16(got) if dtype == "bfloat16" else got.astype(np.float32)
    want = (x - x.max(-1, keepdims=True)) * w
    # the difference and the product are rounded to fp32 once each, the result to the stored type
    unit = {"bfloat16": 2.0 ** -8, "float16": 2.0 ** -11, "float32": 2.0 ** -23}[dtype]
    assert np.all(np.abs(got - want) <= 2.0 * unit * np.abs(want) + 2.0 ** -24)
