"""Normalisations over runs of any length and alignment, on the row kernel and on the interpreter, against float64."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batchnorm(shape, dtype, offset=0):
    """Training batch-norm of an NCHW tensor that starts `offset` elements into its buffer; float64 expectation."""
    from dvm_b200 import workloads as W
    from dvm_b200.tester import Tester
    n, c, h, w = shape
    rng = np.random.default_rng(n + 3 * c + 7 * h + 11 * w)
    raw = (rng.standard_normal(shape) + rng.standard_normal((1, c, 1, 1))).astype(np.float32)
    x = Tester.convert_to_bf16(raw) if dtype == "bfloat16" else raw.astype(dtype)
    g = rng.normal(1, 0.1, (1, c, 1, 1)).astype(np.float32)
    b = rng.normal(0, 0.1, (1, c, 1, 1)).astype(np.float32)
    code = {"float16": 1, "bfloat16": 2, "float32": 3}[dtype]
    t = Tester("vector")
    if offset:
        buf = np.zeros(x.size + offset, x.dtype)
        buf[offset:] = x.reshape(-1)
        lx = t.view_load(list(shape), [c * h * w, h * w, w, 1], buf, offset)
    else:
        lx = t.load(x, dtype)
    f = lx if code == 3 else t.cast(lx, 3)
    count = 1.0 / (n * h * w)
    if code == 3:   # (the sums as they are: deviations are for 16-bit inputs)
        mean = t.mul(t.sum(f, (0, 2, 3), True), count)
        var = t.sub(t.mul(t.sum(t.mul(f, f), (0, 2, 3), True), count), t.mul(mean, mean))
        y = t.add(t.mul(t.mul(t.sub(f, mean), t.div(1.0, t.sqrt(t.add(var, 1e-5)))), t.load(g)), t.load(b))
        stores = [t.store(v) for v in (y, mean, var)]
    elif code == 2:
        mean = t.mul(t.sum(f, (0, 2, 3), True), count)
        xc = t.sub(f, mean)
        var = t.mul(t.sum(t.mul(xc, xc), (0, 2, 3), True), count)
        y = t.add(t.mul(t.div(xc, t.sqrt(t.add(var, 1e-5))), t.load(g)), t.load(b))
        stores = [t.store(v) for v in (t.cast(y, 2), mean, var)]
    else:
        stores = [t.store(v) for v in W.batchnorm_train(t, lx, t.load(g), t.load(b), n * h * w)]
    t.run()
    assert "kernel=row" not in t.das()   # (statistics do not run on the kernel of RMS norms)
    read = lambda s: Tester.convert_from_bf16(t.output(s)) if s.dtype() == 2 else t.output(s)
    got = [read(s).astype(np.float64) for s in stores]
    xd = (Tester.convert_from_bf16(x) if code == 2 else x).astype(np.float64)
    m = xd.mean((0, 2, 3), keepdims=True)
    v = ((xd - m) ** 2).mean((0, 2, 3), keepdims=True)
    y = (xd - m) / np.sqrt(v + 1e-5) * g + b
    # fp32 sums over the group in a tree, one rounding of the result to its type; the plain fp32 sums of squares give the
    # variance as a difference, off by a few 2^-24 of the mean square
    square = float((xd * xd).mean((0, 2, 3)).max())
    assert np.allclose(got[1], m, rtol=1e-5, atol=1e-5 * float(np.abs(xd).max()))
    assert np.allclose(got[2], v, rtol=1e-4, atol=1e-6 if code != 3 else 1e-6 + 2.0 ** -20 * square)
    slack = 1e-3 if code != 3 else 1e-3 + 2.0 ** -21 * square / float((v + 1e-5).min()) * float(np.abs(y).max() + 1.0)
    assert np.all(np.abs(got[0] - y) <= {1: 2.0 ** -10, 2: 2.0 ** -8, 3: 2.0 ** -20}[code] * np.abs(y) + slack), float(np.abs(got[0] - y).max())


# planes of one 16-byte unit and less, odd planes, runs that end on a unit, short groups and long ones
@pytest.mark.parametrize("dtype", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("shape", [(4, 5, 1, 3), (2, 3, 4, 2), (9, 17, 7, 7), (3, 300, 5, 5), (16, 20, 16, 16), (8, 6, 41, 43),
                                   (32, 4, 57, 55), (12, 3, 112, 111), (64, 2, 64, 64), (1, 4, 200, 203)])
def test_batchnorm_planes(shape, dtype):
    _batchnorm(shape, dtype)


@pytest.mark.parametrize("offset", [1, 3, 8])
def test_batchnorm_input_at_any_address(offset):
    _batchnorm((6, 5, 9, 9), "float16", offset)


@pytest.mark.parametrize("residual,weight,gate", [(1, 1, 1), (0, 1, 0), (1, 0, 0), (0, 0, 1)])
@pytest.mark.parametrize("tokens,hidden", [(1, 8), (3, 65), (5, 255), (2, 515), (7, 1024), (130, 1031), (1, 4097), (3, 8185), (600, 700)])
def test_rmsnorm_rows(tokens, hidden, residual, weight, gate):
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(tokens * 31 + hidden)
    bf = lambda x: Tester.convert_from_bf16(Tester.convert_to_bf16(x.astype(np.float32)))
    h, r, g, u = (bf(rng.standard_normal((tokens, hidden))) for _ in range(4))
    w = bf(rng.normal(1, 0.1, (hidden,)))
    t = Tester("vector")
    s = t.cast(t.load(h, "bfloat16"), 3)
    sd = h.astype(np.float64)
    if residual:
        s = t.add(s, t.cast(t.load(r, "bfloat16"), 3))
        sd = sd + r
    ss = t.sum(t.mul(s, s), (1,), True)
    y = t.mul(s, t.div(1.0, t.sqrt(t.add(t.mul(ss, 1.0 / hidden), 1e-6))))
    want = sd / np.sqrt((sd * sd).mean(1, keepdims=True) + 1e-6)
    if weight:
        y = t.mul(y, t.cast(t.load(w, "bfloat16"), 3))
        want = want * w
    stores, wants = [t.store(t.cast(y, 2))], [want]
    if gate:
        gf = t.cast(t.load(g, "bfloat16"), 3)
        sig = t.div(1.0, t.add(t.exp(t.mul(gf, -1.0)), 1.0))
        stores.append(t.store(t.cast(t.mul(t.mul(gf, sig), t.cast(t.load(u, "bfloat16"), 3)), 2)))
        gd = g.astype(np.float64)
        wants.append(gd / (1 + np.exp(-gd)) * u)
    t.run()
    for st, want in zip(stores, wants):
        got = Tester.convert_from_bf16(t.output(st)).astype(np.float64)
        # one rounding to bf16 (2^-9), fp32 arithmetic in front of it
        assert np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-5), float(np.abs(got - want).max())


def test_scalar_sections_of_any_form_run_as_words():
    """Statistics whose scalar sections are not the usual closed form (a clamp, several stored scalars)."""
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(5)
    x = rng.standard_normal((37, 1500)).astype(np.float32)
    t = Tester("vector")
    lx = t.load(x)
    s1, s2 = t.sum(lx, (1,), True), t.sum(t.mul(lx, lx), (1,), True)
    a = t.maximum(t.sqrt(t.mul(s2, 1.0 / 1500)), 0.5)
    stores = [t.store(t.mul(t.sub(lx, t.mul(s1, 1.0 / 1500)), a)), t.store(a), t.store(s1)]
    t.run()
    xd = x.astype(np.float64)
    ad = np.maximum(np.sqrt((xd * xd).mean(1, keepdims=True)), 0.5)
    for st, want in zip(stores, [(xd - xd.mean(1, keepdims=True)) * ad, ad, xd.sum(1, keepdims=True)]):
        assert np.allclose(t.output(st), want, rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("stored", [1, 4, 5, 6])
def test_any_number_of_stored_scalars(stored):
    """(the compiler moves up to four stores of group scalars behind the last body; the others stay in front of it)"""
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(stored)
    x = rng.standard_normal((37, 1500)).astype(np.float32)
    t = Tester("vector")
    lx = t.load(x)
    s1, s2 = t.sum(lx, (1,), True), t.sum(t.mul(lx, lx), (1,), True)
    mean, square = t.mul(s1, 1.0 / 1500), t.mul(s2, 1.0 / 1500)
    root = t.sqrt(t.add(square, 0.25))
    scalars = [s1, s2, mean, square, root, t.mul(root, 2.0)][:stored]
    stores = [t.store(t.mul(t.sub(lx, mean), root))] + [t.store(v) for v in scalars]
    t.run()
    xd = x.astype(np.float64)
    d1, d2 = xd.sum(1, keepdims=True), (xd * xd).sum(1, keepdims=True)
    rd = np.sqrt(d2 / 1500 + 0.25)
    wants = [(xd - d1 / 1500) * rd, d1, d2, d1 / 1500, d2 / 1500, rd, 2 * rd]
    for st, want in zip(stores, wants):
        assert np.allclose(t.output(st), want, rtol=1e-5, atol=1e-4)   # (fp32 sums of 1500 terms of size 1)


@pytest.mark.parametrize("shape,dims", [((1300, 64), (1,)), ((2500, 63), (1,)), ((2500, 64), (1,)), ((2500, 500), (1,)), ((2500, 512), (1,)),
                                        ((4, 2100, 3, 3), (0, 2, 3)), ((3, 5100, 2, 2), (0, 2, 3)), ((2, 2100, 5, 5), (0, 2, 3))])
@pytest.mark.parametrize("dtype,code", [("float16", 1), ("bfloat16", 2)])
def test_statistics_of_many_groups(shape, dims, dtype, code):
    """Short and long groups, few and many, in whole granules and not."""
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(len(shape) + shape[-1])
    raw = rng.standard_normal(shape).astype(np.float32)
    x = raw.astype(np.float16) if code == 1 else Tester.convert_to_bf16(raw)
    xd = (x if code == 1 else Tester.convert_from_bf16(x)).astype(np.float64)
    n = float(np.prod([shape[d] for d in dims]))
    t = Tester("vector")
    f = t.cast(t.load(x, dtype), 3)
    d = t.sub(f, t.mul(t.sum(f, dims, True), 1.0 / n))
    st = t.store(t.cast(t.div(d, t.sqrt(t.add(t.mul(t.sum(t.mul(d, d), dims, True), 1.0 / n), 1e-3))), code))
    t.run()
    got = t.output(st)
    got = (got if code == 1 else Tester.convert_from_bf16(got)).astype(np.float64)
    m = xd.mean(dims, keepdims=True)
    want = (xd - m) / np.sqrt(((xd - m) ** 2).mean(dims, keepdims=True) + 1e-3)
    # one rounding of the result; the fp32 sums (deviations from the group's first element) in front of it
    assert np.all(np.abs(got - want) <= {1: 2.0 ** -11, 2: 2.0 ** -8}[code] * np.abs(want) + 1e-4), float(np.abs(got - want).max())


@pytest.mark.parametrize("rows,cols", [(20000, 16), (30000, 24), (30000, 17), (3000, 64), (2000, 6144), (1300, 4608)])
def test_rms_norm_of_many_rows(rows, cols):
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(cols)
    x = Tester.convert_to_bf16(rng.standard_normal((rows, cols)).astype(np.float32))
    t = Tester("vector")
    f = t.cast(t.load(x, "bfloat16"), 3)
    st = t.store(t.cast(t.mul(f, t.div(1.0, t.sqrt(t.add(t.mul(t.sum(t.mul(f, f), (1,), True), 1.0 / cols), 1e-6)))), 2))
    t.run()
    got = Tester.convert_from_bf16(t.output(st)).astype(np.float64)
    xd = Tester.convert_from_bf16(x).astype(np.float64)
    want = xd / np.sqrt((xd * xd).mean(1, keepdims=True) + 1e-6)
    assert np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-5)   # (one rounding to bf16)


# both sides of the rule for 64 or 72 registers: launches that are on the chip at once, CTAs of 128 threads that leave room for the next's
@pytest.mark.parametrize("rows,cols", [(1, 4104), (148, 8192), (149, 8192), (75, 5003), (600, 2048), (1036, 1024), (1038, 520), (1184, 768), (1186, 1017),
                                       (2072, 900), (2074, 1024)])
@pytest.mark.parametrize("dtype,code", [("float16", 1), ("bfloat16", 2)])
def test_rms_norm_with_few_and_many_registers(rows, cols, dtype, code):
    from dvm_b200.tester import Tester
    rng = np.random.default_rng(rows + cols)
    raw = [rng.standard_normal((rows, cols)).astype(np.float32) for _ in range(2)]
    x, r = (v.astype(np.float16) if code == 1 else Tester.convert_to_bf16(v) for v in raw)
    t = Tester("vector")
    f = t.add(t.cast(t.load(x, dtype), 3), t.cast(t.load(r, dtype), 3))
    st = t.store(t.cast(t.mul(f, t.div(1.0, t.sqrt(t.add(t.mul(t.sum(t.mul(f, f), (1,), True), 1.0 / cols), 1e-6)))), code))
    t.run()
    wide = lambda v: (v if code == 1 else Tester.convert_from_bf16(v)).astype(np.float64)
    sd = wide(x) + wide(r)
    want = sd / np.sqrt((sd * sd).mean(1, keepdims=True) + 1e-6)
    # one rounding of the result, fp32 arithmetic in front of it
    assert np.all(np.abs(wide(t.output(st)) - want) <= {1: 2.0 ** -11, 2: 2.0 ** -8}[code] * np.abs(want) + 1e-5)


@pytest.mark.parametrize("rows,cols", [(7, 3), (33, 257), (5, 8)])
def test_other_scalar_sections_run_on_the_interpreter(rows, cols):
    """A sum alone, two group scalars of different types, an immediate factor and a stored 16-bit mean, the result in place of the
    input: an earlier kernel for statistics, since taken out, faulted on [7, 3]."""
    import torch
    import dvm_b200 as dvm
    g = torch.Generator(device="cuda").manual_seed(5)
    buf = torch.randn(rows * cols + 8, generator=g, device="cuda").half()
    gamma, beta = torch.randn(rows, generator=g, device="cuda").half(), torch.randn(rows + 3, generator=g, device="cuda")
    mean = torch.zeros(rows, device="cuda").half()
    k = dvm.PyKernel("vector")
    x, lg, lb = k.load([rows, cols], dvm.float16), k.load([rows, 1], dvm.float16), k.load([rows, 1], dvm.float32)
    f = k.cast(x, dvm.float32)
    m = k.mul(k.sum(f, (1,), True), 1.0 / cols)
    y = k.add(k.mul(k.mul(k.sub(f, m), k.cast(lg, dvm.float32)), 1.5), lb)
    stores = [k.store(k.cast(y, dvm.float16)), k.store(k.cast(m, dvm.float16))]
    for op, t, off in ((x, buf, 8), (lg, gamma, 0), (lb, beta, 3), (stores[0], buf, 8), (stores[1], mean, 0)):
        k.bind_device(op, t.data_ptr() + off * t.element_size(), (t.numel() - off) * t.element_size())
    k.codegen()
    assert "kernel=interpreter" in k.das()
    xd = buf[8:].double().reshape(rows, cols)
    want_mean = xd.mean(1)
    want = (xd - want_mean[:, None]) * gamma.double()[:, None] * 1.5 + beta[3:].double()[:, None]
    k.launch(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    # one rounding to fp16, fp32 sums in front of it
    assert bool(((buf[8:].double().reshape(rows, cols) - want).abs() <= 2.0 ** -11 * want.abs() + 1e-5).all())
    assert bool(((mean.double() - want_mean).abs() <= 2.0 ** -11 * want_mean.abs() + 1e-5).all())
