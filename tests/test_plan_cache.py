"""Plans of recent shapes are kept with a kernel: coming back to a shape, a scalar, a reduce axis or a slice bound gives the program that
a new kernel gives, also when more values pass by than plans are kept (16), and with new addresses and a workspace."""
import numpy as np
import pytest

import dvm_b200 as dvm


def _norm(k, ref):
    x = k.load(ref, dvm.float32)
    k.store(k.sub(x, k.max(x, (1,), True)))


def _normalised(k, ref):
    x = k.cast(k.load(ref, dvm.float16), dvm.float32)
    d = k.sub(x, k.mul(k.sum(x, (1,), True), 1.0 / 64))
    v = k.mul(k.sum(k.mul(d, d), (1,), True), 1.0 / 64)
    k.store(k.cast(k.div(d, k.sqrt(k.add(v, 1e-5))), dvm.float16))


def _odd_matmul(k, ref):
    a, b = k.load(ref, dvm.float16), k.load([1001, 2003], dvm.float16)
    k.store(k.sum(k.cast(k.matmul(a, b, False, False), dvm.float32), (1,), True))


@pytest.mark.parametrize("build,kind,shape", [(_norm, "vector", lambda i: [3 + i, 40 + 24 * i]), (_normalised, "vector", lambda i: [100 + 300 * i, 64]),
                                              (_odd_matmul, "split", lambda i: [5 + 61 * i, 1001])])
def test_shapes_that_come_back(build, kind, shape):
    def kernel(dims):
        k, ref = dvm.PyKernel(kind, "das", 0), dvm.IntArrayRef(dims)
        build(k, ref)
        return k, ref

    fresh = []
    for i in range(20):
        k, _ = kernel(shape(i))
        k.codegen()
        fresh.append(k.das())
    assert len(set(fresh)) == 20
    k, ref = kernel(shape(0))
    order = list(range(20)) * 2 + [3, 4, 3, 4, 19, 0, 10, 3]
    for i in order:
        ref.update(shape(i))
        k.codegen()
        assert k.das() == fresh[i], i


def test_scalars_axes_and_bounds_that_come_back():
    def kernel():
        k = dvm.PyKernel("vector", "das", 0)
        scale, dims, begin, end = k.scalar(), dvm.IntArrayRef([1]), k.scalar(), k.scalar()
        x = k.load([12, 40], dvm.float32)
        w = k.slice_dim(x, 1, begin, end)
        k.store(k.mul(w, scale))
        k.store(k.max(k.mul(w, 2.0), dims, True))
        return k, (scale, dims, begin, end)

    def program(k, refs, values):
        refs[0].update(values[0])
        refs[1].update([values[1]])
        refs[2].update(values[2])
        refs[3].update(values[3])
        k.codegen()
        return k.das()

    values = [(1.5, 1, 0, 40), (2.5, 1, 0, 40), (2.5, 0, 0, 40), (2.5, 0, 4, 40), (2.5, 0, 4, 36)]
    fresh = [program(*kernel(), v) for v in values]
    assert len(set(fresh)) == len(values)
    k, refs = kernel()
    for i in (0, 1, 2, 3, 4, 3, 2, 1, 0, 4, 0):
        assert program(k, refs, values[i]) == fresh[i], i


@pytest.mark.gpu
def test_results_with_new_buffers_and_a_workspace():
    import torch
    rows = [7 + 29 * i for i in range(19)]
    k, ref = dvm.PyKernel("split"), dvm.IntArrayRef([rows[0], 257])
    la, lb = k.load(ref, dvm.float16), k.load([257, 1003], dvm.float16)
    product = k.cast(k.matmul(la, lb, False, False), dvm.float32)
    stores = [k.store(k.sum(product, (1,), True)), k.store(k.mul(product, 2.0))]
    b = torch.randn((257, 1003), device="cuda").half()
    stream = torch.cuda.current_stream().cuda_stream
    for m in rows * 2:
        ref.update([m, 257])
        a = torch.randn((m, 257), device="cuda").half()
        outs = [torch.zeros((m, 1), device="cuda"), torch.zeros((m, 1003), device="cuda")]
        for op, t in zip([la, lb] + stores, [a, b] + outs):
            k.bind_device(op, t.data_ptr(), t.numel() * t.element_size())
        k.codegen()
        k.launch(stream)
        torch.cuda.synchronize()
        want = a.double() @ b.double()
        # one rounding of the product to fp16 (2^-11 of it, values up to 100), 257 and 1003 terms in fp32
        bound = 2.0 ** -11 * want.abs() + 2.0 ** -24 * 258 * 257 ** 0.5 + 2.0 ** -25
        assert bool(((outs[1].double() / 2 - want).abs() <= bound).all()), m
        assert bool(((outs[0].double() - want.sum(1, keepdim=True)).abs() <= bound.sum(1, keepdim=True)).all()), m
