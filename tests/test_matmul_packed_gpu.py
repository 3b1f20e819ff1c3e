"""MatMul operands in rows that do not start on 16 bytes: repacked in the workspace, or loaded as they are without one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trans", ["", "a", "b"])
@pytest.mark.parametrize("batch,m,n,k", [((), 1, 9, 1), ((), 300, 259, 65), ((), 129, 1001, 127), ((3,), 257, 63, 71), ((2, 3), 66, 130, 33),
                                         ((), 513, 264, 1023), ((5,), 8, 7, 1025)])
def test_both_paths(batch, m, n, k, trans):
    from dvm_b200 import _capi
    from dvm_b200.tester import Tester
    lib = _capi.load()
    rng = np.random.default_rng(m + 3 * n + 5 * k)
    a = rng.standard_normal(batch + (m, k)).astype(np.float16)
    b = (rng.standard_normal(batch[-1:] + (k, n)) / np.sqrt(k)).astype(np.float16)   # (a leading batch axis is broadcast)
    t = Tester("mix")
    la = t.load(np.ascontiguousarray(np.swapaxes(a, -1, -2)) if trans == "a" else a)
    lb = t.load(np.ascontiguousarray(np.swapaxes(b, -1, -2)) if trans == "b" else b)
    s = t.store(t.matmul(la, lb, trans == "a", trans == "b"))
    t.run()
    want = a.astype(np.float64) @ b.astype(np.float64)
    # one rounding to fp16 (2^-11 of the result); the fp32 sum of k terms of size 1 / sqrt(k) is off by less than k 2^-24
    bound = 2.0 ** -11 * np.abs(want) + 2.0 ** -24 * (k + 1.0) + 2.0 ** -25
    assert np.all(np.abs(t.output(s).astype(np.float64) - want) <= bound)
    ops = [la, lb, s]
    relocs = (_capi.Reloc * len(ops))()
    for i, op in enumerate(ops):
        relocs[i].io, relocs[i].addr = op._h, t.device_ptr(op)
    assert lib.dvm_rt_memset(t.device_ptr(s), 0, want.size * 2, None) == 0
    assert lib.dvm_launch_reloc(t._k, relocs, len(relocs), None, None) == 0, _capi.last_error()   # no workspace
    assert lib.dvm_rt_sync(None) == 0, _capi.last_error()
    assert np.all(np.abs(t.output(s).astype(np.float64) - want) <= bound)


@pytest.mark.parametrize("trans", [False, True])
def test_one_kernel_on_two_streams(trans):
    """Launches on two streams, bound to other tensors in between, do not see each other's operands."""
    import torch
    import dvm_b200 as dvm
    m, n, kk, rounds = 515, 2001, 1001, 12
    g = torch.Generator(device="cuda").manual_seed(1)
    k = dvm.PyKernel("mix")
    la, lb = k.load([kk, m] if trans else [m, kk], dvm.float16), k.load([kk, n], dvm.float16)
    st = k.store(k.matmul(la, lb, trans, False))
    sets = []
    for _ in range(rounds):
        a, b = (torch.randn(shape, generator=g, device="cuda").half() for shape in ((kk, m) if trans else (m, kk), (kk, n)))
        sets.append((a, b, torch.zeros((m, n), device="cuda", dtype=torch.float16)))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for i, tensors in enumerate(sets):
        for op, t in zip((la, lb, st), tensors):
            k.bind_device(op, t.data_ptr(), t.numel() * 2)
        k.codegen()
        k.launch(streams[i % 2].cuda_stream)
    torch.cuda.synchronize()
    for a, b, c in sets:
        want = (a.double().T if trans else a.double()) @ b.double()
        # (the bound of test_both_paths, for operands of size 1)
        bound = 2.0 ** -11 * want.abs() + 2.0 ** -24 * (kk + 1.0) * kk ** 0.5 + 2.0 ** -25
        assert bool(((c.double() - want).abs() <= bound).all())


def test_captured_launch_needs_no_workspace():
    """The graph of a captured launch is replayed after the kernel, and with it its workspace, is gone."""
    import gc
    import torch
    import dvm_b200 as dvm
    m, n, kk = 300, 1001, 257
    a, b = torch.randn((m, kk), device="cuda").half(), torch.randn((kk, n), device="cuda").half()
    c = torch.zeros((m, n), device="cuda", dtype=torch.float16)
    k = dvm.PyKernel("mix")
    la, lb = k.load([m, kk], dvm.float16), k.load([kk, n], dvm.float16)
    st = k.store(k.matmul(la, lb, False, False))
    for op, t in ((la, a), (lb, b), (st, c)):
        k.bind_device(op, t.data_ptr(), t.numel() * 2)
    k.codegen()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    k.launch(stream.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        k.launch(stream.cuda_stream)
    del k, la, lb, st
    gc.collect()
    a.copy_(torch.randn((m, kk), device="cuda"))
    c.zero_()
    graph.replay()
    torch.cuda.synchronize()
    want = a.double() @ b.double()
    bound = 2.0 ** -11 * want.abs() + 2.0 ** -24 * (kk + 1.0) * kk ** 0.5 + 2.0 ** -25
    assert bool(((c.double() - want).abs() <= bound).all())
