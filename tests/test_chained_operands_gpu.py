"""Launches back to back on one stream, each reading an operand that the launch in front of it has just written: every kernel and
every kind of operand that is not fetched by the copy engine.  The outputs have to be those of the same launches with a
synchronisation between them, bit for bit."""
import math

import pytest

pytestmark = pytest.mark.gpu

ROUNDS = 6


def _consumers():
    """name -> (kernel type, input shapes and types, index of the input that is written late, output shapes and types, graph)"""
    import dvm_b200 as dvm
    from dvm_b200 import workloads as W
    f32, f16, bf16 = dvm.float32, dvm.float16, dvm.bfloat16

    def gelu(k, a, b, bias):
        return [k.cast(W.gelu_tanh(k, k.cast(k.matmul(a, b, False, False, bias), f32)), bf16)]

    def scaled(k, a, b, row):
        return [k.mul(k.cast(k.matmul(a, b, False, False), f32), row)]

    def rms(k, h, r, w, g, u):
        return list(W.rmsnorm_swiglu(k, h, r, w, g, u, 1031))

    def norm(k, x, g, b):
        return list(W.batchnorm_train(k, x, g, b, 8 * 20 * 21))

    def row_max(k, x, w):
        return [k.mul(k.sub(x, k.max(x, (1,), True)), w)]

    def plain(k, a, b):
        return [k.matmul(a, b, False, False)]

    def attention(k, q, kk, v):
        return [W.attention(k, q, kk, v, 1.0 / math.sqrt(64), bf16)]

    mm = lambda m, n, kk: [((m, kk), bf16), ((kk, n), bf16)]
    out = {
        "bias of a tile": ("mix", mm(16, 520, 512) + [((520,), bf16)], 2, [((16, 520), bf16)], gelu),
        "bias of a pair": ("mix", mm(2048, 2304, 128) + [((2304,), bf16)], 2, [((2048, 2304), bf16)], gelu),
        "bias, fp32 rows": ("mix", mm(2048, 2304, 128) + [((1, 2304), f32)], 2, [((2048, 2304), f32)], scaled),
        "epilogue matrix of a tile": ("mix", mm(40, 264, 192) + [((40, 264), f32)], 2, [((40, 264), f32)], scaled),
        "unaligned operand, repacked": ("mix", mm(700, 1001, 513), 1, [((700, 1001), bf16)], plain),
        "unaligned operand, loaded": ("mix", mm(7, 129, 65), 1, [((7, 129), bf16)], plain),
        "weight of an RMS norm": ("vector", [((33, 1031), bf16)] * 2 + [((1031,), bf16)] + [((33, 1031), bf16)] * 2, 2, [((33, 1031), bf16)] * 2, rms),
        "scale of a batch norm": ("vector", [((8, 12, 20, 21), f16)] + [((1, 12, 1, 1), f32)] * 2, 1,
                                  [((8, 12, 20, 21), f16)] + [((1, 12, 1, 1), f32)] * 2, norm),
        "input of the interpreter": ("vector", [((90, 777), f32), ((1, 777), f32)], 1, [((90, 777), f32)], row_max),
        "keys of a decode step": ("split", [((4, 8, 1, 64), bf16)] + [((4, 8, 333, 64), bf16)] * 2, 1, [((4, 8, 1, 64), bf16)], attention),
    }
    return out


NAMES = ["bias of a tile", "bias of a pair", "bias, fp32 rows", "epilogue matrix of a tile", "unaligned operand, repacked",
         "unaligned operand, loaded", "weight of an RMS norm", "scale of a batch norm", "input of the interpreter", "keys of a decode step"]


@pytest.mark.parametrize("name", NAMES)
def test_operand_written_by_the_launch_before(name):
    import torch
    import dvm_b200 as dvm
    kind, ins, late, outs, graph = _consumers()[name]
    types = {int(dvm.float32): torch.float32, int(dvm.float16): torch.float16, int(dvm.bfloat16): torch.bfloat16}
    gen = torch.Generator(device="cuda").manual_seed(3)
    inputs = [torch.randn(s, generator=gen, device="cuda").to(types[int(t)]) for s, t in ins]
    fresh = [torch.randn(ins[late][0], generator=gen, device="cuda").to(types[int(ins[late][1])]) for _ in range(ROUNDS)]
    stream = torch.cuda.Stream()

    def kernel(kind, shapes, build, tensors):
        k = dvm.PyKernel(kind)
        loads = [k.load(list(s), t) for s, t in shapes]
        ops = loads + [k.store(v) for v in build(k, *loads)]
        for op, t in zip(ops, tensors):
            k.bind_device(op, t.data_ptr(), t.numel() * t.element_size())
        k.codegen()
        return k

    def run(synchronise):
        for t in [inputs[late]] + [t for r in results for t in r]:
            t.zero_()
        torch.cuda.synchronize()
        for w, c in launches:
            for k in (w, c):
                k.launch(stream.cuda_stream)
                if synchronise:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return [t.clone() for r in results for t in r]

    results = [[torch.zeros(s, dtype=types[int(t)], device="cuda") for s, t in outs] for _ in range(ROUNDS)]
    copy = lambda k, x: [k.maximum(x, x)]
    launches = [(kernel("vector", [ins[late]], copy, [fresh[i], inputs[late]]), kernel(kind, ins, graph, inputs + results[i]))
                for i in range(ROUNDS)]
    want = run(True)
    assert all(bool(torch.isfinite(t.float()).all()) for t in want)
    for _ in range(20):
        got = run(False)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
