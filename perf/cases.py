"""Timed cases of the framework: fused operator graphs as a program runs them, through the Python package.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges, ``prepare(case, seed)`` makes what a
program holds before the call (device tensors, a planned kernel bound to them), ``run(state)`` is one pass.

Graph kinds, with the ranges that the drawn cases cover:

* ``elementwise``: exp(x) * y + 0.5 on [rows, cols] in fp32, fp16 or bf16, 16 elements to 8192 x 8192.
* ``batchnorm``: training forward of an NCHW fp16 activation with fp32 statistics, up to [64, 256, 56, 56].
* ``rmsnorm``: residual add + RMSNorm and SwiGLU gate of [tokens, hidden] bf16, 1 to 16384 tokens.  With ``new_shapes``
  a pass is two steps of a serving loop whose token count changes from step to step: the kernel is planned again for the
  step's shape and launched.
* ``attention``: softmax(Q K^T scale) V, head size 64 or 128, from one query row against a key/value cache (decode) to
  square prefill.
* ``matmul``: A B with bias and tanh-GeLU (a layer's forward, from one row of tokens up), or a plain product with one
  operand transposed (the two products of its backward); widths that are and that are not multiples of eight elements.
* ``numpy_call``: a function decorated with ``@kernel`` called on NumPy arrays, the whole call.
"""
import math

import numpy as np
import torch

import dvm_b200 as dvm
from dvm_b200 import workloads

_TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_DVM = {"f32": dvm.float32, "f16": dvm.float16, "bf16": dvm.bfloat16}
_BYTES = {"f32": 4, "f16": 2, "bf16": 2}

# upper limits of the drawn cases: those of the largest listed case of a kind
_ELEMENTS = 8192 * 8192
_BATCHNORM = 64 * 256 * 56 * 56
_RMSNORM = 16384 * 4096
_ATTENTION_FLOPS = 4 * 8 * 32 * 2048 * 2048 * 128
_MATMUL_FLOPS = 2 * 16384 * 8192 * 8192
_MATMUL_ODD_FLOPS = 2 * 1024 * 1001 * 5003


def listed():
    return [
        # a small step of an element-wise chain: all launch
        {"name": "elementwise_small", "kind": "elementwise", "rows": 16, "cols": 1000, "dtype": "bf16"},
        # the same chain on a tensor far beyond the caches
        {"name": "elementwise_large", "kind": "elementwise", "rows": 8192, "cols": 8192, "dtype": "f32"},
        # training batch-norm of a convolution's output, the benchmark's shape
        {"name": "batchnorm_train", "kind": "batchnorm", "n": 64, "c": 256, "h": 56, "w": 56},
        # a late layer of a small batch: odd planes, few elements per channel
        {"name": "batchnorm_odd_plane", "kind": "batchnorm", "n": 32, "c": 200, "h": 27, "w": 27},
        # decode steps of a serving loop: a handful of tokens, another count in every step
        {"name": "rmsnorm_decode_steps", "kind": "rmsnorm", "tokens": 7, "hidden": 4096, "new_shapes": True},
        # a long prefill
        {"name": "rmsnorm_prefill", "kind": "rmsnorm", "tokens": 16384, "hidden": 4096, "new_shapes": False},
        # attention of a prefill, the benchmark's shape
        {"name": "attention_prefill", "kind": "attention", "batch": 8, "heads": 32, "sq": 2048, "skv": 2048, "d": 128, "dtype": "bf16"},
        # one new token against a cache of odd length
        {"name": "attention_decode", "kind": "attention", "batch": 2, "heads": 32, "sq": 1, "skv": 3999, "d": 128, "dtype": "bf16"},
        # a layer's forward on many tokens, the benchmark's shape
        {"name": "matmul_gelu_large", "kind": "matmul", "m": 16384, "n": 8192, "k": 8192, "form": "gelu", "dtype": "bf16"},
        # the same layer in decode: sixteen rows against the whole weight
        {"name": "matmul_gelu_decode", "kind": "matmul", "m": 16, "n": 8192, "k": 8192, "form": "gelu", "dtype": "bf16"},
        # weight gradient of a head of odd width: X^T dY over an odd number of rows
        {"name": "matmul_grad_odd_width", "kind": "matmul", "m": 1024, "n": 5003, "k": 1001, "form": "trans_a", "dtype": "f16"},
        # the decorator's call on host arrays
        {"name": "numpy_call", "kind": "numpy_call", "rows": 1000, "cols": 1024},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def _width(rng, lo, hi):
    """A width over the logarithm of the range; half of them multiples of 64, as layers have, the rest as they fall."""
    v = _log_int(rng, lo, hi)
    return max(64, v // 64 * 64) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(["elementwise", "batchnorm", "rmsnorm", "prefill", "decode", "matmul", "matmul_decode", "matmul_odd",
                       "numpy_call"])
    if kind == "elementwise":
        return {"kind": kind, "rows": _log_int(rng, 1, 8192), "cols": _width(rng, 16, 8192),
                "dtype": rng.choice(["f32", "f16", "bf16"])}
    if kind == "batchnorm":
        n, c, h = _log_int(rng, 4, 64), _log_int(rng, 16, 512), _log_int(rng, 7, 112)
        w = max(7, h + rng.choice([0, 0, 0, -1, 1]))
        return {"kind": kind, "n": max(1, min(n, _BATCHNORM // (c * h * w))), "c": c, "h": h, "w": w}
    if kind == "rmsnorm":
        hidden = _width(rng, 256, 8192)
        tokens = min(_log_int(rng, 1, 16384), _RMSNORM // hidden)
        return {"kind": kind, "tokens": tokens, "hidden": hidden, "new_shapes": tokens <= 512}
    if kind == "prefill":
        heads, d, s = rng.choice([4, 8, 12, 16, 32]), rng.choice([64, 128]), _log_int(rng, 64, 4096)
        batch = max(1, min(_log_int(rng, 1, 8), _ATTENTION_FLOPS // (4 * heads * s * s * d)))
        return {"kind": "attention", "batch": batch, "heads": heads, "sq": s, "skv": s, "d": d, "dtype": rng.choice(["bf16", "f16"])}
    if kind == "decode":
        return {"kind": "attention", "batch": _log_int(rng, 1, 16), "heads": rng.choice([4, 8, 12, 16, 32]),
                "sq": rng.choice([1, 1, 1, 2, 4]), "skv": _log_int(rng, 128, 8192), "d": rng.choice([64, 128]),
                "dtype": rng.choice(["bf16", "f16"])}
    if kind == "numpy_call":
        return {"kind": kind, "rows": _log_int(rng, 1, 4096), "cols": _width(rng, 64, 4096)}
    dtype = rng.choice(["bf16", "f16"])
    if kind == "matmul_odd":   # an odd width or an odd depth: rows that do not start on 16 bytes
        form = rng.choice(["gelu", "trans_a", "trans_b"])
        n, k = _log_int(rng, 64, 5003) | 1, _log_int(rng, 64, 4096)
        m = min(_log_int(rng, 8, 4096), _MATMUL_ODD_FLOPS // (2 * n * k))
        return {"kind": "matmul", "m": max(1, m), "n": n, "k": k, "form": form, "dtype": dtype}
    n, k = (8 * _log_int(rng, 32, 1024) for _ in range(2))
    if kind == "matmul_decode":
        return {"kind": "matmul", "m": _log_int(rng, 1, 64), "n": n, "k": k, "form": "gelu", "dtype": dtype}
    form = rng.choice(["gelu", "gelu", "trans_a", "trans_b"])
    m = min(_log_int(rng, 65, 16384), _MATMUL_FLOPS // (2 * n * k))
    if form == "trans_a":
        m = max(8, m // 8 * 8)
    return {"kind": "matmul", "m": m, "n": n, "k": k, "form": form, "dtype": dtype}


def _tensors(case, seed):
    """(inputs, output shapes and types): the tensors of one call, in the order the graph loads and stores them."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(shape, dtype, mean=0.0, std=1.0):
        t = torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=g)
        return t.to(_TORCH[dtype])

    kind = case["kind"]
    if kind == "elementwise":
        shape = (case["rows"], case["cols"])
        xs = [torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(-1, 1, generator=g).to(_TORCH[case["dtype"]])
              for _ in range(2)]
        return xs, [(shape, case["dtype"])]
    if kind == "batchnorm":
        shape, per_c = (case["n"], case["c"], case["h"], case["w"]), (1, case["c"], 1, 1)
        return ([normal(shape, "f16"), normal(per_c, "f32", 1.0, 0.1), normal(per_c, "f32", 0.0, 0.1)],
                [(shape, "f16"), (per_c, "f32"), (per_c, "f32")])
    if kind == "rmsnorm":
        # (with changing shapes the second step has one token more)
        shape = (case["tokens"] + (1 if case["new_shapes"] else 0), case["hidden"])
        h, r, gate, up = (normal(shape, "bf16") for _ in range(4))
        return [h, r, normal((case["hidden"],), "bf16", 1.0, 0.02), gate, up], [(shape, "bf16"), (shape, "bf16")]
    if kind == "attention":
        head = (case["batch"], case["heads"])
        return ([normal(head + (s, case["d"]), case["dtype"]) for s in (case["sq"], case["skv"], case["skv"])],
                [(head + (case["sq"], case["d"]), case["dtype"])])
    m, n, k, dt = case["m"], case["n"], case["k"], case["dtype"]
    a = normal((k, m) if case["form"] == "trans_a" else (m, k), dt, 0.0, 0.02 if case["form"] == "gelu" else 1.0)
    b = normal((n, k) if case["form"] == "trans_b" else (k, n), dt, 0.0, 0.02)
    return [a, b] + ([normal((n,), dt, 0.0, 0.02)] if case["form"] == "gelu" else []), [((m, n), dt)]


def _graph(k, case, x):
    kind = case["kind"]
    if kind == "elementwise":
        return [workloads.fused_elementwise(k, *x)]
    if kind == "batchnorm":
        return list(workloads.batchnorm_train(k, *x, case["n"] * case["h"] * case["w"]))
    if kind == "rmsnorm":
        return list(workloads.rmsnorm_swiglu(k, *x, case["hidden"]))
    if kind == "attention":
        return [workloads.attention(k, *x, 1.0 / math.sqrt(case["d"]), _DVM[case["dtype"]])]
    if case["form"] != "gelu":
        return [k.matmul(x[0], x[1], case["form"] == "trans_a", case["form"] == "trans_b")]
    y = workloads.gelu_tanh(k, k.cast(k.matmul(x[0], x[1], False, False, x[2]), dvm.float32))
    return [k.cast(y, _DVM[case["dtype"]])]


_KERNEL_TYPE = {"elementwise": "vector", "batchnorm": "vector", "rmsnorm": "vector:spec,dyn", "attention": "split", "matmul": "mix"}


def _bind(k, op, t):
    k.bind_device(op, t.data_ptr(), t.numel() * t.element_size())


def prepare(case, seed):
    if case["kind"] == "numpy_call":
        rng = np.random.default_rng(seed)
        shape = (case["rows"], case["cols"])

        @dvm.kernel
        def chain(k, x, y):
            return k.store(workloads.fused_elementwise(k, k.load(x, dvm.float32), k.load(y, dvm.float32)))

        return {"call": chain, "arrays": [rng.uniform(-1, 1, shape).astype(np.float32) for _ in range(2)]}
    inputs, outs = _tensors(case, seed)
    outputs = [torch.empty(shape, dtype=_TORCH[dt], device="cuda") for shape, dt in outs]
    k = dvm.PyKernel(_KERNEL_TYPE[case["kind"]], "dev", torch.cuda.current_device())
    names = {v: n for n, v in _TORCH.items()}
    shapes = [dvm.IntArrayRef(list(t.shape)) for t in inputs]
    loads = [k.load(s, _DVM[names[t.dtype]]) for s, t in zip(shapes, inputs)]
    stores = [k.store(v) for v in _graph(k, case, loads)]
    for op, t in zip(loads + stores, inputs + outputs):
        _bind(k, op, t)
    k.codegen()
    state = {"kernel": k, "inputs": inputs, "outputs": outputs, "stream": torch.cuda.current_stream().cuda_stream}
    if case.get("new_shapes"):
        # the tensors of the two steps: views of one buffer each, as a serving loop's activations are
        state["steps"] = []
        for i, tokens in enumerate((case["tokens"], case["tokens"] + 1)):
            step_in = [t if t.dim() == 1 else t[:tokens] for t in inputs]
            step_out = [t[:tokens] if i else torch.empty_like(t[:tokens]) for t in outputs]
            state["steps"].append((step_in, step_out))
        state["shapes"], state["loads"], state["stores"] = shapes, loads, stores
    return state


def run(state):
    if "call" in state:
        return state["call"](*state["arrays"])
    k, stream = state["kernel"], state["stream"]
    if "steps" not in state:
        k.launch(stream)
        return state["outputs"]
    done = []
    for step_in, step_out in state["steps"]:
        for ref, op, t in zip(state["shapes"], state["loads"], step_in):
            ref.update(t.shape)
            _bind(k, op, t)
        for op, t in zip(state["stores"], step_out):
            _bind(k, op, t)
        k.codegen()
        k.launch(stream)
        done += step_out
    return done


def work(case):
    kind = case["kind"]
    if kind in ("elementwise", "numpy_call"):
        n = case["rows"] * case["cols"]
        return {"bytes": 3 * n * _BYTES[case.get("dtype", "f32")], "flops": 3 * n}
    if kind == "batchnorm":
        n = case["n"] * case["c"] * case["h"] * case["w"]
        return {"bytes": 4 * n + 16 * case["c"], "flops": 8 * n}
    if kind == "rmsnorm":
        tokens = 2 * case["tokens"] + 1 if case["new_shapes"] else case["tokens"]
        steps = 2 if case["new_shapes"] else 1
        return {"bytes": 12 * tokens * case["hidden"] + 2 * steps * case["hidden"], "flops": 12 * tokens * case["hidden"]}
    if kind == "attention":
        heads, d = case["batch"] * case["heads"], case["d"]
        return {"bytes": 4 * heads * d * (case["sq"] + case["skv"]), "flops": 4 * heads * case["sq"] * case["skv"] * d}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": 2 * (m * k + k * n + m * n + (n if case["form"] == "gelu" else 0)), "flops": 2 * m * n * k}


def tolerance(case):
    """What the stored types give: one rounding to fp32 with a 2-ulp division or exponential, or roundings to 8 or 11 bits
    (a batch-norm's fp32 mean of a centred input is a sum that nearly cancels, and stays inside the fp16 figure)."""
    dtype = case.get("dtype", {"batchnorm": "f16", "rmsnorm": "bf16"}.get(case["kind"], "f32"))
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[dtype]}
