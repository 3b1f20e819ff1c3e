"""Statistics kernel: groups around its units, tiles, clusters and threads, group scalars in every form, against float64."""
import pytest

pytestmark = pytest.mark.gpu

EPS = 1e-5


def _run(shape, dims, dtype="float16", offset=0, unlike=0, in_place=False, gamma=None, beta=None, stored=("mean", "var"), special=None):
    """y = (x - mean) / std [gamma] [beta] of x over `dims`, x `offset` elements into its buffer and y at another one relative to 16
    bytes by `unlike`.  Returns the listing's kernel and (result, float64 expectation) of y and of what is stored."""
    import torch
    import dvm_b200 as dvm
    types = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}
    codes = {"float16": dvm.float16, "bfloat16": dvm.bfloat16, "float32": dvm.float32}
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    per = [1 if d in dims else s for d, s in enumerate(shape)]
    numel = 1
    for s in shape:
        numel *= s
    raw = torch.randn(shape, generator=g, device="cuda") * 1.5 + torch.randn(per, generator=g, device="cuda")
    if special is not None:
        special(raw)
    buf = torch.zeros(offset + numel, dtype=types[dtype], device="cuda")
    buf[offset:] = raw.to(types[dtype]).reshape(-1)
    x = buf[offset:].reshape(shape)
    out = buf if in_place else torch.full((offset + unlike + numel + 8,), 7.0, dtype=types[dtype], device="cuda")
    y_at = offset if in_place else offset + unlike
    x64 = x.double().clone()
    k = dvm.PyKernel("vector")
    binds, scalars = [(k.load(list(shape), codes[dtype]), buf, offset)], {}
    f = k.cast(binds[0][0], dvm.float32)
    count = 1.0
    for d in dims:
        count *= shape[d]
    mean = k.mul(k.sum(f, dims, True), 1.0 / count)
    d = k.sub(f, mean)
    var = k.mul(k.sum(k.mul(d, d), dims, True), 1.0 / count)
    std = k.sqrt(k.add(var, EPS))
    y = k.div(d, std)
    for name, kind in (("gamma", gamma), ("beta", beta)):
        if kind is None:
            continue
        scalars[name] = (1.0 + 0.1 * torch.randn(per, generator=g, device="cuda")).to(types[kind])
        v = k.load(per, codes[kind])
        binds.append((v, scalars[name], 0))
        v = v if kind == "float32" else k.cast(v, dvm.float32)
        y = k.mul(y, v) if name == "gamma" else k.add(y, v)
    y_op = k.store(k.cast(y, codes[dtype]))
    binds.append((y_op, out, y_at))
    results = [torch.zeros(per, device="cuda") for _ in stored]
    for name, t in zip(stored, results):
        binds.append((k.store({"mean": mean, "var": var, "std": std}[name]), t, 0))
    for op, t, at in binds:
        k.bind_device(op, t.data_ptr() + at * t.element_size(), (t.numel() - at) * t.element_size())
    k.codegen()
    k.launch(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    if not in_place:   # nothing is written beside y
        assert bool((out[:y_at] == 7.0).all()) and bool((out[y_at + numel:] == 7.0).all())
    elif offset:
        assert bool((buf[:offset] == 0.0).all())
    m = x64.mean(dims, keepdim=True)
    v = ((x64 - m) ** 2).mean(dims, keepdim=True)
    want = (x64 - m) / (v + EPS).sqrt()
    if gamma is not None:
        want = want * scalars["gamma"].double()
    if beta is not None:
        want = want + scalars["beta"].double()
    pairs = [(out[y_at:y_at + numel].reshape(shape).double(), want)]
    pairs += [(t.double(), {"mean": m, "var": v, "std": (v + EPS).sqrt()}[name]) for name, t in zip(stored, results)]
    return k.das().split("kernel=")[1].split(")")[0], pairs


def _close(pairs, dtype):
    """Sums of 8 x (16 units + warps) fp32 terms in a tree, deviations from the group's first element, which lies within 5 std of the
    mean here: the variance is off by about 40 2^-24 (1 + 25), y by half of that and its own rounding; the mean by 40 2^-24 of 5 std
    (std about 1.5)."""
    (y, want), rest = pairs[0], pairs[1:]
    ulp = {"float16": 2.0 ** -11, "bfloat16": 2.0 ** -8}[dtype]
    assert bool(((y - want).abs() <= ulp * want.abs() + 1e-4 * (1.0 + want.abs())).all()), float((y - want).abs().max())
    for got, ref in rest:
        assert bool(((got - ref).abs() <= 1e-4 * ref.abs() + 2e-5).all()), float((got - ref).abs().max())


# one unit and less, planes that start anywhere, 4 / 8 / 14 units a thread and one more, 1 to 8 CTAs a group, tiles of 55 KB (3552 units) and
# above, two to four CTAs on an SM
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("shape", [(1, 3, 1, 2), (2, 5, 1, 3), (3, 2, 2, 4), (5, 4, 3, 3), (4, 300, 5, 5), (7, 40, 7, 7), (2, 150, 16, 16),
                                   (1, 160, 128, 128), (1, 160, 128, 129), (2, 160, 128, 127), (32, 200, 27, 27), (9, 700, 28, 28),
                                   (16, 48, 55, 55), (4, 16, 112, 113), (64, 256, 14, 56), (3, 310, 130, 129), (8, 3, 255, 257),
                                   (12, 2, 256, 256), (1, 2, 905, 905), (111, 300, 16, 16), (111, 600, 16, 16), (112, 300, 16, 16),
                                   (65, 444, 16, 16), (65, 445, 16, 16), (38, 300, 27, 27), (38, 500, 27, 27), (222, 160, 16, 16)])
def test_planes_of_a_channel(shape, dtype):
    kernel, pairs = _run(shape, (0, 2, 3), dtype, gamma="float32", beta="float32")
    assert kernel == "stats_affine"
    _close(pairs, dtype)


# groups of two coordinates (an instance norm), rows, everything; scalars of any type, present or not; what is stored
@pytest.mark.parametrize("shape,dims,gamma,beta,stored", [
    ((5, 6, 9, 11), (2, 3), "float32", "float16", ("var",)), ((6, 7, 1001), (2,), None, "bfloat16", ("std", "mean")),
    ((33, 515), (1,), "float16", None, ()), ((33, 512), (1,), None, None, ("mean", "var", "std")), ((7, 33), (0, 1), None, None, ("mean",))])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("offset", [0, 1, 6, 8])
def test_group_scalars_addresses_and_in_place(shape, dims, gamma, beta, stored, in_place, offset):
    kernel, pairs = _run(shape, dims, "float16", offset=offset, in_place=in_place, gamma=gamma, beta=beta, stored=stored)
    assert kernel == "stats_affine"
    _close(pairs, "float16")


@pytest.mark.parametrize("unlike,kernel", [(0, "stats_affine"), (8, "stats_affine"), (1, "interpreter"), (4, "interpreter")])
def test_a_result_that_lies_otherwise_takes_the_interpreter(unlike, kernel):
    ran, pairs = _run((6, 5, 9, 9), (0, 2, 3), offset=3, unlike=unlike, gamma="float32", beta="float32")
    assert ran == kernel
    _close(pairs, "float16")


def test_special_values_stay_in_their_group():
    """A NaN or an infinity makes its own group NaN, as the graph does; the edges of neighbouring groups share 16-byte units."""
    import torch

    def special(raw):
        raw[1, 2, 3, 4] = float("nan")
        raw[0, 4, 8, 8] = float("inf")
        raw[:, 6] = 0.25   # a constant channel: (x - mean) is 0 exactly

    kernel, pairs = _run((3, 9, 9, 9), (0, 2, 3), special=special, gamma="float32", beta="float32")
    assert kernel == "stats_affine"
    (y, want), (mean, m), (var, v) = pairs
    for c in (2, 4):
        assert bool(torch.isnan(y[:, c]).all()) and bool(torch.isnan(want[:, c]).all())
    rest = [0, 1, 3, 5, 6, 7, 8]
    _close([(y[:, rest], want[:, rest]), (mean[:, rest], m[:, rest]), (var[:, rest], v[:, rest])], "float16")
    assert float(var[0, 6, 0, 0]) == 0.0 and float(mean[0, 6, 0, 0]) == 0.25
