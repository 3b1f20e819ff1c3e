"""The calls of a loop's steps (csrc/py_calls.cc) against the general methods of the front-end: same plans and addresses, same errors."""
import numpy as np
import pytest

import dvm_b200 as dvm
from dvm_b200.frontend import _ExternalBuf


def _graph():
    """A kernel that takes itself to be on a device (planning and binding need none), its tensors at made-up addresses."""
    k = dvm.PyKernel("vector:spec,dyn", "das")
    k._run_type, k._on_device = "dev", True
    refs = [dvm.IntArrayRef([8, 64]), dvm.IntArrayRef([64])]
    loads = [k.load(r, dvm.float32) for r in refs]
    store = k.store(k.mul(k.add(loads[0], loads[1]), 2.0))
    for i, op in enumerate(loads + [store]):
        k.bind_device(op, 0x100000 * (i + 1), 1 << 16)
    return k, refs, loads, store


@pytest.mark.parametrize("rows", [8, 3, 1, 16])
def test_a_step_is_what_the_general_methods_make_of_it(rows):
    k, refs, loads, store = _graph()
    k.codegen()
    refs[0].update([rows, 64])
    k.bind_device(loads[0], 0x7000000, rows * 256)
    k.bind_device(store, 0x9000000, rows * 256)
    k.codegen()
    plain, shape = k.das(), k._stores[0][4]
    k._codegen_any()
    assert k.das() == plain and "0x7000000" in plain and "0x9000000" in plain
    assert shape == k._stores[0][4] == [rows, 64]
    other, refs2, loads2, store2 = _graph()
    refs2[0].update((rows, 64))
    other._bind_device_any(loads2[0], 0x7000000, rows * 256)
    other._bind_device_any(store2, 0x9000000, rows * 256)
    other._codegen_any()
    assert other.das() == plain


@pytest.mark.parametrize("values", [[3, 4], (3, 4), np.array([3, 4]), np.array([3, 4], np.int32), (3.9, 4), ("3", "4"), iter([3, 4]), range(3, 5)])
def test_update_takes_what_int_takes(values):
    r = dvm.IntArrayRef([1])
    r.update(values)
    assert r.shape() == (3, 4)
    r.update(shape=[5])
    assert r.shape() == (5,)
    r.update(list(range(40)))   # longer than what is compared
    r.update(list(range(40)))
    assert r.shape() == tuple(range(40))
    r.update([])
    assert r.shape() == ()
    r.update([2 ** 62, -1])
    assert r.shape() == (2 ** 62, -1)


@pytest.mark.parametrize("bad,error", [(3, TypeError), ([None], TypeError), (["x"], ValueError), ([[1]], TypeError)])
def test_update_refuses_what_int_refuses(bad, error):
    r = dvm.IntArrayRef([7, 8])
    with pytest.raises(error):
        r.update(bad)
    assert r.shape() == (7, 8)
    with pytest.raises(TypeError):
        r.update()
    with pytest.raises(TypeError):
        r.update(values=[1])


def test_errors_are_those_of_the_general_methods():
    k, refs, loads, store = _graph()
    k.codegen()
    with pytest.raises(dvm.DvmError, match="not a load or store"):
        k.bind_device(k.add(loads[0], loads[0]), 16, 16)
    with pytest.raises(TypeError):
        k.bind_device(loads[0], 16)
    with pytest.raises(TypeError):
        k.bind_device(loads[0], None, 16)
    k.bind_device(obj=loads[0], ptr=np.int64(0x8000000), nbytes=4096)   # by keyword, and a number of another type
    k.codegen(pass_names=None)
    assert "0x8000000" in k.das()
    with pytest.raises(TypeError):
        k.codegen(1, 2)
    refs[1].update([63])   # does not broadcast
    with pytest.raises(dvm.DvmError):
        k.codegen()
    refs[1].update([64])
    k.codegen()
    fresh = dvm.PyKernel("vector", "das")
    fresh._run_type, fresh._on_device = "dev", True
    fresh.store(fresh.load([4], dvm.float32))
    with pytest.raises(dvm.DvmError):   # (no memory for its tensors)
        fresh.codegen()
    with pytest.raises(dvm.DvmError, match="launch"):
        dvm.PyKernel("vector", "das").launch()


def test_external_buffers():
    b = _ExternalBuf(np.int64(64), 7.0)
    assert (b.ptr, b.nbytes) == (64, 7)
    b.free()
    assert b.ptr is None
    with pytest.raises(TypeError):
        _ExternalBuf(None, 1)


def test_update_of_a_list_that_changes_while_it_is_read():
    """An element's __int__ may do anything: what counts is what tuple(map(int, shape)) makes of it."""
    class Whole:
        def __init__(self, value, act=None):
            self.value, self.act = value, act

        def __int__(self):
            if self.act is not None:
                self.act()
            return self.value

    for act, want in ((lambda: vals.clear(), (3,)), (lambda: vals.__setitem__(1, 9), (3, 9, 5)), (lambda: vals.extend(range(60)), (3, 4, 5, *range(60)))):
        r = dvm.IntArrayRef([1])
        vals = [Whole(3, act), Whole(4), 5]
        r.update(vals)
        assert r.shape() == want


def test_update_goes_through_the_iterator_of_a_subclass():
    class Doubled(tuple):
        def __iter__(self):
            return (2 * v for v in tuple.__iter__(self))

    r = dvm.IntArrayRef([1])
    r.update(Doubled((2, 3)))
    assert r.shape() == (4, 6)


def test_a_failed_attach_leaves_what_the_array_is_known_to_hold():
    r = dvm.IntArrayRef([7, 8])
    with pytest.raises(TypeError):
        r._attach(r._h, [9, None])
    r.update([9, 8])
    assert r.shape() == (9, 8)


def test_launch_takes_a_stream_and_nothing_else(monkeypatch):
    """A second argument was the code of a failed launch, and 0 as one of them meant that nothing was launched and nothing said."""
    k = dvm.PyKernel("vector", "das")
    launched = []
    monkeypatch.setattr(k._lib, "dvm_launch", lambda *a: launched.append(a) or 0)
    for args, kw in (((0, 0), {}), ((None, 3), {}), ((), {"rc": 0}), ((0,), {"rc": None})):
        with pytest.raises(TypeError):
            k.launch(*args, **kw)
    assert not launched


def test_external_buffers_beyond_63_bits():
    """A size that no memory has is as good as any that is large enough, and a refused one changes nothing."""
    k, refs, loads, store = _graph()
    k.codegen()
    for big in (2 ** 63, 2 ** 64 - 1, 2 ** 70):
        k.bind_device(store, 0x9000000, big)
        k.codegen()
        assert "0x9000000" in k.das() and k.device_ptr(store) == 0x9000000
    k.bind_device(store, 0x5000000, -2 ** 70)   # (too small)
    assert k._stores[0][1].nbytes < 0
    b = _ExternalBuf(64, 7)
    with pytest.raises(TypeError):
        b.__init__(128, None)
    assert (b.ptr, b.nbytes) == (64, 7)


def _fake_memory(monkeypatch):
    """Device allocations as made-up addresses; their sizes."""
    import dvm_b200.frontend as F
    made = []

    class Buf:
        def __init__(self, nbytes):
            self.nbytes = nbytes
            self.ptr = 0x70000000 + 0x1000 * len(made)
            made.append(nbytes)

        def free(self):
            self.ptr = None

    monkeypatch.setattr(F, "_DevBuf", Buf)
    return made


def test_a_result_larger_than_any_number_of_64_bits_is_not_taken_for_a_small_one(monkeypatch):
    made = _fake_memory(monkeypatch)
    k, refs, loads, store = _graph()
    k.codegen()
    refs[0].update([2 ** 57, 64])   # 2 ** 65 bytes
    try:
        k.codegen()
    except dvm.DvmError:
        pass
    assert made == [2 ** 65]


def test_a_buffer_too_small_for_the_new_shape_is_replaced(monkeypatch):
    made = _fake_memory(monkeypatch)
    k, refs, loads, store = _graph()
    k.codegen()
    k.bind_device(store, 0x9000000, 8 * 64 * 4)
    k.codegen()
    assert not made and "0x9000000" in k.das()
    refs[0].update([9, 64])
    k.codegen()
    assert made == [9 * 64 * 4] and k.device_ptr(store) == 0x70000000 and "0x70000000" in k.das() and "0x9000000" not in k.das()
    refs[0].update([8, 64])
    k.codegen()   # (the kernel's own memory: the general method, and large enough)
    assert len(made) == 1 and "0x70000000" in k.das()
    k.bind_device(store, 0x9000000, 1 << 16)
    k.codegen()
    assert "0x9000000" in k.das() and "0x70000000" not in k.das()


def test_a_kernel_that_grows_after_its_first_code_generation():
    k, refs, loads, store = _graph()
    k.codegen()
    ref = dvm.IntArrayRef([8, 64])
    extra = k.load(ref, dvm.float32)
    second = k.store(k.mul(extra, loads[0]))
    with pytest.raises(dvm.DvmError):   # (nothing bound to them yet; without a device no memory either)
        k.codegen()
    k.bind_device(extra, 0xa000000, 1 << 16)
    k.bind_device(second, 0xb000000, 1 << 16)
    for rows in (8, 5):
        for r in (refs[0], ref):
            r.update([rows, 64])
        k.codegen()
        plan = k.das()
        assert "0xa000000" in plan and "0xb000000" in plan and k._stores[1][4] == [rows, 64]
        k._codegen_any()
        assert k.das() == plan


def test_steps_of_several_threads():
    """A kernel per thread, all stepping at once: the plans of each are those that it makes alone."""
    import threading

    def steps(at, rounds):
        k, refs, loads, store = _graph()
        plans = []
        for i in range(rounds):
            rows = 1 + (i * 7 + at) % 40   # (more shapes than plans are kept)
            refs[0].update([rows, 64])
            k.bind_device(loads[0], 0x10000000 * (at + 1) + 0x1000 * i, 1 << 16)
            k.bind_device(store, 0x20000000 * (at + 1) + 0x1000 * i, 1 << 16)
            k.codegen()
            plans.append(k.das())
        return plans

    alone = [steps(at, 60) for at in range(6)]
    got, failed = [None] * 6, []
    start = threading.Barrier(6)

    def work(at):
        try:
            start.wait(30)
            got[at] = steps(at, 60)
        except Exception as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(at,)) for at in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not failed and got == alone
