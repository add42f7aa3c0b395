"""Inputs and results on their way between the host and the device: the pinned page of a program (tensors of at most
64 KB), staged copies above it, results in pinned memory, quantize_rows in pieces. Values are compared for equality."""
import ctypes as C

import numpy as np
import pytest

from tensorlisp_b200 import graph as G
from tensorlisp_b200._lib import check
from tensorlisp_b200.native import Native, NativeProgram, quantize_rows

pytestmark = pytest.mark.gpu

# around the page's limit (16384 f32), its 16-byte pieces, the chunk sizes and thread counts of the staged copies
SIZES = [1, 3, 4, 1023, 4097, 16383, 16384, 16385, 65536, 65537, 262144, 262145, 524287, 524289, 4194304, 4194305]


@pytest.mark.parametrize("n", SIZES)
def test_every_run_sees_the_inputs_set_last(n):
    native = Native.load([])
    g = G.Graph()
    x, z = g.input(G.F32, [n], "x"), g.input(G.F32, [4], "z")
    y, w = g.output(g.scale(x, 2.0)), g.output(g.scale(z, 3.0))
    prog = NativeProgram.compile(native, g)
    rng = np.random.default_rng(n)
    held = []
    for i in range(4):      # from the second run on the small results come through the page
        a, b = rng.standard_normal(n).astype(np.float32), rng.standard_normal(4).astype(np.float32)
        prog.set_input(0, np.zeros(n, np.float32))
        prog.set_input(0, a)
        if i != 2:
            prog.set_input(1, b)
            last = b
        prog.run()
        got = prog.read(y)
        assert np.array_equal(got.reshape(-1), 2 * a)
        assert np.array_equal(prog.read(w).reshape(-1), 3 * last)
        held.append((got, 2 * a))
    prog.enqueue()          # nothing set in between: the same again, and read() waits for it
    assert np.array_equal(prog.read(y).reshape(-1), 2 * a)
    for got, want in held:  # results are the caller's: later runs leave them alone
        assert np.array_equal(got.reshape(-1), want)
    assert np.array_equal(prog.read(x).reshape(-1), a)
    prog.free()
    native.close()


def test_a_device_side_input_and_the_page_keep_their_order():
    native = Native.load([])
    g = G.Graph()
    x = g.input(G.F32, [8], "x")
    y = g.output(g.scale(x, 2.0))
    prog = NativeProgram.compile(native, g)
    ones = np.ones(8, np.float32)
    prog.set_input(0, ones)
    prog.run()
    prog.set_input(0, 5 * ones)     # overtaken by the copy behind it
    prog.feed_input(0, y)
    prog.run()
    assert np.array_equal(prog.read(y).reshape(-1), 4 * ones)
    prog.feed_input(0, y)           # overtaken by the input set behind it
    prog.set_input(0, 7 * ones)
    prog.enqueue()
    prog.enqueue()
    assert np.array_equal(prog.read(y).reshape(-1), 14 * ones)
    for _ in range(3):              # a loop that never waits
        prog.feed_input(0, y)
        prog.enqueue()
    assert np.array_equal(prog.read(y).reshape(-1), 112 * ones)
    prog.free()
    native.close()


def test_a_known_device_address_sees_every_input_and_every_result():
    import torch

    class At:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3, strides=None)

    native = Native.load([])
    g = G.Graph()
    x = g.input(G.F32, [16], "x")
    y = g.output(g.scale(x, 2.0))
    prog = NativeProgram.compile(native, g)
    a = np.arange(16, dtype=np.float32)
    prog.set_input(0, a)
    prog.run()
    prog.read(y)
    prog.run()
    dx, dy = torch.as_tensor(At(prog.tensor_ptr(x)[0], 16), device="cuda"), torch.as_tensor(At(prog.tensor_ptr(y)[0], 16), device="cuda")
    prog.set_input(0, a + 1)
    assert np.array_equal(dx.cpu().numpy(), a + 1)
    dx.add_(1)
    torch.cuda.synchronize()
    prog.run()
    assert np.array_equal(prog.read(y).reshape(-1), 2 * (a + 2))
    dy.fill_(9)
    torch.cuda.synchronize()
    assert np.array_equal(prog.read(y).reshape(-1), np.full(16, 9, np.float32))
    prog.free()
    native.close()


@pytest.mark.parametrize("n", [16385, 65536, 524288])
def test_a_result_that_the_run_has_written_is_handed_over_once(n):
    """Above 64 KB a result comes in the block that the run has written: a second read() of the same run, reads behind runs that were not
    waited for, and arrays that are kept (no block is left at some point) all see their own run's values."""
    native = Native.load([])
    g = G.Graph()
    x, z = g.input(G.F32, [n], "x"), g.input(G.F32, [4], "z")
    y, w = g.output(g.scale(x, 2.0)), g.output(g.scale(x, 3.0))
    prog = NativeProgram.compile(native, g)
    rng = np.random.default_rng(n)
    kept = []
    for i in range(12):
        a = rng.standard_normal(n).astype(np.float32)
        prog.set_input(0, a)
        prog.enqueue()
        if i % 3 == 0:
            prog.enqueue()
        got = [prog.read(y), prog.read(w), prog.read(y)]
        for r, f in zip(got, (2, 3, 2)):
            assert np.array_equal(r.reshape(-1), f * a)
        got[2][...] = -1        # the caller's to write to
        assert np.array_equal(prog.read(y).reshape(-1), 2 * a)
        if i >= 4:
            kept.append((got[:2], a))
    for got, a in kept:
        assert np.array_equal(got[0].reshape(-1), 2 * a) and np.array_equal(got[1].reshape(-1), 3 * a)
    prog.free()
    for got, a in kept:
        assert np.array_equal(got[0].reshape(-1), 2 * a)
    native.close()


def test_a_large_result_that_is_read_now_and_then_is_not_pushed_every_run():
    """Two runs that were not read end the pushing of a result above 64 KB, waited for or not; two runs in a row that were read bring it
    back. Every read sees the last run."""
    n = 65536
    native = Native.load([])
    g = G.Graph()
    y = g.output(g.scale(g.input(G.F32, [n], "x"), 2.0))
    prog = NativeProgram.compile(native, g)
    a = np.arange(n, dtype=np.float32)

    def go(wait=True):
        nonlocal a
        if not wait:
            return prog.enqueue()       # (a new input would wait for the runs before)
        a = a + 1
        prog.set_input(0, a)
        prog.run()

    def read():
        assert np.array_equal(prog.read(y).reshape(-1), 2 * a)

    def pushed():
        p = C.c_void_p()
        check(native.L.tlb_program_take(prog.h, y, 4 * n, C.byref(p)))
        if p.value:
            assert np.array_equal(np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (n,)), 2 * a)
            native.L.tlb_host_free(p)
        return bool(p.value)

    for wait in (True, False):
        for _ in range(3):
            go()
            read()
        go()
        assert pushed()
        for _ in range(4):
            go(wait)
        assert not pushed()
        read()              # one run is read, the next is not: not pushed
        go()
        go()
        assert not pushed()
        for _ in range(2):
            read()
            go()
        assert pushed()
        read()
    prog.free()
    native.close()


@pytest.mark.parametrize("held", ["a view", "the tensor of a view", "the tensor itself"])
def test_an_address_into_a_result_through_another_tensor_of_its_storage(held):
    """Who holds the address of a view writes into the root's memory (and the other way round): what read() returns then comes from
    there, not from the copy that runs push to the host."""
    import torch

    class At:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(ptr, False), version=3, strides=None)

    native = Native.load([])
    g = G.Graph()
    x = g.input(G.F32, [16], "x")
    y = g.output(g.scale(x, 2.0))
    v = g.output(g.view(y, [8], offset=16))
    other = g.output(g.scale(x, 3.0))
    prog = NativeProgram.compile(native, g)
    a = np.arange(16, dtype=np.float32)
    prog.set_input(0, a)
    for _ in range(2):      # from the second run on the results are pushed
        prog.run()
        prog.read(y), prog.read(v), prog.read(other)
    first, t = (4, v) if held == "a view" else (0, y)
    ptr, nbytes = prog.tensor_ptr(t)
    at = torch.as_tensor(At(ptr, nbytes // 4), device="cuda")
    watched = {"a view": y, "the tensor of a view": v, "the tensor itself": y}[held]
    for i in range(3):
        prog.run()
        want = 2 * a
        assert np.array_equal(prog.read(watched).reshape(-1), want if watched == y else want[4:12])
        at.fill_(9 + i)
        torch.cuda.synchronize()
        want[first:first + nbytes // 4] = 9 + i
        assert np.array_equal(prog.read(y).reshape(-1), want)
        assert np.array_equal(prog.read(v).reshape(-1), want[4:12])
        assert np.array_equal(prog.read(other).reshape(-1), 3 * a)
    prog.free()
    native.close()


def test_a_single_launch_is_captured_when_it_runs_again():
    native = Native.load([])
    g = G.Graph()
    s, x = g.state(G.F32, [64], "s"), g.input(G.F32, [64], "x")
    y = g.output(g.add(s, x))
    native.alloc_states([256])
    prog = NativeProgram.compile(native, g)
    blocks = [native.new_state_block() for _ in range(3)]
    rng = np.random.default_rng(0)
    held = rng.standard_normal((3, 64)).astype(np.float32)
    for b, h in zip(blocks, held):
        b.write(0, h)
    for turn in range(4):
        for i, (b, h) in enumerate(zip(blocks, held)):
            a = rng.standard_normal(64).astype(np.float32)
            prog.set_input(0, a)
            prog.run(b)
            assert np.array_equal(prog.read(y).reshape(-1), h + a)
            assert native.L.tlb_program_graph_count(prog.h) == (0 if turn == 0 else (i + 1 if turn == 1 else 3))
    prog.free()
    for b in blocks:
        b.free()
    native.close()


@pytest.mark.parametrize("ty,name", [(G.Q8_0, "q8_0"), (G.Q4_K, "q4_K")])
@pytest.mark.parametrize("rows,n", [(1, 256), (300, 256), (1025, 4096), (5000, 4096), (7, 1 << 20)])
def test_quantize_rows_in_pieces(oracle, ty, name, rows, n):
    native = Native(0)
    x = np.random.default_rng(rows).standard_normal((rows, n)).astype(np.float32)
    got = quantize_rows(native, ty, x)
    plain = np.zeros_like(np.empty(got.shape, np.uint8))        # ordinary memory takes the staged way down
    check(native.L.tlb_quantize_rows(native.dev, ty, x.ctypes.data_as(C.c_void_p), rows, n, plain.ctypes.data_as(C.c_void_p)))
    assert np.array_equal(got, plain)
    some = np.unique(np.concatenate([[0, rows - 1], np.random.default_rng(1).integers(0, rows, 40)]))
    assert np.array_equal(got[some], oracle.quantize(ty, x[some]))
    native.close()


def test_programs_of_many_sizes_come_and_go():
    """Arenas and inputs of up to 4 MB are cut from slabs of 16 MB, two at most; what does not fit there, and larger ones, are blocks of
    their own. Programs that live side by side share no bytes, in whatever order they come and go, and the memory goes back with the device."""
    import torch

    def cycle(rounds):
        rng = np.random.default_rng(rounds)
        native = Native.load([])
        live = []
        for _ in range(rounds):
            for _ in range(int(rng.integers(1, 8))):
                n = int(rng.choice([1, 100, 70001, 300000, 524288, 1048448, 1048576, 1048577, 1400000]))
                g = G.Graph()
                y = g.output(g.scale(g.input(G.F32, [n], "x"), 2.0))
                prog = NativeProgram.compile(native, g)
                a = rng.integers(-1000, 1000, n).astype(np.float32)
                prog.set_input(0, a)
                prog.enqueue()
                live.append((prog, y, a))
            for prog, y, a in live:
                assert np.array_equal(prog.read(y).reshape(-1), 2 * a)
            for prog, _, _ in live:     # the inputs are still there, too
                prog.enqueue()
            for i in rng.permutation(len(live))[:len(live) // 2]:
                live[i][0].free()
                live[i] = None
            live = [x for x in live if x]
            for prog, y, a in live:
                assert np.array_equal(prog.read(y).reshape(-1), 2 * a)
        for prog, _, _ in live:
            prog.free()
        native.close()

    cycle(2)
    before = torch.cuda.mem_get_info()[0]
    cycle(12)
    assert torch.cuda.mem_get_info()[0] >= before - (4 << 20)
