"""A MatMul and the addition of a residual to its result as one call against the two instructions, on every kernel that may
serve it: the same bits in both slices, whatever the slices share."""
import numpy as np
import pytest

import oracle as orc
import fastnn_b200 as fnn
from fastnn_b200 import _lib as L
from helpers import normal
from test_qmatmul_gpu import Rig, meta_of

pytestmark = pytest.mark.gpu

KERNELS = {orc.FMT_I8: "matmul_i8", orc.FMT_I4: "matmul_i4", orc.FMT_F8: "matmul_f8", orc.FMT_F4: "matmul_f4",
           orc.FMT_I4CB: "matmul_i4"}


def slots(m, k, n):
    """a | out | add | sum | weight, in floats from the start of the arena"""
    al = lambda x: -(-x // 64) * 64
    a, out = 0, al(m * k)
    add = out + al(m * n)
    return a, out, add, add + al(m * n), add + 2 * al(m * n)


# rows (K < 128), fragment kernels of one and of several rows, whole and shared tcgen05 tiles, two-SM tiles; ragged N
@pytest.mark.parametrize("fmt", list(orc.FMT_NAMES))
@pytest.mark.parametrize("m,k,n", [(3, 100, 37), (1, 1024, 600), (1, 4100, 2500), (4, 1024, 333), (7, 640, 1000),
                                   (20, 1280, 130), (64, 256, 19100), (130, 384, 1001)])
def test_sum_and_result_are_those_of_two_calls(backend, fmt, m, k, n):
    q = orc.quantize_kn(fmt, normal(900 + k, (k, n), 0.02))
    a, out, add, total, end = slots(m, k, n)
    arena = backend.allocate_arena(4 * end)
    w = backend.upload_qweight(q.payload, meta_of(q))
    try:
        def run(fused, sum_at):
            backend.write_arena(arena, 0, np.zeros(end, np.float32).tobytes())
            backend.write_arena(arena, 0, normal(901 + m, (m, k), 1.0).tobytes())
            backend.write_arena(arena, 4 * add, normal(902 + n, (m, n), 1.0).tobytes())
            args = (backend.ctx, w.handle, arena.handle, 4 * a, 4 * out, -1, m, L.EPI_SILU, L.PATH_AUTO)
            if fused:
                assert backend.lib.fnn_cuda_qmatmul_add(*args, 4 * add, 4 * sum_at) == 0, L.last_error()
            else:
                assert backend.lib.fnn_cuda_qmatmul(*args) == 0, L.last_error()
                assert backend.lib.fnn_cuda_elementwise(backend.ctx, L.EW_ADD, arena.handle, 4 * out, m * n, 4 * add, m * n,
                                                        4 * sum_at, m * n) == 0
            return np.frombuffer(backend.read_arena(arena, 0, 4 * end), np.uint32).copy()

        # a slice of its own; in place of the residual, of the result, of the activations (where they are large enough)
        for sum_at in (total, add, out) + ((a,) if k >= n else ()):
            assert (run(True, sum_at) == run(False, sum_at)).all(), sum_at
    finally:
        w.close()
        arena.close()


def test_plans_fuse_whole_residuals_only(backend):
    """One launch less where the addition takes the MatMul's whole result and an equal slice; a broadcast, another
    operand and a chain run as they stand."""
    m, k, n = 2, 512, 256
    q = orc.quantize_kn(orc.FMT_I8, normal(910, (k, n), 0.02))
    a, out, add, total, end = slots(m, k, n)
    payload = q.payload
    arena = backend.allocate_arena(4 * end + len(payload) + 256)
    f = lambda at, count: fnn.BufferSlice(4 * at, 4 * count)
    weight = fnn.BufferSlice(4 * end, len(payload))
    matmul = fnn.CallKernel("matmul_i8", [f(a, m * k), weight], f(out, m * n), [m, k, n, L.EPI_NONE], weight_meta=meta_of(q))
    try:
        backend.write_arena(arena, 4 * end, payload)
        x, r = normal(911, (m, k), 1.0), normal(912, (m, n), 1.0)

        def launches(second):
            backend.write_arena(arena, 0, x.tobytes())
            backend.write_arena(arena, 4 * add, r.tobytes())
            plan = fnn.ExecutablePlan([matmul, second], arena.total_bytes)
            backend.dispatch(plan, arena, fnn.ShapeEnv())       # (first use builds the layouts)
            before = backend.launch_count()
            backend.dispatch(plan, arena, fnn.ShapeEnv())
            got = np.frombuffer(backend.read_arena(arena, 4 * total, 4 * m * n), np.float32).reshape(m, n)
            y = np.frombuffer(backend.read_arena(arena, 4 * out, 4 * m * n), np.float32).reshape(m, n)
            return backend.launch_count() - before, y, got

        for ins in ([f(out, m * n), f(add, m * n)], [f(add, m * n), f(out, m * n)]):
            count, y, got = launches(fnn.CallKernel("add_f32", ins, f(total, m * n), []))
            assert count == 1 and (got == y + r).all()
        count, y, got = launches(fnn.CallKernel("add_f32", [f(out, m * n), f(add, n)], f(total, m * n), []))
        assert count == 2 and (got == y + r[0]).all()
        count, y, got = launches(fnn.CallKernel("add_f32", [f(add, m * n), f(add, m * n)], f(total, m * n), []))
        assert count == 2 and (got == r + r).all()
        count, y, got = launches(fnn.CallKernel("mul_f32", [f(out, m * n), f(add, m * n)], f(total, m * n), []))
        assert count == 2 and (got == y * r).all()
    finally:
        arena.close()


# where the guards between the slices decide: one or two fragment rows, shared and whole tcgen05 tiles
@pytest.mark.parametrize("m,k,n", [(1, 1024, 608), (4, 1024, 336), (20, 1280, 144), (64, 256, 19104)])
def test_slices_that_may_not_be_written_by_one_epilogue(backend, m, k, n):
    """One launch where the slices allow it; one more where the sum lies over something that the MatMul or the addition still
    reads, or the residual over the result.  Both ways the bits are those of the two calls."""
    q = orc.quantize_kn(orc.FMT_I8, normal(920 + k, (k, n), 0.02))
    al = lambda x: -(-x // 64) * 64
    size, payload = m * n, q.payload
    a, out = 0, al(m * k)
    add = out + al(size) + 64
    total = add + al(size) + al(size) + 64
    bias = total + al(size) + 64
    weight = bias + al(size) + al(n)          # (a sum that begins over the bias ends ahead of the rows)
    end = weight + max(len(payload) // 4, size + 64) + 64
    arena = backend.allocate_arena(4 * end)
    first = np.zeros(end, np.float32)
    first[a:a + m * k], first[add:add + size] = normal(921, (m * k,), 1.0), normal(922, (size,), 1.0)
    first[bias:bias + n] = normal(923, (n,), 0.1)
    raw = bytearray(first.tobytes())
    raw[4 * weight:4 * weight + len(payload)] = payload
    raw = bytes(raw)
    backend.write_arena(arena, 0, raw)
    w = backend.upload_qweight(b"", meta_of(q), arena, 4 * weight, len(payload))   # (its rows stay where they are)
    try:
        def run(fused, add_at, sum_at):
            backend.write_arena(arena, 0, raw)
            before = backend.launch_count()
            args = (backend.ctx, w.handle, arena.handle, 4 * a, 4 * out, 4 * bias, m, L.EPI_SILU, L.PATH_AUTO)
            if fused:
                assert backend.lib.fnn_cuda_qmatmul_add(*args, 4 * add_at, 4 * sum_at) == 0, L.last_error()
            else:
                assert backend.lib.fnn_cuda_qmatmul(*args) == 0, L.last_error()
                assert backend.lib.fnn_cuda_elementwise(backend.ctx, L.EW_ADD, arena.handle, 4 * out, size, 4 * add_at, size,
                                                        4 * sum_at, size) == 0
            launches = backend.launch_count() - before
            return launches, np.frombuffer(backend.read_arena(arena, 0, 4 * end), np.uint32).copy()

        run(True, add, total)                      # first use: layouts, scratch
        two = run(False, add, total)[0]
        for add_at, sum_at, apart in [(add, total, False), (add, add, False),
                                      (out, total, True), (out + 4, total, True),   # the residual over the result
                                      (add, out, True),                             # the sum over the result
                                      (add, bias, True), (add, bias + n - 4, True),
                                      (add, weight, True), (add, weight + 8, True)] + (
                                      [(add, a + 4, True)] if size + 4 <= out else []):
            count, got = run(True, add_at, sum_at)
            assert count == two - (not apart), (add_at, sum_at)
            assert (got == run(False, add_at, sum_at)[1]).all(), (add_at, sum_at)
        # half over the residual, ahead of it and behind it, and half over the result: an addition whose operand is overwritten
        # as it runs, so what it makes of the overlap is open, but not what lies beside the two slices
        for over, sum_at in ((add, add + 4), (add, add + size // 8 * 4), (add, add - 4), (out, out + 4)):
            count, got = run(True, add, sum_at)
            assert count == two, sum_at
            plain = run(False, add, sum_at)[1]
            lo, hi = min(over, sum_at), max(over, sum_at) + size
            assert (got[:lo] == plain[:lo]).all() and (got[hi:] == plain[hi:]).all(), sum_at
    finally:
        w.close()
        arena.close()
