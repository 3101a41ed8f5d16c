"""Calls of a few batch rows against the CPU oracle: rows rewritten once for all blocks, the single codebook row, the
dispatch between the kernel families, and what a capture does that finds no scratch.

Bar: 1e-3 of the output's RMS (15-bit activations, or three e4m3 terms), as for every skinny call.
"""
import ctypes

import numpy as np
import pytest

import oracle as orc
import fastnn_b200 as fnn
from fastnn_b200 import _lib as L
from helpers import max_err_vs_rms, normal
from test_kernel_choice_gpu import codes, columns
from test_qmatmul_gpu import TOL_F32, Rig
from test_tcgen05_tiles_gpu import random_codes

pytestmark = pytest.mark.gpu


# more and fewer than 16384 elements (and 8192 from five rows on); K no multiple of 16, of 8, of a k-block; more rows than fit
# beside the ring in one pass
@pytest.mark.parametrize("fmt", list(orc.FMT_NAMES))
@pytest.mark.parametrize("kn", [(1024, 70), (4100, 100), (5461, 65), (8200, 200), (20000, 64)])
def test_fragment_kernel_rows(backend, fmt, kn):
    k, n = kn
    q = orc.quantize_kn(fmt, normal(800 + k, (k, n), 0.02))
    bias = normal(801, (n,), 0.01)
    rig = Rig(backend, q, 8)
    try:
        for m in (1, 2, 3, 4, 5, 8):
            x = normal(810 + m, (m, k), 1.0)
            x[0, : k // 3] = 0.0
            got = rig.run(x, bias if m % 2 else None, L.EPI_NONE, L.PATH_MMA)
            err = max_err_vs_rms(got, orc.qmatmul(q, x, bias if m % 2 else None, L.EPI_NONE))
            assert err <= TOL_F32, (orc.FMT_NAMES[fmt], kn, m, err)
    finally:
        rig.close()


# one row: lengths on both sides of what a thread keeps of it (4096, 8192 and 16384 elements), ragged ones among them, by up to
# a tile of 16 channels per SM, more, and (I8) four: the launch shapes of the fragment kernels for a single row
@pytest.mark.parametrize("fmt,k,n", [
    (fmt, k, n) for fmt in (orc.FMT_I8, orc.FMT_I4, orc.FMT_F4, orc.FMT_I4CB, orc.FMT_F8)
    for k, n in [(4096, 200), (4097, 200), (8199, 72), (8192, 2400), (4094, 2400), (10001, 2385), (16388, 40)]
] + [(orc.FMT_I8, 520, 9488), (orc.FMT_I4, 520, 9488)])
def test_single_row_launches(backend, fmt, k, n):
    q = orc.quantize_kn(fmt, normal(850 + k, (k, n), 0.02))
    bias = normal(851, (n,), 0.01)
    rig = Rig(backend, q, 1)
    try:
        x = normal(852 + n, (1, k), 1.0)
        got = rig.run(x, bias, L.EPI_NONE, L.PATH_MMA)
        err = max_err_vs_rms(got, orc.qmatmul(q, x, bias, L.EPI_NONE))
        assert err <= TOL_F32, (orc.FMT_NAMES[fmt], k, n, err)
    finally:
        rig.close()


# both sides of the lines that automatic dispatch draws by format, rows, K and size of the weights
@pytest.mark.parametrize("fmt,k,n,m,tc", [
    (orc.FMT_I8, 4096, 2304, 4, False), (orc.FMT_I8, 4096, 2304, 5, True), (orc.FMT_I8, 1024, 512, 8, False),
    (orc.FMT_I4, 4096, 512, 8, False), (orc.FMT_I4, 14336, 512, 4, True), (orc.FMT_I4, 14336, 512, 3, False),
    (orc.FMT_F4, 4096, 4352, 4, False), (orc.FMT_F4, 4096, 4352, 5, True), (orc.FMT_F4, 1024, 512, 9, True),
    (orc.FMT_F8, 4096, 512, 8, False), (orc.FMT_I4CB, 4096, 512, 12, False), (orc.FMT_I4CB, 4096, 512, 13, True)])
def test_dispatch_of_few_rows(backend, fmt, k, n, m, tc):
    q = orc.quantize_kn(fmt, normal(820 + k, (k, n), 0.02))
    rig = Rig(backend, q, m)
    try:
        x = normal(821 + m, (m, k), 1.0)
        got = rig.run(x)
        assert (backend.last_path() == "tc") == tc
        narrow = fmt == orc.FMT_I4CB and tc   # fp16 operands
        assert max_err_vs_rms(got, orc.qmatmul(q, x)) <= (1e-2 if narrow else TOL_F32)
    finally:
        rig.close()


@pytest.mark.parametrize("fmt,k,n,m", [(orc.FMT_I8, 4096, 2304, 8), (orc.FMT_I4, 14336, 256, 4), (orc.FMT_I4, 8192, 256, 4)])
def test_capture_without_scratch(fmt, k, n, m):
    """A first call inside a capture cannot grow the scratch buffer: it runs on the kernels that need none."""
    fresh = fnn.CudaBackend(0)
    lib = fresh.lib
    q = orc.quantize_kn(fmt, normal(830 + k, (k, n), 0.02))
    rig = Rig(fresh, q, m)
    g = ctypes.c_void_p()
    try:
        assert lib.fnn_cuda_qweight_prepare(fresh.ctx, rig.w.handle, L.PATH_MMA) == 0, L.last_error()
        x = normal(831, (m, k), 1.0)
        fresh.write_arena(rig.arena, rig.a_off, x.tobytes())
        assert lib.fnn_cuda_graph_begin(fresh.ctx) == 0
        rc = lib.fnn_cuda_qmatmul(fresh.ctx, rig.w.handle, rig.arena.handle, rig.a_off, rig.out_off, -1, m, L.EPI_NONE,
                                  L.PATH_AUTO)
        assert lib.fnn_cuda_graph_end(fresh.ctx, ctypes.byref(g)) == 0
        assert rc == 0, L.last_error()
        assert lib.fnn_cuda_graph_launch(fresh.ctx, g) == 0
        fresh.synchronize()
        got = np.frombuffer(fresh.read_arena(rig.arena, rig.out_off, m * n * 4), np.float32).reshape(m, n)
        assert max_err_vs_rms(got, orc.qmatmul(q, x)) <= TOL_F32
    finally:
        if g:
            lib.fnn_cuda_graph_free(g)
        rig.close()


@pytest.mark.parametrize("fmt,k,n,m", [(orc.FMT_I8, 4096, 2304, 8), (orc.FMT_I4, 14336, 256, 4), (orc.FMT_I4, 8192, 256, 4),
                                       (orc.FMT_F4, 4096, 4352, 5), (orc.FMT_F8, 4096, 512, 40)])
def test_own_stream_captured_without_scratch(fmt, k, n, m):
    """The same for a program that captures the stream it gave the context; what needs scratch all the same gets it."""
    import torch
    stream = torch.cuda.Stream()
    fresh = fnn.CudaBackend(0, stream=stream.cuda_stream)
    lib = fresh.lib
    q = orc.quantize_kn(fmt, normal(840 + k, (k, n), 0.02))
    rig = Rig(fresh, q, m)
    graph = torch.cuda.CUDAGraph()
    try:
        assert lib.fnn_cuda_qweight_prepare(fresh.ctx, rig.w.handle, L.PATH_MMA) == 0, L.last_error()
        x = normal(841, (m, k), 1.0)
        fresh.write_arena(rig.arena, rig.a_off, x.tobytes())
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            rc = lib.fnn_cuda_qmatmul(fresh.ctx, rig.w.handle, rig.arena.handle, rig.a_off, rig.out_off, -1, m,
                                      L.EPI_NONE, L.PATH_AUTO)
        assert rc == 0, L.last_error()
        with torch.cuda.stream(stream):
            graph.replay()
        fresh.synchronize()
        got = np.frombuffer(fresh.read_arena(rig.arena, rig.out_off, m * n * 4), np.float32).reshape(m, n)
        assert max_err_vs_rms(got, orc.qmatmul(q, x)) <= TOL_F32
    finally:
        del graph
        rig.close()
        fresh.close()


# one FP8 row of at least eight tiles of 16 channels per SM and a ragged last one: two small blocks per SM up to 8192 elements,
# one larger one beyond
@pytest.mark.parametrize("k", [4104, 8192, 8200])
def test_single_fp8_row_in_front_of_many_tiles(backend, k):
    import torch
    n = 8 * 16 * torch.cuda.get_device_properties(0).multi_processor_count + 5
    q = random_codes(orc.FMT_F8, k, n, 860 + k)
    x, bias = normal(861, (1, k), 1.0), normal(862, (n,), 0.01)
    rig = Rig(backend, q, 1)
    try:
        got = rig.run(x, bias, L.EPI_NONE, L.PATH_MMA)
        assert backend.last_kernel() == "mma"
        for lo, hi in ((0, 130), (n - 150, n)):
            err = max_err_vs_rms(got[:, lo:hi], orc.qmatmul(columns(q, lo, hi), x, bias[lo:hi], L.EPI_NONE))
            assert err <= TOL_F32, (k, lo, err)
    finally:
        rig.close()


# launch shapes by tiles of 16 channels per SM and length: the codebook's single row on both sides of its lines, FP4 a little over
# a tile per SM; several I8 rows brought by all threads; two and three rows scanned by three groups of warps
@pytest.mark.parametrize("fmt,m,k,tiles", [
    (orc.FMT_I4CB, 1, 2048, 1.1), (orc.FMT_I4CB, 1, 4096, 1.45), (orc.FMT_I4CB, 1, 2080, 2.4), (orc.FMT_I4CB, 1, 4128, 1.7),
    (orc.FMT_I4CB, 1, 8320, 1.2), (orc.FMT_I4CB, 1, 16416, 1.2), (orc.FMT_F4, 1, 4090, 1.1), (orc.FMT_F4, 1, 2056, 1.3),
    (orc.FMT_I8, 2, 8195, 1.2), (orc.FMT_I8, 4, 8208, 1.2), (orc.FMT_I8, 8, 8192, 1.9), (orc.FMT_I8, 13, 8200, 1.1),
    (orc.FMT_I8, 4, 40000, 1.1), (orc.FMT_I8, 2, 4104, 5.4), (orc.FMT_I4, 3, 5001, 5.4), (orc.FMT_F4, 2, 4104, 5.4)])
def test_launch_shapes(backend, fmt, m, k, tiles):
    import torch
    n = int(tiles * torch.cuda.get_device_properties(0).multi_processor_count) * 16 - 5
    q = codes(fmt, k, n, 870 + k)
    x, bias = normal(871 + m, (m, k), 1.0), normal(872, (n,), 0.01)
    rig = Rig(backend, q, m)
    try:
        got = rig.run(x, bias, L.EPI_NONE, L.PATH_MMA)
        backend.synchronize()
        assert backend.last_path() == "mma8"
        for lo, hi in ((0, 130), (n - 150, n)):
            err = max_err_vs_rms(got[:, lo:hi], orc.qmatmul(columns(q, lo, hi), x, bias[lo:hi], L.EPI_NONE))
            assert err <= TOL_F32, (lo, err)
    finally:
        rig.close()
