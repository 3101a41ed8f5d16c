"""Host-to-host steps: recorded transfers of pinned memory as kernels (small) and as copy-engine nodes (large)."""
import numpy as np
import pytest

import oracle as orc
import fastnn_b200 as fnn
from fastnn_b200 import _lib as L
from helpers import max_err_vs_rms, normal

pytestmark = pytest.mark.gpu


# outputs of a whole number of 16-byte units, of 4-byte units only, and above the size that a kernel moves
@pytest.mark.parametrize("m,n", [(1, 512), (3, 1001), (130, 1001)])
def test_pinned_step_equals_plain_step(m, n):
    k = 512
    nodes = [{"op_type": "MatMul", "inputs": "[x, w]", "outputs": "[y]"}]
    ex = fnn.AotExecutor(nodes, {"w": normal(870, (k, n), 0.02)}, ["x"], ["y"], {"x": [m, k]}, quantize=8,
                         backend=fnn.CudaBackend(0))
    a, b = normal(871, (m, k), 1.0), normal(872, (m, k), 1.0)
    want = [np.array(ex.forward({"x": v})["y"]) for v in (a, b)]
    ex.bind_pinned()
    for v, w in ((a, want[0]), (b, want[1]), (a, want[0])):
        ex.pinned_inputs["x"][...] = v
        assert np.array_equal(np.asarray(ex.forward_pinned()["y"]).reshape(w.shape), w)


# A bias that is an input of the plan is written by the recorded copy just before the matmul: every step has to see
# its own.  The 8-bit and the fp16 fragment kernel, one row and several (rewritten inside the kernel and before it).
@pytest.mark.parametrize("quantize", [8, "f8"])
@pytest.mark.parametrize("m,k", [(1, 512), (4, 512), (4, 4608)])
def test_runtime_bias_changes_every_step(quantize, m, k):
    n = 1000
    nodes = [{"op_type": "MatMul", "inputs": "[x, w]", "outputs": "[h]"},
             {"op_type": "Add", "inputs": "[h, b]", "outputs": "[s]"},
             {"op_type": "Relu", "inputs": "[s]", "outputs": "[y]"}]
    ex = fnn.AotExecutor(nodes, {"w": normal(873, (k, n), 0.02)}, ["x", "b"], ["y"], {"x": [m, k], "b": [n]},
                         quantize=quantize, backend=fnn.CudaBackend(0))
    steps = [{"x": normal(880 + i, (m, k), 1.0), "b": normal(890 + i, (n,), 1.0)} for i in range(4)]
    want = [np.array(ex.forward(step)["y"]) for step in steps]
    ex.bind_pinned()
    for _ in range(25):
        for step, w in zip(steps, want):
            for name, v in step.items():
                ex.pinned_inputs[name][...] = v
            assert np.array_equal(np.asarray(ex.forward_pinned()["y"]).reshape(w.shape), w)


# The same for the weight of a norm.
def test_runtime_norm_weight_changes_every_step():
    m, k = 3, 1024
    nodes = [{"op_type": "RMSNorm", "inputs": "[x, g]", "outputs": "[y]"}]
    ex = fnn.AotExecutor(nodes, {}, ["x", "g"], ["y"], {"x": [m, k], "g": [k]}, backend=fnn.CudaBackend(0))
    steps = [{"x": normal(900 + i, (m, k), 1.0), "g": normal(910 + i, (k,), 1.0)} for i in range(4)]
    want = [np.array(ex.forward(step)["y"]) for step in steps]
    ex.bind_pinned()
    for _ in range(25):
        for step, w in zip(steps, want):
            for name, v in step.items():
                ex.pinned_inputs[name][...] = v
            assert np.array_equal(np.asarray(ex.forward_pinned()["y"]).reshape(w.shape), w)


def test_recorded_copy_into_a_weight_used_in_place():
    """The tcgen05 kernel requests its weights before it waits for the kernel ahead of it: a recorded copy into them has to
    order what follows all the same."""
    import ctypes
    k, n, m = 512, 256, 16
    be = fnn.CudaBackend(0)
    lib = be.lib
    qs = [orc.quantize_kn(orc.FMT_I8, normal(920 + i, (k, n), 0.02)) for i in range(2)]
    qs[1].scales[:], qs[1].zeros[:] = qs[0].scales, qs[0].zeros   # the weight object keeps the first one's
    x = normal(922, (m, k), 1.0)
    want = [orc.qmatmul(q, x) for q in qs]
    rows = n * k
    arena = be.allocate_arena(rows + 4096 + (m * k + m * n) * 4)
    a_off, out_off = rows + 4096, rows + 4096 + m * k * 4
    be.write_arena(arena, 0, qs[0].payload)
    be.write_arena(arena, a_off, x.tobytes())
    meta = fnn.QuantizedWeightMeta(bit_width=8, scales=qs[0].scales, zero_points=qs[0].zeros, shape=[n, k],
                                   quant_block_size=0, codebooks=[], fmt=orc.FMT_I8)
    w = be.upload_qweight(b"", meta, arena, 0, len(qs[0].payload))
    host = ctypes.c_void_p()
    g = ctypes.c_void_p()
    assert lib.fnn_cuda_host_alloc(rows, ctypes.byref(host)) == 0
    try:
        def call():
            assert lib.fnn_cuda_arena_write_async(arena.handle, 0, host, rows) == 0, L.last_error()
            assert lib.fnn_cuda_qmatmul(be.ctx, w.handle, arena.handle, a_off, out_off, -1, m, L.EPI_NONE,
                                        L.PATH_TC) == 0, L.last_error()
        ctypes.memmove(host, qs[0].payload, rows)
        call()
        be.synchronize()
        assert lib.fnn_cuda_graph_begin(be.ctx) == 0
        call()
        assert lib.fnn_cuda_graph_end(be.ctx, ctypes.byref(g)) == 0
        for i in range(60):
            ctypes.memmove(host, qs[i & 1].payload, rows)
            assert lib.fnn_cuda_graph_launch(be.ctx, g) == 0
            be.synchronize()
            got = np.frombuffer(be.read_arena(arena, out_off, m * n * 4), np.float32).reshape(m, n)
            assert max_err_vs_rms(got, want[i & 1]) <= 1e-3
    finally:
        if g:
            lib.fnn_cuda_graph_free(g)
        lib.fnn_cuda_host_free(host)
        w.close()
        arena.close()
        be.close()
