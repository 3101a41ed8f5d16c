"""Which additions `dispatch` takes into the MatMul before them, against a recording stand-in for the library: whatever the
element-wise instruction refuses or treats otherwise still reaches it."""
from types import SimpleNamespace

import numpy as np
import pytest

from fastnn_b200 import BufferSlice, CallKernel, CudaBackend, ExecutablePlan, QuantizedWeightMeta, ShapeEnv, _lib as L

M, K, N = 2, 128, 64
SIZE = 4 * M * N
A, OUT, ADD, SUM, WEIGHT, TOTAL = 0, 1024, 2048, 3072, 4096, 4096 + N * K


class RecordingLib:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return L.FNN_OK
        return call


def calls_of(add, params=(M, K, N, L.EPI_NONE)):
    backend = CudaBackend.__new__(CudaBackend)
    backend.lib, backend.ctx, backend.path = RecordingLib(), None, L.PATH_AUTO
    weight = BufferSlice(WEIGHT, N * K)
    arena = SimpleNamespace(total_bytes=TOTAL, handle=1, latched_error=None,
                            qweights={(weight.offset, weight.size): SimpleNamespace(handle=2)})
    meta = QuantizedWeightMeta(bit_width=8, scales=np.ones(N, np.float32), zero_points=np.zeros(N, np.float32),
                               shape=[N, K], fmt=L.FMT_I8)
    matmul = CallKernel("matmul_i8", [BufferSlice(A, 4 * M * K), weight], BufferSlice(OUT, SIZE), list(params), weight_meta=meta)
    backend.dispatch(ExecutablePlan([matmul, add], TOTAL), arena, ShapeEnv())
    return [name.replace("fnn_cuda_", "") for name, _ in backend.lib.calls]


def add_f32(x, y, out=BufferSlice(SUM, SIZE), **kw):
    return CallKernel("add_f32", [x, y], out, [], **kw)


RESULT, RESIDUAL = BufferSlice(OUT, SIZE), BufferSlice(ADD, SIZE)


@pytest.mark.parametrize("add", [add_f32(RESULT, RESIDUAL), add_f32(RESIDUAL, RESULT),
                                 add_f32(RESULT, BufferSlice(ADD, 2 * SIZE)),              # (its first half)
                                 add_f32(RESULT, BufferSlice(TOTAL - SIZE, SIZE + 3))])    # (a slice counts in whole elements)
def test_an_addition_to_the_whole_result_joins_the_matmul(add):
    assert calls_of(add) == ["qmatmul_add"]


@pytest.mark.parametrize("add", [
    add_f32(RESULT, BufferSlice(TOTAL - SIZE, SIZE + 4)),        # the operands' slices end outside the arena: refused
    add_f32(BufferSlice(OUT, TOTAL - OUT + 4), RESIDUAL),
    add_f32(RESULT, BufferSlice(ADD, 4 * N)),                    # a broadcast
    add_f32(RESIDUAL, RESIDUAL),
    add_f32(RESULT, RESIDUAL, BufferSlice(SUM, SIZE // 2)),
    add_f32(RESULT, RESIDUAL, param_dims=[M, N // 2]),
    CallKernel("mul_f32", [RESULT, RESIDUAL], BufferSlice(SUM, SIZE), []),
])
def test_everything_else_stays_an_instruction_of_its_own(add):
    assert calls_of(add) == ["qmatmul", "elementwise"]


def test_no_rows_stay_two_instructions():
    assert calls_of(add_f32(RESULT, BufferSlice(ADD + 1, 0), BufferSlice(SUM, 0)), (0, K, N, L.EPI_NONE)) == ["qmatmul", "elementwise"]
