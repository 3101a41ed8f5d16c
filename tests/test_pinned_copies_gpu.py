"""Host-to-host steps: recorded transfers of pinned memory as kernels (small) and as copy-engine nodes (large)."""
import numpy as np
import pytest

import fastnn_b200 as fnn
from helpers import normal

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
