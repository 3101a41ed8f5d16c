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
