"""The order in which f32 sums are taken, to the last bit: it depends neither on the number of batch rows nor on how the work is
spread over blocks, so that a stack of layers, whose rewrites round what the layer before stored, repeats itself."""
import numpy as np
import pytest

import oracle as orc
from fastnn_b200 import _lib as L
from helpers import normal
from test_qmatmul_gpu import Rig

pytestmark = pytest.mark.gpu


# shares of a K loop in six parts: -2, 3 and 2^24 lie in the first, a middle and the last part, and the others are zero.  The CTA that
# finishes a chunk adds the shares behind its own from the first on: 2^24 wherever its own one stands, but 2^24 + 2
# if 3 and 2^24 meet before the -2
def test_shares_of_a_cluster_meet_from_the_first_on(backend):
    k, n, m = 8192, 2048, 64
    book = np.linspace(-1.0, 1.0, 16, dtype=np.float32)     # (code 15 is 1)
    q = orc.QWeight(orc.FMT_I4CB, n, k, np.full(n * (k // 8) + 16, 0xFFFFFFFF, np.uint32),
                    np.ones(n * (k // 32), np.float32), np.zeros(0, np.float32), book, 32)
    rig = Rig(backend, q, m)
    try:
        x = np.zeros((m, k), np.float32)
        x[:, 0], x[:, k // 2], x[:, k - 1] = -2.0, 3.0, 2.0 ** 24
        got = rig.run(x, None, L.EPI_NONE, L.PATH_TC)
        assert backend.last_kernel() == "tc-split"
        assert (got == np.float32(2.0 ** 24)).all(), np.unique(got)
    finally:
        rig.close()
