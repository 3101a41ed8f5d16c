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


def fold(partial):
    """What the kernels make of the threads' sums: halves of a warp on one another down to one lane, then the warps in turn."""
    lanes = partial.reshape(-1, 32)
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, np.arange(32) ^ o]
    total = np.float32(0.0)
    for s in lanes[:, 0]:
        total = np.float32(total + s)
    return total


def sum_of_units(row, threads):
    """Thread t adds the elements of its units of eight (t, t + threads, ...) one after another."""
    rounds = -(-len(row) // (8 * threads))
    units = np.zeros((rounds, threads, 8), np.float32)
    units.reshape(-1)[:len(row)] = row
    s = np.zeros(threads, np.float32)
    for i in range(rounds):
        for j in range(8):
            s = s + units[i, :, j]
    return fold(s)


def row_sums(backend, fmt, k, n, x, path, kernel):
    """The row sums that a call used: codes of zero and zero points of one leave nothing else of the product."""
    q = orc.QWeight(fmt, n, k, np.zeros(orc.packed_words(fmt, n, k), np.uint32), np.ones(n, np.float32),
                    np.ones(n, np.float32))
    rig = Rig(backend, q, len(x))
    try:
        got = rig.run(x, None, L.EPI_NONE, path)
        assert backend.last_kernel().startswith(kernel), backend.last_kernel()
        assert (got == got[:, :1]).all()
        return got[:, 0]
    finally:
        rig.close()


# whatever the number of rows, up to one per SM and more; every number of units that a thread holds; rows that start on 16
# bytes and rows that do not
@pytest.mark.parametrize("k", [4104, 6001, 14336, 20009, 28672, 28680, 32768])
def test_row_sums_of_rewritten_rows(backend, k):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = normal(930 + k, (sms + 1, k), 1.0)
    want = np.array([sum_of_units(row, 256) for row in x])
    for m in (31, 32, 64, sms, sms + 1):
        got = row_sums(backend, orc.FMT_I4, k, 24, x[:m], L.PATH_TC, "tc")
        assert (got == want[:m]).all(), (k, m)


def sum_of_quads(row, threads):
    """Thread t adds the sums of its quads (t, t + threads, ...)."""
    rounds = -(-len(row) // (4 * threads))
    quads = np.zeros((rounds, threads, 4), np.float32)
    quads.reshape(-1)[:len(row)] = row
    s = np.zeros(threads, np.float32)
    for i in range(rounds):
        s = s + ((quads[i, :, 0] + quads[i, :, 1]) + (quads[i, :, 2] + quads[i, :, 3]))
    return fold(s)


# a single long row, held or scanned (from 16384 elements on): up to a tile of 16 channels per SM by one group of warps, with
# two by two groups
@pytest.mark.parametrize("fmt", [orc.FMT_I8, orc.FMT_I4, orc.FMT_F4])
@pytest.mark.parametrize("k,tiles,threads", [(4104, 1, 256), (8192, 1, 256), (8196, 1, 256), (11008, 1, 256), (16384, 1, 256),
                                             (16388, 1, 256), (8200, 2, 512), (11008, 2, 512), (12004, 2, 512), (16384, 2, 512),
                                             (16388, 2, 512)])
def test_row_sum_of_a_long_single_row(backend, fmt, k, tiles, threads):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = normal(940 + k, (1, k), 1.0)
    got = row_sums(backend, fmt, k, 16 * tiles * sms - 5, x, L.PATH_MMA, "mma8")
    assert got[0] == sum_of_quads(x[0], threads), k
