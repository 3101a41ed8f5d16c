"""Tile edges of the tcgen05 kernels against the CPU oracle: K loops shared by a cluster of CTAs, and the two-SM tiles of
large batches.

Bars: 1e-3 of the output's RMS where the activations travel as int8 pairs (15-bit fixed point of the row) or e4m3
triples; 1e-2 for two e4m3 terms (each keeps four significant bits of what is left: 2^-8 of the row maximum) and for
fp16 operands, as for the other tests of these kernels.
"""
import pytest

import oracle as orc
from fastnn_b200 import _lib as L
from helpers import max_err_vs_rms, normal
from test_qmatmul_gpu import TOL_F32, TOL_TC, Rig

pytestmark = pytest.mark.gpu


def check(backend, fmt, k, n, ms):
    if fmt == orc.FMT_I4CB and k % 128:
        k += 128 - k % 128   # the tcgen05 kernels take this format in whole K blocks
    q = orc.quantize_kn(fmt, normal(700 + k + n, (k, n), 0.02))
    bias = normal(710 + n, (n,), 0.01)
    rig = Rig(backend, q, max(ms))
    try:
        for m in ms:
            x = normal(720 + m, (m, k), 1.0)
            # no activation that cuts outputs off: the bars are relative to the RMS of what is left (with a ReLU over
            # 17 outputs the RMS fell from 0.86 to 0.13, and the 15-bit activations alone are 1.8e-3 of that)
            b, epi = (bias, L.EPI_NONE) if m % 2 else (None, L.EPI_SILU)
            got = rig.run(x, b, epi, L.PATH_TC)
            backend.synchronize()   # a bounded wait that gave up would raise here
            assert backend.last_path() == "tc"
            again = rig.run(x, b, epi, L.PATH_TC)
            assert (got == again).all()   # shares of K meet in a fixed order
            narrow = (m >= 128 and fmt in (orc.FMT_F8, orc.FMT_F4)) or fmt == orc.FMT_I4CB
            err = max_err_vs_rms(got, orc.qmatmul(q, x, b, epi))
            assert err <= (TOL_TC if narrow else TOL_F32), (orc.FMT_NAMES[fmt], k, n, m, err)
    finally:
        rig.close()


# one tile and a ragged second one; K of 2 to 112 blocks, shares of unequal length
@pytest.mark.parametrize("fmt", list(orc.FMT_NAMES))
@pytest.mark.parametrize("kn", [(1280, 130), (2176, 24), (3000, 257), (8192, 100), (14336, 48)])
def test_k_shares_of_a_cluster(backend, fmt, kn):
    check(backend, fmt, *kn, [5, 8, 17, 64])


# around one pair tile (256 channels) and one CTA's half of it; around the heights of a tile in batch rows
@pytest.mark.parametrize("fmt", list(orc.FMT_NAMES))
@pytest.mark.parametrize("kn", [(128, 256), (520, 129), (777, 513), (1152, 1100)])
def test_two_sm_tiles(backend, fmt, kn):
    check(backend, fmt, *kn, [65, 127, 128, 129, 161, 257, 530])
