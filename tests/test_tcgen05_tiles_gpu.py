"""Tile edges of the tcgen05 kernels against the CPU oracle: K loops shared by a cluster of CTAs, and the two-SM tiles of
large batches.

Bars: 1e-3 of the output's RMS where the activations travel as int8 pairs (15-bit fixed point of the row) or e4m3
triples; 1e-2 for two e4m3 terms (each keeps four significant bits of what is left: 2^-8 of the row maximum) and for
fp16 operands, as for the other tests of these kernels.
"""
import numpy as np
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


# the rewrite of the rows: both sides of the lengths a thread's registers take, rows that start on 16 bytes and rows that do
# not, the last unit of eight whole, short, and followed by one of padding; the longest ones in two passes
@pytest.mark.parametrize("fmt", [orc.FMT_I8, orc.FMT_I4, orc.FMT_F8])
@pytest.mark.parametrize("k", [1028, 4096, 4099, 8196, 8209, 16388, 20002, 32768, 32777])
def test_rewritten_rows_of_any_length(backend, fmt, k):
    check(backend, fmt, k, 40, [3, 9])


# I4 rows of more than 4096 elements are shared by the blocks of a cluster from 32 rows up to a row per SM: both sides of
# those lines, whole and short last units, parts of unequal length; and up to 4096 the form of at most 32 rows
@pytest.mark.parametrize("k", [4091, 4104, 8209])
def test_rewritten_rows_by_cluster_or_by_block(backend, k):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    check(backend, orc.FMT_I4, k, 40, [31, 32, 33, sms, sms + 1])


# the cluster's longest rows: eight parts, and a last unit of one element
@pytest.mark.parametrize("k", [14336, 20009, 32768])
def test_long_rows_rewritten_by_clusters(backend, k):
    check(backend, orc.FMT_I4, k, 40, [32, 40])


def random_codes(fmt, k, n, seed):
    """A weight of random finite codes (no host quantization: these layers are large)."""
    rng = np.random.Generator(np.random.Philox(seed))
    per_word = 4 if fmt in (orc.FMT_I8, orc.FMT_F8) else 8
    words = rng.integers(0, 1 << 32, (n, -(-k // per_word)), dtype=np.uint32)
    if fmt == orc.FMT_F8:
        words &= np.uint32(0xB7B7B7B7)   # no exponent 15 (exponent bit 3 off): |v| < 2
    tail = np.zeros(16, np.uint32)
    return orc.QWeight(fmt, n, k, np.concatenate([words.ravel(), tail]), np.full(n, 0.01, np.float32),
                       np.zeros(n if fmt == orc.FMT_F4 else 0, np.float32))


# Three e4m3 terms keep 12 bits of each activation: 1.55e-5 of the output's norm at any K as long as every term has f32
# accumulators of its own (1.9e-5 at K=8192 when they share one).
@pytest.mark.parametrize("fmt", [orc.FMT_F8, orc.FMT_F4])
@pytest.mark.parametrize("k,n,m", [(8192, 18944, 100), (4096, 18944, 65), (2048, 4096, 127)])
def test_three_terms_keep_their_accuracy(backend, fmt, k, n, m):
    q = random_codes(fmt, k, n, 730 + k)
    x = normal(731 + m, (m, k), 1.0)
    rig = Rig(backend, q, m)
    try:
        got = rig.run(x, None, L.EPI_NONE, L.PATH_TC)[:, 256:512]
        row = (len(q.words) - 16) // n
        part = orc.QWeight(fmt, 256, k, np.concatenate([q.words[256 * row:512 * row], q.words[-16:]]), q.scales[256:512],
                           q.zeros[256:512])
        want = x.astype(np.float64) @ orc.dequant(part).astype(np.float64).T
        err = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert err <= 1.7e-5, (orc.FMT_NAMES[fmt], k, n, m, err)
    finally:
        rig.close()
