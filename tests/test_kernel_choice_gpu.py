"""Every instantiation of the two-SM kernel, and the other kernels beside it, at shapes that automatic dispatch gives them,
against the CPU oracle on slices of output channels (the first ones and the ragged last tile).

Weights are random codes.  Bars as in test_tcgen05_tiles_gpu.py.
"""
import numpy as np
import pytest

import oracle as orc
from fastnn_b200 import _lib as L
from helpers import max_err_vs_rms, normal
from test_qmatmul_gpu import TOL_F32, TOL_TC, Rig
from test_tcgen05_tiles_gpu import random_codes

pytestmark = pytest.mark.gpu


def codes(fmt, k, n, seed):
    if fmt != orc.FMT_I4CB:
        q = random_codes(fmt, k, n, seed)
        if fmt in (orc.FMT_I8, orc.FMT_I4):
            q.zeros = normal(seed + 1, (n,), 0.002)
        return q
    rng = np.random.Generator(np.random.Philox(seed))
    words = rng.integers(0, 1 << 32, n * (k // 8) + 16, dtype=np.uint32)
    book = np.linspace(-1.0, 1.0, 16, dtype=np.float32)
    return orc.QWeight(fmt, n, k, words, rng.uniform(0.01, 0.03, n * (k // 32)).astype(np.float32),
                       np.zeros(0, np.float32), book, 32)


def columns(q, lo, hi):
    row = (len(q.words) - 16) // q.n
    per = len(q.scales) // q.n
    return orc.QWeight(q.fmt, hi - lo, q.k, np.concatenate([q.words[lo * row:hi * row], q.words[-16:]]),
                       q.scales[lo * per:hi * per], q.zeros[lo:hi] if len(q.zeros) else q.zeros, q.codebook,
                       q.quant_block_size)


# (a B200 has 74 pairs of SMs: with more tiles than that, a pair runs a second one)
@pytest.mark.parametrize("fmt,k,n,m,kernel", [
    # codebook: one tile per pair with a ragged last one, heights 160 and 192; two waves of 256 rows
    (orc.FMT_I4CB, 640, 4100, 530, "tc-pair"), (orc.FMT_I4CB, 2048, 4300, 700, "tc-pair"),
    (orc.FMT_I4CB, 4096, 14336, 512, "tc-pair"), (orc.FMT_I4CB, 512, 8320, 674, "tc"),
    (orc.FMT_I4CB, 1024, 2048, 129, "tc-split"),
    # three terms: heights 32 and 64, K of many blocks and not of whole ones, one and two waves
    (orc.FMT_F8, 1032, 9500, 65, "tc-pair"), (orc.FMT_F4, 1032, 12100, 127, "tc-pair"),
    (orc.FMT_F4, 1160, 9000, 127, "tc-pair"), (orc.FMT_F8, 2050, 8200, 100, "tc-pair"),
    # two terms: int8 pairs and e4m3 pairs, two waves; the tallest tile
    (orc.FMT_I4, 520, 8200, 300, "tc-pair"), (orc.FMT_I4, 1160, 9400, 512, "tc-pair"),
    (orc.FMT_I8, 1032, 8200, 300, "tc-pair"), (orc.FMT_I8, 2056, 5000, 512, "tc-pair"),
    (orc.FMT_F8, 1160, 8200, 300, "tc-pair"), (orc.FMT_F4, 2056, 5000, 512, "tc-pair"),
    # below the pair kernel's line, and a split of K
    (orc.FMT_I8, 1160, 9400, 256, "tc"), (orc.FMT_I8, 8192, 2048, 17, "tc-split")])
def test_kernel_and_result(backend, fmt, k, n, m, kernel):
    q = codes(fmt, k, n, 1000 + k + m)
    x, bias = normal(1001 + m, (m, k), 1.0), normal(1002, (n,), 0.01)
    rig = Rig(backend, q, m)
    try:
        got = rig.run(x, bias, L.EPI_NONE)
        backend.synchronize()   # a bounded wait that gave up would raise here
        assert backend.last_kernel() == kernel
        narrow = fmt == orc.FMT_I4CB or (fmt in (orc.FMT_F8, orc.FMT_F4) and m >= 128)
        for lo, hi in ((0, 130), (n - 150, n)):
            err = max_err_vs_rms(got[:, lo:hi], orc.qmatmul(columns(q, lo, hi), x, bias[lo:hi], L.EPI_NONE))
            assert err <= (TOL_TC if narrow else TOL_F32), (lo, hi, err)
        assert np.array_equal(rig.run(x, bias, L.EPI_NONE), got)
    finally:
        rig.close()


# codebook tiles on both sides of the number that runs as clusters of three
@pytest.mark.parametrize("n", [5500, 5504, 5505, 5700, 5769])
def test_codebook_tiles_around_the_clusters_of_three(backend, n):
    k, m = 2944, 48
    q = codes(orc.FMT_I4CB, k, n, 1100)
    x, bias = normal(1101, (m, k), 1.0), normal(1102, (n,), 0.01)
    rig = Rig(backend, q, m)
    try:
        got = rig.run(x, bias, L.EPI_NONE, L.PATH_TC)
        backend.synchronize()
        for lo, hi in ((0, 130), (n - 150, n)):
            err = max_err_vs_rms(got[:, lo:hi], orc.qmatmul(columns(q, lo, hi), x, bias[lo:hi], L.EPI_NONE))
            assert err <= TOL_TC, (lo, err)
    finally:
        rig.close()
