// tcgen05 kernel for large batches: two SMs of a cluster work on one tile (cta_group::2).
//
// Bound by the tensor pipe.  A single-SM tile of 128 output channels x 256 accumulator columns moves
// 16 KB of weights and 32 KB of activations through L2 and shared memory for every 512 cycles of
// MMA (94 B per cycle and SM, 27 TB/s over the chip at the full 8-bit rate), which L2 cannot feed.  Here the
// pair computes 256 channels: each SM holds its own 128 weight rows and half of the activation tile,
// and the tensor cores of both read both halves, so the activation traffic of an SM halves.
//
// Each narrow term of an activation (see qmm_tc.cu) has accumulator columns of its own: one MMA per K step over the
// (term, batch row) columns, a multiple of 32 and at most 256 of them, each SM holding half.  One term (codebook): half
// of the batch rows each; two: a plane each; three: a plane and half of the middle one (64 B per cycle and SM
// at 256 columns).  A form that let the terms of FP8 and FP4 meet in the same columns moved fewer bytes, but its f32
// accumulators take two or three times the additions: error 1.65e-5 against 1.56e-5 at M=96 K=4096, 1.9e-5 against
// 1.5e-5 at K=8192.
//
// Weight formats, warp roles, TMEM double buffering and the epilogue arithmetic are those of qmm_tc.cu.
// Differences: the MMA issuer runs in the pair's first CTA only; the operand copies of both CTAs
// report to that CTA's `full` barrier; commits arrive at both CTAs' `empty` and `tfull` barriers.
// Every mbarrier wait is bounded; both CTAs meet at a cluster barrier before either exits, so no
// arrival can reach the shared memory of a CTA that is gone.
#include "tc_common.cuh"

#include <algorithm>

namespace fnn {

namespace {

using namespace tc;

constexpr int kPairRows = 2 * kTileN;   // output channels per pair tile

// ---- PTX wrappers of the two-SM forms -----------------------------------------------------------

// Arrival at the first CTA's barrier.  What it announces is never read through the generic proxy by the
// waiting thread: TMEM columns that tcgen05.ld has finished reading, operand tiles handed to the
// async proxy by fence.proxy.async.  Waits therefore acquire at CTA scope: an acquire at cluster scope also
// invalidates L1, and in the step loop that cost more than the step (0.6 us against 0.25).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Copies into this CTA's shared memory that report to a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void *dst, const CUtensorMap *map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map, uint32_t bar, int c0, int c1,
                                                 int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// Arrives at the barrier of this offset in both CTAs once the MMAs issued so far have finished.
__device__ __forceinline__ void tc_commit_pair(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
            smem_u32(bar)),
        "h"((uint16_t)3)
        : "memory");
}
template <int KIND>
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
    if (KIND == KIND_I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else if (KIND == KIND_F8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

struct PairParams {
    const float *scales;
    const float *zeros;
    const float *bias;
    const float *dq;
    const float *rowsum;
    const float *codebook;   // WF_CB: 16 centroids
    float *out;
    const float *add;   // sum = out + add, where sum is given
    float *sum;
    int *err_flag;
    int M, N;
    int Mb;        // batch rows per tile
    int n_tiles, m_tiles;   // tiles of 256 channels, of Mb batch rows
    int kblocks;
    int a_fmt;
    float acc_scale;
    int stages;
    int epilogue;
};

template <int KIND, int T, int WF>
__global__ void __launch_bounds__((2 + kEpiWarps + xf_warps(WF)) * 32, 1)
qmm_tc_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                   const __grid_constant__ CUtensorMap map_s, PairParams p) {
    constexpr int ATOMS = (KIND == KIND_F16) ? 2 : 1;
    constexpr int kRawBytes = (WF == WF_TMA) ? 0 : kTileN * 64;        // packed nibbles: 64 bytes per row
    constexpr int kScBytes = (WF == WF_CB) ? kTileN * 16 : 0;          // four block scales per row
    constexpr int kXf0 = 2 + kEpiWarps;                                // first transform warp
    constexpr int kXfArrivals = 2 * xf_warps(WF);     // of both CTAs
    constexpr int a_atom = kTileN * kKBlockBytes, a_bytes = ATOMS * a_atom;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // both CTAs of the pair lay their shared memory out alike: an MMA names one offset for both
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int acc_cols = T * p.Mb;                         // accumulator columns of a tile = MMA N
    const int b_rows = T * p.Mb / 2;                       // activation rows this CTA holds per K block
    const int b_atom = b_rows * kKBlockBytes;              // (b_rows is a multiple of 8)
    const int b_bytes = ATOMS * b_atom;
    unsigned char *s_a = smem;
    unsigned char *s_b = s_a + (size_t)p.stages * a_bytes;
    unsigned char *s_raw = s_b + (size_t)p.stages * b_bytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(s_raw + (size_t)p.stages * (kRawBytes + kScBytes));
    uint64_t *full = bars, *empty = bars + p.stages, *rawfull = bars + 2 * p.stages;
    uint64_t *tfull = bars + 3 * p.stages, *tempty = tfull + 2;
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(tempty + 2);
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);
    float *s_cb = table_after(s_tmem + 2);                                // [16]

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = blockIdx.x & 1;   // clusters are pairs of consecutive blocks (a uniform value)
    pdl_launch_dependents();
    uint32_t ncols = 32;
    while ((int)ncols < 2 * acc_cols) ncols <<= 1;
    const int total_tiles = p.n_tiles * p.m_tiles;
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_a);
        if (WF == WF_CB) prefetch_tensormap(&map_s);
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1 + kXfArrivals);   // (the first CTA's is the one in use)
            mbar_init(&empty[s], 1);
            mbar_init(&rawfull[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], 2 * kEpiWarps);   // (the first CTA's is the one in use)
        }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (WF == WF_CB && threadIdx.x >= 64 && threadIdx.x < 80) s_cb[threadIdx.x - 64] = p.codebook[threadIdx.x - 64];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the other CTA's barriers exist
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem;

    if (warp == 0) {
        // ---------------- TMA producer (one in each CTA, for its own halves) ----------------
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            // bytes that both CTAs' copies of a stage report to the first CTA's barrier (the unpacking
            // 4-bit tensor-map type counts the packed source bytes)
            const uint32_t full_tx = 2u * (uint32_t)((WF == WF_TMA ? (p.a_fmt == kFmtE2M1 ? a_bytes / 2 : a_bytes) : 0) + b_bytes);
            auto load_w = [&](int st, int nt, int kb) {
                const int n0 = nt * kPairRows + (int)rank * kTileN;
                if (WF == WF_TMA) {
                    const uint32_t bar = mapa(&full[st], 0);
#pragma unroll
                    for (int at = 0; at < ATOMS; ++at)
                        tma_load_2d_pair(s_a + (size_t)st * a_bytes + at * a_atom, &map_w, bar,
                                         (kb * ATOMS + at) * kKBlockBytes, n0);
                } else {
                    unsigned char *raw = s_raw + (size_t)st * (kRawBytes + kScBytes);
                    mbar_expect_tx(&rawfull[st], (uint32_t)(kRawBytes + kScBytes));
                    tma_load_2d(raw, &map_w, &rawfull[st], kb * 64, n0);
                    if (WF == WF_CB) tma_load_2d(raw + kRawBytes, &map_s, &rawfull[st], kb * 16, n0);
                }
            };
            auto load_b = [&](int st, int mt, int kb) {
                const uint32_t bar = mapa(&full[st], 0);
                // This CTA's half of the (term, batch row) columns: plane `rank` for two terms, else T of the 2 T
                // halves of planes.
#pragma unroll
                for (int at = 0; at < ATOMS; ++at)
#pragma unroll
                    for (int i = 0; i < (T == 2 ? 1 : T); ++i) {
                        const int h = (int)rank * T + i;
                        const int row = mt * p.Mb + (T == 2 ? 0 : (h & 1) * (p.Mb / 2)), plane = T == 2 ? (int)rank : h >> 1;
                        tma_load_3d_pair(s_b + (size_t)st * b_bytes + at * b_atom + i * (p.Mb / 2) * kKBlockBytes, &map_a,
                                         bar, (kb * ATOMS + at) * kKBlockBytes, row, plane);
                    }
            };
            // the first ring of weight tiles does not depend on the kernel before this one
            int head = 0;
            if (pair < total_tiles) {
                head = min(p.stages, p.kblocks);
                for (int i = 0; i < head; ++i) {
                    if (rank == 0) mbar_expect_tx(&full[i], full_tx);
                    load_w(i, pair / p.m_tiles, i);
                }
            }
            pdl_wait();
            for (int i = 0; i < head; ++i) load_b(i, pair % p.m_tiles, i);
            s = head;
            if (s == p.stages) {
                s = 0;
                phase = 1;
            }
            for (int tile = pair; tile < total_tiles && ok; tile += pairs) {
                const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
                for (int kb = (tile == pair ? head : 0); kb < p.kblocks; ++kb) {
                    if (!mbar_wait(&empty[s], phase ^ 1, s_abort, p.err_flag, 0x10)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0) mbar_expect_tx(&full[s], full_tx);
                    load_w(s, nt, kb);
                    load_b(s, mt, kb);
                    if (++s == p.stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) {  // let copies already in flight land before the CTA can exit
                for (int i = 0; i < 64; ++i) __nanosleep(1000);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (first CTA) ----------------
        if (rank == 0) if (elect_one()) {
            const uint32_t idesc = make_idesc(KIND, acc_cols, p.a_fmt, kPairRows);
            int s = 0;
            uint32_t phase = 0;
            int as = 0;
            uint32_t aphase = 0;
            bool ok = true;
            for (int tile = pair; tile < total_tiles && ok; tile += pairs) {
                if (!mbar_wait(&tempty[as], aphase ^ 1, s_abort, p.err_flag, 0x20)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(as * acc_cols);
                for (int kb = 0; kb < p.kblocks; ++kb) {
                    if (!mbar_wait(&full[s], phase, s_abort, p.err_flag, 0x40)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int at = 0; at < ATOMS; ++at) {
                        const uint64_t da = make_desc_sw128(smem_u32(s_a + (size_t)s * a_bytes + at * a_atom));
                        const uint64_t db = make_desc_sw128(smem_u32(s_b + (size_t)s * b_bytes + at * b_atom));
#pragma unroll
                        for (int k = 0; k < kKBlockBytes / 32; ++k)
                            tc_mma_pair<KIND>(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc,
                                              (kb > 0 || at > 0 || k > 0) ? 1u : 0u);
                    }
                    tc_commit_pair(&empty[s]);
                    if (++s == p.stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                tc_commit_pair(&tfull[as]);
                if (++as == 2) {
                    as = 0;
                    aphase ^= 1;
                }
            }
        }
    } else if (WF != WF_TMA && warp >= kXf0) {
        // ---------------- transform warps (each CTA widens its own weight rows) ----------------
        const int xt = threadIdx.x - kXf0 * 32;
        int s = 0;
        uint32_t phase = 0;
        bool filled = true;
        for (int tile = pair; tile < total_tiles; tile += pairs) {
            for (int kb = 0; kb < p.kblocks; ++kb) {
                // (A lane that gives up stays with its warp through this step and the others, whatever the stages hold, and reports
                // no stage any more.  A vote, which ends the loop for all, cost 1 % of a decoder step, and so did a branch here.)
                const bool here = mbar_wait(&rawfull[s], phase, s_abort, p.err_flag, 0x200);
                const unsigned char *raw = s_raw + (size_t)s * (kRawBytes + kScBytes);
                unsigned char *dst = s_a + (size_t)s * a_bytes;
#pragma unroll
                for (int it = 0; it < (WF == WF_TMA ? 0 : (kTileN * 4) / (xf_warps(WF == WF_TMA ? WF_I4 : WF) * 32)); ++it) {
                    // a 16-byte unit of a row -> its place in the 128-byte-swizzled operand tile
                    const int item = xt + it * xf_warps(WF) * 32, row = item >> 2, c = item & 3;
                    const uint4 w = *reinterpret_cast<const uint4 *>(raw + row * 64 + ((c ^ ((row >> 1) & 3)) << 4));
                    uint32_t o[16];
                    if (WF == WF_I4)
                        widen_i4(w, o);
                    else
                        widen_cb(w, *reinterpret_cast<const float *>(raw + kRawBytes + row * 16 + c * 4), smem_u32(s_cb), o);
                    unsigned char *r = dst + (WF == WF_CB ? (c >> 1) * a_atom : 0) + row * 128;
                    constexpr int kUnits = (WF == WF_CB) ? 4 : 2;   // 16-byte chunks the unit widens to
#pragma unroll
                    for (int u = 0; u < kUnits; ++u)
                        *reinterpret_cast<uint4 *>(r + ((((c * kUnits + u) & 7) ^ (row & 7)) << 4)) =
                            make_uint4(o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
                }
                fence_proxy_async();   // these stores are read by the tensor cores (async proxy)
                __syncwarp();
                filled &= here;
                if (lane == 0 && filled) mbar_arrive_cluster(mapa(&full[s], 0));
                if (++s == p.stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp < kXf0) {
        // ---------------- epilogue (each CTA: its own 128 channels) ----------------
        pdl_wait();   // dq, rowsum and the output buffer belong to kernels before this one
        const int quad = warp & 3;
        const int chunk0 = ((warp - 2) >> 2) * 16;
        constexpr int kStep = 16 * (kEpiWarps / 4);
        int as = 0;
        uint32_t aphase = 0;
        const bool has_zero = p.zeros != nullptr;
        const int row = quad * 32 + lane;
        auto load_rowfac = [&](int mt, int c0) -> float {
            const int j = lane & 15, m = mt * p.Mb + c0 + j;
            const bool want = c0 + j < p.Mb && m < p.M && (lane < 16 || has_zero);
            return want ? (lane < 16 ? p.dq : p.rowsum)[m] : 0.0f;
        };
        for (int tile = pair; tile < total_tiles; tile += pairs) {
            const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
            const int n = nt * kPairRows + (int)rank * kTileN + row;
            const bool n_ok = n < p.N;
            const float scale = n_ok ? (p.scales ? __ldg(p.scales + n) : 1.0f) : 0.0f;
            const float zero = (n_ok && has_zero) ? __ldg(p.zeros + n) : 0.0f;
            const float bias = (n_ok && p.bias) ? p.bias[n] : 0.0f;
            float fac = load_rowfac(mt, chunk0);
            if (!mbar_wait_warp(&tfull[as], aphase, s_abort, p.err_flag, 0x80)) break;
            tc_fence_after();
            const uint32_t t_base = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(as * acc_cols);
            for (int c0 = chunk0; c0 < p.Mb; c0 += kStep) {
                uint32_t r[T][16];
#pragma unroll
                for (int t = 0; t < T; ++t) tmem_ld16(t_base + (uint32_t)(t * p.Mb + c0), r[t]);
                const float fac_next = load_rowfac(mt, c0 + kStep);
                tmem_ld_wait();
                float v[16];
                finish_chunk<KIND, T>(r, fac, scale, zero, bias, p.bias != nullptr, p.acc_scale, p.epilogue, v);
                const int m0 = mt * p.Mb + c0;
                const int jmax = n_ok ? min(16, min(p.Mb - c0, p.M - m0)) : 0;   // rows of this chunk that exist
                store_chunk(p.out, p.add, p.sum, (size_t)m0 * p.N + n, p.N, jmax, v);
                fac = fac_next;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa(&tempty[as], 0));
            if (++as == 2) {
                as = 0;
                aphase ^= 1;
            }
        }
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing more arrives at this CTA's barriers, and the MMAs that read its operands are done
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(ncols) : "memory");
    }
}

template <int KIND, int T, int WF>
int launch_pair(fnn_cuda_ctx *ctx, const QmmArgs &a, const PairTiling &tl) {
    const fnn_cuda_qweight *w = a.w;
    constexpr int ES = (KIND == KIND_F16) ? 2 : 1;
    constexpr int ATOMS = (KIND == KIND_F16) ? 2 : 1;
    const int M = (int)a.M, N = (int)w->N, K = (int)w->K;
    const int Kbytes = K * ES;
    const int n_tiles = (N + kPairRows - 1) / kPairRows;
    const int pairs = ctx->sm_count / 2;
    const int kblocks = (Kbytes + kKBlockBytes * ATOMS - 1) / (kKBlockBytes * ATOMS);
    const int Mb = tl.Mb, m_tiles = tl.m_tiles;

    const PrepLayout lay = prep_layout(T, ES, M, K);
    int rc = ensure_scratch(ctx, lay.bytes);
    if (rc != FNN_OK) return rc;
    uint8_t *bq = (uint8_t *)ctx->scratch;
    float *dq = (float *)(bq + lay.dq), *rowsum = (float *)(bq + lay.rowsum);
    rc = launch_act_prep(ctx, a, KIND, T, WF == WF_I4, (int)lay.Kp, bq, dq, rowsum);
    if (rc != FNN_OK) return rc;

    CUtensorMap map_w, map_a, map_s;
    rc = encode_weight_map(&map_w, w);
    if (rc != FNN_OK) return rc;
    // one CTA's half of the activation tile (see load_b)
    rc = encode_act_map(&map_a, bq, lay, T, M, T == 2 ? Mb : Mb / 2, 1);
    if (rc != FNN_OK) return rc;
    if (WF == WF_CB) {
        rc = encode_block_scale_map(&map_s, w);
        if (rc != FNN_OK) return rc;
    } else {
        map_s = map_a;   // unused
    }
    PairParams p{};
    p.scales = (w->fmt == FNN_FMT_I4CB) ? nullptr : w->scales;
    p.zeros = w->zeros;
    p.bias = a.bias;
    p.dq = dq;
    p.rowsum = rowsum;
    p.codebook = w->codebook;
    p.out = a.out;
    p.add = a.add;
    p.sum = a.sum;
    p.err_flag = ctx->err_flag;
    p.M = M;
    p.N = N;
    p.Mb = Mb;
    p.n_tiles = n_tiles;
    p.m_tiles = m_tiles;
    p.kblocks = kblocks;
    p.a_fmt = (w->fmt == FNN_FMT_F4) ? kFmtE2M1 : kFmtE4M3;
    p.acc_scale = (WF == WF_I4) ? 0.0625f : 1.0f;
    p.epilogue = a.epilogue;
    const int stage_bytes = ATOMS * (kTileN + T * Mb / 2) * kKBlockBytes +
                            ((WF == WF_TMA) ? 0 : kTileN * 64 + (WF == WF_CB ? kTileN * 16 : 0));
    const size_t tail = (3 * 8 + 4) * 8 + 8 + kTableBytes;
    p.stages = (int)std::min<size_t>(8, (kMaxSmem - 1024 - tail) / stage_bytes);
    const size_t smem = 1024 + (size_t)p.stages * stage_bytes + tail;
    const int grid = 2 * std::min(n_tiles * m_tiles, pairs);
    const int threads = (2 + kEpiWarps + xf_warps(WF)) * 32;
    auto kern = qmm_tc_pair_kernel<KIND, T, WF>;
    FNN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   FNN_ERR_DISPATCH);
    FNN_CUDA_CHECK(launch_pdl_cluster(kern, grid, 2, threads, smem, ctx, map_w, map_a, map_s, p), FNN_ERR_DISPATCH);
    ctx->launches++;
    ctx->last_path = "tc";
    ctx->last_kernel = "tc-pair";
    return FNN_OK;
}

}  // namespace

// Batch rows per pair tile.  All pairs run whole tiles and the accumulators of two tiles share the 512 TMEM columns
// (tile_time).  Among the first tile heights that cover M the cheapest is taken, a lower one only if it is 3 % cheaper: more
// tiles also move more bytes.  I8, M = 512, N = 11008 is 172 tiles of 128 rows (three waves of 128 on 74 pairs) or
// 215 tiles of 112 (three waves of 112).
PairTiling pair_tiling(int fmt, int M, int N, int K, int sm_count) {
    const int n_tiles = (N + kPairRows - 1) / kPairRows, pairs = std::max(1, sm_count / 2);
    const int kblocks = (K + kKBlockBytes - 1) / kKBlockBytes;
    const int terms = tc_terms(fmt, M);
    const TileCosts &c = tile_costs(fmt, terms);
    PairTiling best{};
    // terms x rows columns: at most 256, a multiple of 32
    const int mb_max = terms == 1 ? 256 : terms == 2 ? 128 : 64, gran = terms == 2 ? 16 : 32;
    for (int q = (M + mb_max - 1) / mb_max, i = 0; i < 8; ++i, ++q) {
        const int rows = (M + q - 1) / q;
        const int Mb = std::min(mb_max, (rows + gran - 1) / gran * gran);
        const int m_tiles = (M + Mb - 1) / Mb;
        const double step = c.pair_step + c.pair_step_256 * terms * Mb / 256.0;
        const double epilogue = c.pair_row * Mb * (splits_sectors(M, N) ? 1.3 : 1.0);
        const double cost = c.pair_fixed + tile_time((long long)n_tiles * m_tiles, pairs, kblocks * step, epilogue, true);
        if (best.Mb == 0 || cost < 0.97 * best.cost) best = {Mb, m_tiles, terms, cost};
    }
    return best;
}

// From 65 batch rows on, where the estimate is 4 % below the single-SM kernel's (which may split K); the codebook format
// from K=2560 on a tie, where the fit understates the single-SM kernel.  Over 760 shapes of all formats (M 65 to
// 4096, K 128 to 8192, N 512 to 28672) the kernel and tile height so chosen are 0.6 % from the fastest on average.
// us single / pair: I8 N=4096 M=100 K=4096 14.9 / 11.5; I8 N=11008 M=256 K=4096 32.4 / 25.2; I4 N=28672 M=1024 K=4096 203 /
// 173; I4 N=4096 M=128 K=14336 25.5 split / 36.6.  Codebook: N=16384 M=2048 K=512 87.0 / 89.6, K=1024 108 / 118, K=2048 177 /
// 173; N=16384 M=1024 K=4096 166 / 147; N=4096 M=333 K=4096 26.8 split / 36.6.
bool qmm_tc_uses_pair(const fnn_cuda_ctx *ctx, const fnn_cuda_qweight *w, size_t M) {
    if (M <= 64) return false;
    const PairTiling tl = pair_tiling(w->fmt, (int)M, (int)w->N, (int)w->K, ctx->sm_count);
    const double margin = w->fmt == FNN_FMT_I4CB && w->K >= 2560 ? 1.0 : 1.04;
    return tl.cost * margin < tc_single_cost(ctx, w, M);
}

int launch_qmm_tc_pair(fnn_cuda_ctx *ctx, const QmmArgs &a) {
    const PairTiling tl = pair_tiling(a.w->fmt, (int)a.M, (int)a.w->N, (int)a.w->K, ctx->sm_count);
    switch (a.w->fmt) {
    case FNN_FMT_I8:
        return launch_pair<KIND_I8, 2, WF_TMA>(ctx, a, tl);
    case FNN_FMT_I4:
        return launch_pair<KIND_I8, 2, WF_I4>(ctx, a, tl);
    case FNN_FMT_F8:
    case FNN_FMT_F4:
        return tl.terms == 3 ? launch_pair<KIND_F8, 3, WF_TMA>(ctx, a, tl) : launch_pair<KIND_F8, 2, WF_TMA>(ctx, a, tl);
    case FNN_FMT_I4CB:
        return launch_pair<KIND_F16, 1, WF_CB>(ctx, a, tl);
    }
    return set_error(FNN_ERR_UNSUPPORTED, "qmatmul: tcgen05 path does not cover format %d", a.w->fmt);
}

}  // namespace fnn
