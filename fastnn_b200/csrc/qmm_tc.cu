// tcgen05 / TMEM / TMA kernel for the quantized MatMul.
//
// Weight operand (the MMA's M side, 128 output channels per CTA tile), always fetched from the
// packed rows as the reference stores them -- no expanded copy exists in device memory:
//   I8    kind::i8, FP8 kind::f8f6f4 (e4m3): TMA drops the K-contiguous rows into 128-byte-swizzled
//         shared memory and the tensor core reads them; no ALU touches a weight bit
//   FP4   kind::f8f6f4 with an e2m1 A operand: the 4-bit tensor-map type unpacks sixteen packed
//         codes (8 bytes) into each 16-byte slot of the swizzled tile; again no ALU
//   I4    TMA brings the packed nibbles (64 bytes per row and K block); transform warps widen them
//         into TMEM as int8 holding 16*q (two logic operations per eight weights) for kind::i8
//   I4CB  TMA brings the nibbles and the block scales; transform warps write fp16 of
//         block scale x centroid (one rounding) for kind::f16
//
// Orientation: the weight tile is the MMA's M operand and the batch is its N operand, so the same
// kernel serves one batch row and thousands:
//     D[n, (t,m)] += W[n, k] * Aq_t[m, k]          (accumulators in TMEM, 128 lanes = n)
// f32 activations are first rewritten by `act_prep_kernel` as T narrow terms per element
//   int8:  a ~= dq[m] * (128*hi + lo)             (15-bit fixed point per row, T = 2)
//   e4m3:  a ~= dq[m] * (t1 + t2 + t3)            (three 4-bit-significand terms, T = 3)
//   fp16:  one term (codebook format)
// The epilogue reads the accumulators with tcgen05.ld, recombines the terms and applies
//     out[m,n] = act(dq[m]*scale[n]*acc + zero[n]*sum_k a[m,k] + bias[n])
// (src/backend/cpu/microkernels/gemm.rs:2048-2087, src/backend/cpu/matmul.rs:61-71).
//
// Warp roles: warp 0 = TMA producer and TMEM owner, warp 1 = MMA issuer, warps 2-9 = epilogue (a TMEM
// lane quadrant each, two warps per quadrant), from warp 10 on = transform (I4: 8, I4CB: 16).  Every
// mbarrier wait is bounded: a wait that runs out raises the context's error flag, every role leaves
// its loop, TMEM is freed and the kernel returns.
#include "tc_common.cuh"

#include <algorithm>
#include <cuda_fp8.h>

namespace fnn {

namespace {

using namespace tc;

// One activation, already divided by the row's step, as T narrow terms: an int8 pair hi * 128 + lo
// (15 bits), or an e4m3 code followed by the codes of what the earlier terms left over.
template <int KIND, int T>
__device__ __forceinline__ void split_terms(float x, uint8_t t[3]) {
    if (KIND == KIND_I8) {
        int q = __float2int_rn(x);
        q = max(-16256, min(16256, q));
        const int hi = (q + 64) >> 7;
        const int lo = q - hi * 128;
        t[0] = (uint8_t)(int8_t)hi;
        t[1] = (uint8_t)(int8_t)lo;
    } else {
        float r = x;
#pragma unroll
        for (int i = 0; i < T; ++i) {
            __nv_fp8_storage_t c = __nv_cvt_float_to_fp8(r, __NV_SATFINITE, __NV_E4M3);
            t[i] = (uint8_t)c;
            r -= __half2float(__half(__nv_cvt_fp8_to_halfraw(c, __NV_E4M3)));
        }
    }
}

// split_terms for a unit of eight, as the two words of each term (the bytes split_terms gives).  Two elements per conversion and
// four per pack: a block runs this code once per unit it holds, straight through, and fetching it is what it waits for (us
// element by element / so: four FP8 pairs at 16 rows 108.3 / 106.0, at 24 rows of K=3072 94.0 / 90.4; FP4 M=4 K=8192 N=28672
// 29.6 / 29.1; four I4 decoder layers at 64 rows 299.4 / 298.7).
template <int KIND, int T, bool PERM8>
__device__ __forceinline__ void split_unit(float (&x)[8], uint32_t (&w)[T][2]) {
    if constexpr (KIND == KIND_I8) {
        int8_pairs<PERM8>(x, w[0], w[T - 1]);
    } else {
#pragma unroll
        for (int t = 0; t < T; ++t) {
            uint32_t c[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_fp8x2_storage_t two =
                    __nv_cvt_float2_to_fp8x2(make_float2(x[2 * j], x[2 * j + 1]), __NV_SATFINITE, __NV_E4M3);
                c[j] = two;
                if (t + 1 < T) {
                    const float2 back = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(two, __NV_E4M3)));
                    x[2 * j] -= back.x;
                    x[2 * j + 1] -= back.y;
                }
            }
            w[t][0] = c[0] | (c[1] << 16);
            w[t][1] = c[2] | (c[3] << 16);
        }
    }
}

// The activations are written by the kernel before this one on the stream, so they may only be
// read after griddepcontrol.wait (see ld_after_wait; the compiler did move an invariant load above it once, and a
// chain of layers read the previous run's activations).  The activation pointers carry no __restrict__.

// ---- activation rewrite ---------------------------------------------------------------------
// One block per batch row.  Writes T byte planes Bq[t][m][Kp] (rows zero-padded to Kp), the
// per-row factor dq[m] and the row sum.  PERM8: inside every group of eight k the bytes are stored
// in the order 0,2,4,6,1,3,5,7 -- the order in which the I4 transform emits its weights.
template <int KIND, int T, bool PERM8>
__global__ void __launch_bounds__(256)
act_prep_kernel(const float *act, int M, int K, int Kp, uint8_t *bq, float *dq, float *rowsum) {
    __shared__ float s_max[8], s_sum[8];
    // reads the activations and overwrites planes the previous tensor-core kernel may still read
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x, tid = threadIdx.x;
    const float *row = act + (size_t)m * K;
    float mx = 0.0f, sum = 0.0f;
    for (int k = tid; k < K; k += 256) {
        float a = row[k];
        mx = fmaxf(mx, fabsf(a));
        sum += a;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    if ((tid & 31) == 0) {
        s_max[tid >> 5] = mx;
        s_sum[tid >> 5] = sum;
    }
    __syncthreads();
    mx = 0.0f;
    sum = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        mx = fmaxf(mx, s_max[w]);
        sum += s_sum[w];
    }
    if (KIND == KIND_F16) {
        // one fp16 term; the row is scaled by a power of two so that its largest element sits just
        // below 2^15 (exact, any f32 magnitude fits): bq is [M][Kp bytes] of halves
        int ex = 15;
        if (mx > 0.0f && isfinite(mx)) (void)frexpf(mx, &ex);
        const int e = max(-120, min(120, 15 - ex));
        const float up = ldexpf(1.0f, e);
        if (tid == 0) {
            dq[m] = ldexpf(1.0f, -e);
            rowsum[m] = sum;
        }
        __half *dst = reinterpret_cast<__half *>(bq + (size_t)m * Kp);
        for (int k = tid; k < Kp / 2; k += 256) dst[k] = __float2half_rn(k < K ? row[k] * up : 0.0f);
        return;
    }
    const float full = (KIND == KIND_I8) ? 16256.0f : 448.0f;
    const float step = (mx > 0.0f && isfinite(mx)) ? mx / full : 1.0f;
    const float inv = 1.0f / step;
    if (tid == 0) {
        dq[m] = step;
        rowsum[m] = sum;
    }
    for (int k = tid; k < Kp; k += 256) {
        uint8_t t[3];
        split_terms<KIND, T>((k < K) ? row[k] * inv : 0.0f, t);
        const int i8 = k & 7;
        const int kk = PERM8 ? ((k & ~7) | ((i8 >> 1) + (i8 & 1) * 4)) : k;
#pragma unroll
        for (int i = 0; i < T; ++i) bq[((size_t)i * M + m) * Kp + kk] = t[i];
    }
}

// The same rewrite for rows of at most 32768 elements, read once: a thread holds HOLD units of eight consecutive elements
// between the scan and the rewrite, with all loads in flight together, and every plane is written eight bytes at a
// time.  (The loop above is a chain of two passes of 4-byte loads, about 8 us for K=11308.)
// One block per row, whatever the format and the number of rows: the order in which a row is summed, and with it the last
// bit of its outputs, does not depend on the batch.  A cluster that shares a row (4096 elements and 40 registers a thread to
// a block, which find room beside the I4 kernel's 576 threads, and one block more that sums the row in this order) is
// slower: us of a cluster / a block, I4 K=14336 N=4096 M=32 17.5 / 16.5, M=64 18.3 / 17.9, M=148 27.3 / 26.4; K=6000
// N=4096 M=64 14.3 / 12.0; four decoder layers at 64 rows 300.2 / 298.2.
constexpr int kPrepHold = 16;   // units of eight elements a thread can hold
// HOLD: 2, 4, 8 or 16 units, the smallest that covers the row: fewer registers (more rows at once on an SM, and room
// beside the main kernel before it) and less code to fetch, which a kernel of two microseconds notices.  From four units on the
// bound of one block per SM lets the compiler spend registers on loads in flight (64, 106 and 190 instead of 58, 80 and 152: I4
// M=64 K=14336 N=4096 18.0 us instead of 20.1).
// VEC: rows of a multiple of four elements that start on 16 bytes (every layer of a real model); else 4-byte loads.
// LEAN: 32 registers a thread instead of 40.  With a few rows the blocks then fit beside the fragment kernels' 512 threads of 112,
// which leave 8192, and start before those end (I4 M=8 K=4096 N=6144 9.7 -> 8.2 us, N=22528 18.1 -> 15.4); between 16 and 48
// rows the two differ by less than 1.1 % either way, and at 64 the wider form is a little faster (four I4 decoder layers 302.0
// lean, 299.1).
template <int KIND, int T, bool PERM8, int HOLD, bool VEC, bool LEAN>
__global__ void __launch_bounds__(256, LEAN ? 8 : 1)
act_prep_regs_kernel(const float *act, int M, int K, int Kp, uint8_t *bq, float *dq, float *rowsum) {
    __shared__ float2 s_part[8];   // maximum and sum of the warps
    pdl_launch_dependents();
    pdl_wait();
    const int m = blockIdx.x, tid = threadIdx.x;
    const float *row = act + (size_t)m * K;
    const float4 *row4 = reinterpret_cast<const float4 *>(row);
    const int units = (K + 7) >> 3;   // the last one may be partly past the row: zeros there
    float v[HOLD][8];
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
        const int u = tid + i * 256;
        if (VEC) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (8 * u < K) a = ld_after_wait(row4 + 2 * u);
            if (8 * u + 4 < K) b = ld_after_wait(row4 + 2 * u + 1);
            v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w;
            v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[i][j] = 8 * u + j < K ? ld_after_wait(row + 8 * u + j) : 0.0f;
        }
    }
    float mx = 0.0f, sum = 0.0f;
#pragma unroll
    for (int i = 0; i < HOLD; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            mx = fmaxf(mx, fabsf(v[i][j]));
            sum += v[i][j];
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    if ((tid & 31) == 0) s_part[tid >> 5] = make_float2(mx, sum);
    __syncthreads();
    mx = 0.0f;
    sum = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        mx = fmaxf(mx, s_part[w].x);
        sum += s_part[w].y;
    }
    if (KIND == KIND_F16) {
        int ex = 15;
        if (mx > 0.0f && isfinite(mx)) (void)frexpf(mx, &ex);
        const int e = max(-120, min(120, 15 - ex));
        const float up = ldexpf(1.0f, e);
        if (tid == 0) {
            dq[m] = ldexpf(1.0f, -e);
            rowsum[m] = sum;
        }
        uint4 *dst = reinterpret_cast<uint4 *>(bq + (size_t)m * Kp);   // Kp = 16 bytes per unit here
#pragma unroll
        for (int i = 0; i < HOLD; ++i) {
            const int u = tid + i * 256;
            if (u >= units) continue;
            uint32_t h[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 x = __floats2half2_rn(v[i][2 * j] * up, v[i][2 * j + 1] * up);
                h[j] = *reinterpret_cast<const uint32_t *>(&x);
            }
            dst[u] = make_uint4(h[0], h[1], h[2], h[3]);
        }
        return;
    }
    const float full = (KIND == KIND_I8) ? 16256.0f : 448.0f;
    const float step = (mx > 0.0f && isfinite(mx)) ? mx / full : 1.0f;
    const float inv = 1.0f / step;
    if (tid == 0) {
        dq[m] = step;
        rowsum[m] = sum;
        if (Kp > 8 * units) {   // one more unit of zeros pads the row to 16 bytes
#pragma unroll
            for (int i = 0; i < T; ++i)
                *reinterpret_cast<uint2 *>(bq + ((size_t)i * M + m) * Kp + 8 * units) = make_uint2(0u, 0u);
        }
    }
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
        const int u = tid + i * 256;
        if (u >= units) continue;
        uint32_t w[T][2];
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = v[i][j] * inv;
        split_unit<KIND, T, PERM8>(x, w);
#pragma unroll
        for (int q = 0; q < T; ++q)
            *reinterpret_cast<uint2 *>(bq + ((size_t)q * M + m) * Kp + (size_t)u * 8) = make_uint2(w[q][0], w[q][1]);
    }
}

// ---- main kernel ------------------------------------------------------------------------------

struct TcParams {
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
    int M, N, K;
    int Mb;        // batch rows per tile
    int nbuf;      // accumulator buffers in TMEM (1 or 2)
    int ncols;     // TMEM columns to allocate
    int n_tiles, m_tiles;
    int kblocks;   // pipeline stages' worth of K: ceil(operand bytes per row / (128 * atoms))
    AllGatherArgs ag;   // ag.world > 0: outputs go to every rank's gathered buffer
    // Long K with few tiles: `parts` CTAs of a cluster take a share of a tile's K blocks each, exchange their
    // raw accumulators through distributed shared memory and finish every parts-th chunk of the columns.
    int parts;
    int a_fmt;     // A operand format of kind::f8f6f4
    float acc_scale;   // 1/16 when the int8 operand carries 16*q (I4)
    int stages;
    int epilogue;
};

// ATOMS: 128-byte swizzle atoms of K per pipeline stage (2 for fp16 operands: a stage is 128 k for
// every format).  Shared memory per stage: operand tile, raw tile (transformed formats), activations.
// W: batch rows per epilogue chunk.  Each chunk is a chain of TMEM loads, shuffles and stores, so 16 at a time where
// whole tiles are finished (us of a wave of 148 tiles of 128 rows, K=512, SiLU, 8 / 16: I8 5.6 / 4.65, codebook 6.1 / 5.4,
// FP8 5.4 / 4.4).  Eight where the CTAs of a cluster deal the chunks out, for tiles of a single chunk of 16, which
// would leave half of the warps idle, and for three terms, whose 48 accumulators a thread cost the registers that the
// next kernel's early blocks need (FP4 64 rows K=2048: 11.0 / 12.3).
// SPLIT: the K blocks of a tile may be shared by a cluster (p.parts).  I8, FP8 and FP4 take whole tiles of up to 16 rows (FP8
// and FP4 below 128 rows: all) through the same function, so that a program whose layers alternate between the two
// keeps its instructions in the SMs' caches: with a function each every switch cost 0.7 us (six I8 pairs at 16
// rows 161 / 154.5 us, four FP8 ones 119 / 110).  The widened formats, whose function is longer, are better off with
// the two apart (four I4 pairs at 16 rows 75.3 / 72.2, six codebook ones at 64 155.3 / 152.8).
template <int KIND, int T, int WF, int W, bool SPLIT>
__global__ void __launch_bounds__((2 + kEpiWarps + xf_warps(WF)) * 32, 1)
qmm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
              const __grid_constant__ CUtensorMap map_s, TcParams p) {
    constexpr int ATOMS = (KIND == KIND_F16) ? 2 : 1;
    constexpr int raw_bytes = (WF == WF_TMA) ? 0 : kTileN * 64;        // packed nibbles: 64 bytes per row
    constexpr int sc_bytes = (WF == WF_CB) ? kTileN * 16 : 0;          // four block scales per row
    constexpr int kXf0 = 2 + kEpiWarps;                                // first transform warp
    constexpr int kSlotCols = ATOMS * 32;                              // TMEM columns of a widened operand tile
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1024-byte alignment is what the 128B swizzle atoms need
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int BNt = T * p.Mb;                               // MMA N: (term, batch row) columns
    constexpr int a_atom = kTileN * kKBlockBytes;           // 16 KB operand atom; a widened operand is in TMEM instead
    constexpr int a_bytes = (WF == WF_TMA) ? ATOMS * a_atom : 0;
    const int b_bytes = BNt * kKBlockBytes;                 // activation atom
    const int b_atom = (b_bytes + 1023) & ~1023;
    const int b_stride = ATOMS * b_atom;
    unsigned char *s_a = smem;
    unsigned char *s_b = s_a + (size_t)p.stages * a_bytes;
    unsigned char *s_raw = s_b + (size_t)p.stages * b_stride;             // [stages][raw_bytes]
    unsigned char *s_sc = s_raw + (size_t)p.stages * raw_bytes;           // [stages][sc_bytes]
    uint64_t *bars = reinterpret_cast<uint64_t *>(s_sc + (size_t)p.stages * sc_bytes);
    uint64_t *full = bars, *empty = bars + p.stages, *rawfull = bars + 2 * p.stages;
    uint64_t *tfull = bars + 3 * p.stages, *tempty = tfull + 2;
    uint64_t *tlast = tempty + 2;   // the accumulators of this CTA's last tile are complete
    uint32_t *s_tmem = reinterpret_cast<uint32_t *>(tlast + 1);
    float *s_dump = reinterpret_cast<float *>(smem);   // parts > 1: raw accumulators [T * Mb][128], over the drained ring
    volatile int *s_abort = reinterpret_cast<volatile int *>(s_tmem + 1);
    float *s_cb = table_after(s_tmem + 2);                                // [16]

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    pdl_launch_dependents();   // barrier set-up and the TMEM allocation below run under the previous kernel's tail
    const uint32_t ncols = (uint32_t)p.ncols;

    const int total_tiles = p.n_tiles * p.m_tiles;
    // whole tiles blockIdx.x, + gridDim.x, ...; a cluster of `parts` CTAs works on one tile
    const int parts = SPLIT ? p.parts : 1, part = SPLIT ? (int)(blockIdx.x % (unsigned)parts) : 0;
    const bool split = SPLIT && (WF != WF_TMA || parts > 1);
    const int first_tile = (int)(blockIdx.x / (unsigned)parts), tile_step = (int)(gridDim.x / (unsigned)parts);
    const int kb0 = p.kblocks * part / parts, kb1 = p.kblocks * (part + 1) / parts;
    // weights of stage `st`: the operand tile itself, or the packed nibbles (+ block scales) for the
    // transform warps
    auto load_w = [&](int st, int nt, int kb) {
        if (WF == WF_TMA) {
#pragma unroll
            for (int at = 0; at < ATOMS; ++at)
                tma_load_2d(s_a + (size_t)st * a_bytes + at * a_atom, &map_w, &full[st],
                            (kb * ATOMS + at) * kKBlockBytes, nt * kTileN);
        } else {
            mbar_expect_tx(&rawfull[st], (uint32_t)(raw_bytes + sc_bytes));
            tma_load_2d(s_raw + (size_t)st * raw_bytes, &map_w, &rawfull[st], kb * 64, nt * kTileN);
            if (WF == WF_CB) tma_load_2d(s_sc + (size_t)st * sc_bytes, &map_s, &rawfull[st], kb * 16, nt * kTileN);
        }
    };
    // bytes the copies of a stage report to its barrier; the unpacking 4-bit tensor-map type counts
    // the packed source bytes (half of the 16 KB tile it writes)
    const uint32_t full_tx =
        (uint32_t)((WF == WF_TMA ? (p.a_fmt == kFmtE2M1 ? a_bytes / 2 : a_bytes) : 0) + ATOMS * b_bytes);

    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_a);
        if (WF == WF_CB) prefetch_tensormap(&map_s);
        for (int s = 0; s < p.stages; ++s) {
            // the MMA issuer waits for the activation tile (one arrival with a byte count) and, for the
            // formats that are widened, for every transform warp
            mbar_init(&full[s], 1 + xf_warps(WF));
            mbar_init(&empty[s], 1);
            mbar_init(&rawfull[s], 1);
        }
        for (int i = 0; i < 2; ++i) {   // (one of each is unused with a single buffer)
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], kEpiWarps);
        }
        mbar_init(tlast, 1);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // This thread is the TMA producer.  The weights do not depend on the kernel before this one on
        // the stream: the first ring of weight tiles is requested here, before the rest of the CTA
        // has finished setting up and before griddepcontrol.wait; the matching activation tiles
        // follow in the producer's loop.
        {
            const int head = min(p.stages, kb1 - kb0), nt = first_tile / p.m_tiles;
            for (int i = 0; i < head; ++i) {
                mbar_expect_tx(&full[i], full_tx);   // stage i: all stages start empty
                load_w(i, nt, kb0 + i);
            }
            // The activation planes may still be being written: an L2 prefetch of the first tile reads
            // nothing into this SM, but it has the address translated before the copies that follow
            // griddepcontrol.wait ask for it (L2 is the point of coherence, so nothing stale can result).
            tma_prefetch_3d(&map_a, kb0 * ATOMS * kKBlockBytes, (first_tile % p.m_tiles) * p.Mb, 0);
        }
    }
    if (WF == WF_CB && threadIdx.x >= 64 && threadIdx.x < 80) s_cb[threadIdx.x - 64] = p.codebook[threadIdx.x - 64];
    if (warp == 1) {   // the MMA warp owns the tensor memory: it allocates and frees it
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(s_tmem)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *s_tmem;
    const uint32_t tmem_ops = tmem_base + (uint32_t)(p.nbuf * BNt);   // widened operands follow the accumulators

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            auto load_b = [&](int st, int mt, int kb) {
#pragma unroll
                for (int at = 0; at < ATOMS; ++at)
                    tma_load_3d(s_b + (size_t)st * b_stride + at * b_atom, &map_a, &full[st],
                                (kb * ATOMS + at) * kKBlockBytes, mt * p.Mb, 0);
            };
            // The first ring of weight tiles is already on its way (requested during set-up); the
            // activation planes depend on the kernel before this one: their tiles follow
            // griddepcontrol.wait.
            const int head = min(p.stages, kb1 - kb0);
            pdl_wait();
            for (int i = 0; i < head; ++i) load_b(i, first_tile % p.m_tiles, kb0 + i);
            s = head;
            if (s == p.stages) {
                s = 0;
                phase ^= 1;
            }
            for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
                const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
                for (int kb = kb0 + (tile == first_tile ? head : 0); kb < kb1; ++kb) {
                    if (!mbar_wait(&empty[s], phase ^ 1, s_abort, p.err_flag, 0x10)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], full_tx);
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
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
            const uint32_t idesc = make_idesc(KIND, BNt, p.a_fmt, kTileN);
            int s = 0;
            uint32_t phase = 0;
            int as = 0;
            uint32_t aphase = 0;
            bool ok = true;
            for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
                if (!mbar_wait(&tempty[as], aphase ^ 1, s_abort, p.err_flag, 0x20)) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(as * BNt);
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(&full[s], phase, s_abort, p.err_flag, 0x40)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int at = 0; at < ATOMS; ++at) {
                        const uint64_t da = make_desc_sw128(smem_u32(s_a + (size_t)s * a_bytes + at * a_atom));
                        const uint32_t ta = tmem_ops + (uint32_t)(s * kSlotCols + at * 32);
                        const uint64_t db = make_desc_sw128(smem_u32(s_b + (size_t)s * b_stride + at * b_atom));
#pragma unroll
                        for (int k = 0; k < kKBlockBytes / 32; ++k) {
                            // advance both operands by 32 bytes of K (inside the swizzled row; eight TMEM columns)
                            const uint32_t accumulate = (kb > kb0 || at > 0 || k > 0) ? 1u : 0u;
                            if (WF == WF_TMA)
                                tc_mma<KIND>(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, accumulate);
                            else
                                tc_mma_ts<KIND>(d_tmem, ta + (uint32_t)(k * 8), db + (uint64_t)(k * 2), idesc, accumulate);
                        }
                    }
                    tc_commit(&empty[s]);  // frees the stage once these MMAs have read it
                    if (++s == p.stages) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                tc_commit(tile + tile_step < total_tiles ? &tfull[as] : tlast);  // accumulator complete
                if (++as == p.nbuf) {
                    as = 0;
                    aphase ^= 1;
                }
            }
        }
    } else if (WF != WF_TMA && warp >= kXf0) {
        // ---------------- transform warps: packed nibbles -> operand tile in TMEM ----------------
        // All transform warps work on every pipeline step together (every warp meets every phase of
        // every barrier in order, which is what a parity wait needs; letting warps run steps apart
        // would let one of them see a barrier two phases behind and take it for ready).  A thread widens a
        // half (I4) or a quarter of one row: the row is its TMEM lane (a warp reaches the lane quadrant
        // warp % 4), and two or four warps share a quadrant.  The operand never touches shared memory:
        // against a swizzled tile there this takes 16 KB (32 KB fp16) out of every pipeline stage and out of
        // the shared-memory traffic of both the transform and the MMA (I4 M=64 K=4096 N=28672: 30.7 ->
        // 23.8 us, N=6144: 16.4 -> 13.6).
        const int quad = warp & 3, share = (warp - kXf0) >> 2;
        constexpr int kUnits = 4 / (xf_warps(WF) / 4 > 0 ? xf_warps(WF) / 4 : 1);   // 16-byte units per thread
        const int row = quad * 32 + lane;
        const uint32_t t_dst = tmem_ops + ((uint32_t)(quad * 32) << 16);
        int s = 0;
        uint32_t phase = 0;
        bool filled = true;
        for (int tile = first_tile; tile < total_tiles; tile += tile_step) {
            for (int kb = kb0; kb < kb1; ++kb) {
                // (A lane that gives up stays with its warp through this step and the others, whatever the stages hold, and reports
                // no stage any more.  A vote, which ends the loop for all, cost 1 % of a decoder step, and so did a branch here.)
                const bool here = mbar_wait(&rawfull[s], phase, s_abort, p.err_flag, 0x200);
                tc_fence_after();   // the stage's columns were last read by MMAs another thread issued
                const unsigned char *raw = s_raw + (size_t)s * raw_bytes + row * 64;
#pragma unroll
                for (int i = 0; i < kUnits; ++i) {
                    const int c = share * kUnits + i;   // 16-byte unit of the row: 32 codes
                    // (64-byte swizzle: unit index XOR row / 2 mod 4; eight lanes meet no bank twice)
                    const uint4 w = *reinterpret_cast<const uint4 *>(raw + ((c ^ ((row >> 1) & 3)) << 4));
                    uint32_t o[16];
                    if (WF == WF_I4) {
                        widen_i4(w, o);
                        tmem_st8(t_dst + (uint32_t)(s * kSlotCols + c * 8), o);
                    } else {
                        widen_cb(w, *reinterpret_cast<const float *>(s_sc + (size_t)s * sc_bytes + row * 16 + c * 4), smem_u32(s_cb), o);
                        tmem_st16(t_dst + (uint32_t)(s * kSlotCols + c * 16), o);
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                filled &= here;
                if (lane == 0 && filled) mbar_arrive(&full[s]);
                if (++s == p.stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
    }
    if (warp >= 2) {
        // ---------------- epilogue (8 warps: a TMEM lane quadrant each, the two warps of a quadrant taking
        // alternate chunks of the columns).  The transform warps have nothing left to do when the last tile's
        // accumulators are complete and take their share of its chunks: every chunk is a chain of TMEM loads, exchange,
        // shuffles and stores of about a microsecond, and at the end of a call all of it is exposed
        // (us before / now: I4 M=64 K=4096 N=28672 24.1 / 23.7; together with the exchange below, N=4096 in three parts
        // 10.5 / 10.0, codebook M=64 K=2048 N=8192 in two 11.1 / 10.6). ----------------
        pdl_wait();   // dq, rowsum and the output buffer belong to kernels before this one
        const int quad = warp & 3, grp = (warp - 2) >> 2;
        constexpr int kGroups = kEpiWarps / 4, kLastGroups = (kEpiWarps + xf_warps(WF)) / 4;   // warps per quadrant
        int as = 0;
        uint32_t aphase = 0;
        const bool has_zero = p.zeros != nullptr;
        const int row = quad * 32 + lane;            // this thread's row of the tile = its TMEM lane
        const int chunk0 = (part + parts * grp) * W;
        // dq and rowsum of a chunk's batch rows, spread over the lanes (lane j: dq, lane 16 + j: rowsum)
        auto load_rowfac = [&](int mt, int c0) -> float {
            const int j = lane & 15, m = mt * p.Mb + c0 + j;
            const bool want = j < W && c0 + j < p.Mb && m < p.M && (lane < 16 || has_zero);
            return want ? (lane < 16 ? p.dq : p.rowsum)[m] : 0.0f;
        };
        for (int tile = first_tile; tile < total_tiles; tile += tile_step) {
            const bool last = tile + tile_step >= total_tiles;
            if (WF != WF_TMA && !last && warp >= kXf0) {
                if (++as == p.nbuf) as = 0;
                continue;
            }
            const int step = W * (last ? kLastGroups : kGroups);   // columns per round of a quadrant's warps
            const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
            // Everything the epilogue needs besides the accumulator is requested before the wait for
            // it, so these loads (a trip to L2 or HBM each) run under the tile's main loop.
            const int n = nt * kTileN + row;
            const bool n_ok = n < p.N;
            const float scale = n_ok ? (p.scales ? __ldg(p.scales + n) : 1.0f) : 0.0f;
            const float zero = (n_ok && has_zero) ? __ldg(p.zeros + n) : 0.0f;
            const float bias = (n_ok && p.bias) ? p.bias[n] : 0.0f;
            float fac = load_rowfac(mt, chunk0);
            const bool ok = mbar_wait_warp(last ? tlast : &tfull[as], last ? 0u : aphase, s_abort, p.err_flag, 0x80);
            tc_fence_after();
            const uint32_t t_base = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(as * BNt);
            if (split) {
                // Every MMA of this CTA has read its operands, so the ring is free: the chunks that other
                // CTAs finish go there ([column][row]: a warp stores 32 consecutive rows).
                for (int c0 = grp * W; c0 < p.Mb && ok; c0 += step) {
                    if ((c0 / W) % parts == part) continue;
#pragma unroll
                    for (int t = 0; t < T; ++t) {
                        uint32_t x[W];
                        tmem_ld_cols(t_base + (uint32_t)(t * p.Mb + c0), x);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < W; ++j) s_dump[(t * p.Mb + c0 + j) * kTileN + row] = __uint_as_float(x[j]);
                    }
                }
                __syncwarp();
                cluster_sync();
            }
            if (!ok) {
                if (split) cluster_arrive();
                break;
            }
            bool arrived = !split;
            for (int c0 = chunk0; c0 < p.Mb; c0 += parts * step) {
                uint32_t r[T][W];
#pragma unroll
                for (int t = 0; t < T; ++t) tmem_ld_cols(t_base + (uint32_t)(t * p.Mb + c0), r[t]);
                const float fac_next = load_rowfac(mt, c0 + parts * step);   // next chunk's
                tmem_ld_wait();
                if (split) {
                    // This CTA's share, then the others from the first on: the order decides the last bit of an f32 sum.  (Of
                    // integers it does not, and every CTA begins with its neighbour.)  Several in flight at once, as far as the
                    // registers go (I8 M=16 K=11008 N=4096 in three parts 14.4 -> 13.5 us; FP8 in flight behind the
                    // arrival below 10.1 -> 9.4; six codebook pairs at 64 rows with two / three 154.2 / 153.1).
                    constexpr int kFlight = T == 1 ? 3 : T == 2 ? 2 : 1;
                    auto other = [&](int i) {   // i = 1 .. parts - 1
                        if (KIND == KIND_I8) return part + i < parts ? part + i : part + i - parts;
                        return i - 1 < part ? i - 1 : i;
                    };
                    auto fetch = [&](int q, uint32_t (&x)[T][W]) {
                        const uint32_t src = mapa(s_dump + (size_t)c0 * kTileN + row, (uint32_t)q);
#pragma unroll
                        for (int t = 0; t < T; ++t)
#pragma unroll
                            for (int j = 0; j < W; ++j) x[t][j] = ld_cluster(src + (uint32_t)((t * p.Mb + j) * kTileN * 4));
                    };
                    auto add = [&](const uint32_t (&x)[T][W]) {
#pragma unroll
                        for (int t = 0; t < T; ++t)
#pragma unroll
                            for (int j = 0; j < W; ++j)
                                r[t][j] = (KIND == KIND_I8) ? (uint32_t)((int)r[t][j] + (int)x[t][j])
                                                            : __float_as_uint(__uint_as_float(r[t][j]) + __uint_as_float(x[t][j]));
                    };
#pragma unroll 1
                    for (int i = 1; i < parts; i += kFlight) {
                        uint32_t x[kFlight][T][W];
#pragma unroll
                        for (int f = 0; f < kFlight; ++f)
                            if (i + f < parts) fetch(other(i + f), x[f]);
#pragma unroll
                        for (int f = 0; f < kFlight; ++f)
                            if (i + f < parts) add(x[f]);
                    }
                    if (c0 + parts * step >= p.Mb) {   // this warp reads nothing more of the other CTAs
                        __syncwarp();
                        cluster_arrive();
                        arrived = true;
                    }
                }
                // (straight-line code, stored under a predicate)
                float v[W];
                finish_chunk<KIND, T>(r, fac, scale, zero, bias, p.bias != nullptr, p.acc_scale, p.epilogue, v);
                const int m0 = mt * p.Mb + c0;
                const int jmax = n_ok ? min(W, min(p.Mb - c0, p.M - m0)) : 0;   // rows of this chunk that exist
                if (p.ag.world == 0) {
                    store_chunk(p.out, p.add, p.sum, (size_t)m0 * p.N + n, p.N, jmax, v);
                } else {   // plain peer stores over NVLink (and one local store)
                    const size_t at = (size_t)m0 * p.ag.n_total + p.ag.col0 + n;
                    for (int rk = 0; rk < p.ag.world; ++rk) {
                        float *dst = p.ag.peer_out[rk] + at;
#pragma unroll
                        for (int j = 0; j < W; ++j)
                            if (j < jmax) dst[(size_t)j * p.ag.n_total] = v[j];
                    }
                }
                fac = fac_next;
            }
            __syncwarp();
            if (!arrived) cluster_arrive();
            tc_fence_before();
            __syncwarp();
            if (!last && lane == 0) mbar_arrive(&tempty[as]);
            if (++as == p.nbuf) {
                as = 0;
                aphase ^= 1;
            }
        }
    }

    __syncwarp();
    if (split) {
        // The roles without an epilogue meet the exchange here; then nobody leaves while its shares are read.  (The epilogue
        // warps have arrived for that behind their last read.)
        if (warp < 2) {
            cluster_sync();
            cluster_arrive();
        }
        __syncwarp();
        cluster_wait();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(ncols)
                     : "memory");
    }
    if (p.ag.world > 0 && threadIdx.x == 32) {
        // Every store of this CTA happened before the barrier above.  A device-scope fence and a ticket
        // hand them to the CTA that leaves last on this rank; that one CTA makes everything visible
        // system-wide (one system-scope fence per launch: 148 of them at once cost about 10 us) and
        // adds one arrival to every rank's counter (release).  It then waits (bounded) until every
        // rank's arrival for this step is in before the kernel ends, so whatever follows on the
        // stream reads complete rows without a separate consumer kernel.  counters = {arrivals,
        // consumed} live in device memory and only grow: a captured graph can be replayed.
        __threadfence();
        const int ticket = atomicAdd(p.ag.ticket, 1);
        if (ticket == (int)gridDim.x - 1) {
            *p.ag.ticket = 0;
            __threadfence_system();
            for (int r = 0; r < p.ag.world; ++r)
                asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(p.ag.peer_arrive[r]) : "memory");
            unsigned *counters = p.ag.peer_arrive[p.ag.rank];
            const unsigned want = counters[1] + (unsigned)p.ag.world;
            const long long t0 = clock64();
            for (;;) {
                unsigned got;
                asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(got) : "l"(counters) : "memory");
                if ((int)(got - want) >= 0) {
                    counters[1] = want;
                    break;
                }
                if (clock64() - t0 > kWaitCycles) {   // gives up without consuming
                    raise_error(p.err_flag, 0x400);
                    break;
                }
            }
        }
    }
}

}  // namespace

// ---- host side -----------------------------------------------------------------------------------

// cuTensorMapEncodeTiled is looked up through the runtime, so the library itself carries no
// link-time dependency on libcuda (it must load, and fail cleanly, on a machine without a driver).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

int tc::encode_map(CUtensorMap *map, void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
               const cuuint32_t *box, CUtensorMapSwizzle swizzle, CUtensorMapDataType dtype) {
    static EncodeTiledFn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        FNN_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres),
                       FNN_ERR_UNSUPPORTED);
        FNN_REQUIRE(fn != nullptr && qres == cudaDriverEntryPointSuccess, FNN_ERR_UNSUPPORTED,
                    "the CUDA driver does not provide cuTensorMapEncodeTiled");
        encode = (EncodeTiledFn)fn;
    }
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode(map, dtype, (cuuint32_t)rank, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(FNN_ERR_DISPATCH, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return FNN_OK;
}

// Tensor map of the weight operand over the packed rows (row stride ld_u4 * 16 bytes).
//   I8 / FP8: 128 bytes x 128 rows per box, 128-byte swizzle: the operand tile itself.
//   FP4:      the 4-bit type that unpacks sixteen codes (8 bytes) into every 16-byte slot: 128 codes
//             x 128 rows per box, 128-byte swizzle.  Needs 32-byte aligned rows.
//   I4 / I4CB: the packed nibbles as bytes, 64 bytes x 128 rows, 64-byte swizzle (the transform warps
//             read a row per thread).
int tc::encode_weight_map(CUtensorMap *map, const fnn_cuda_qweight *w) {
    const cuuint64_t row_bytes = (cuuint64_t)w->ld_u4 * 16;
    cuuint64_t strides[1] = {row_bytes};
    if (w->fmt == FNN_FMT_I8 || w->fmt == FNN_FMT_F8) {
        cuuint64_t dims[2] = {(cuuint64_t)w->K, (cuuint64_t)w->N};
        cuuint32_t box[2] = {(cuuint32_t)kKBlockBytes, (cuuint32_t)kTileN};
        return encode_map(map, (void *)w->rows, 2, dims, strides, box);
    }
    if (w->fmt == FNN_FMT_F4) {
        cuuint64_t dims[2] = {row_bytes * 2, (cuuint64_t)w->N};   // in codes; a multiple of 128
        cuuint32_t box[2] = {128, (cuuint32_t)kTileN};
        return encode_map(map, (void *)w->rows, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B);
    }
    cuuint64_t dims[2] = {row_bytes, (cuuint64_t)w->N};
    cuuint32_t box[2] = {64, (cuuint32_t)kTileN};
    return encode_map(map, (void *)w->rows, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}

// I4CB: block scales f32 [N][K/32] as bytes, four scales (16 bytes) per row and K block of 128.
int tc::encode_block_scale_map(CUtensorMap *map, const fnn_cuda_qweight *w) {
    cuuint64_t dims[2] = {(cuuint64_t)w->blocks_per_row * 4, (cuuint64_t)w->N};
    cuuint64_t strides[1] = {(cuuint64_t)w->blocks_per_row * 4};
    cuuint32_t box[2] = {16, (cuuint32_t)kTileN};
    return encode_map(map, (void *)w->scales, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

namespace {

template <int KIND, int T, bool PERM8, bool VEC>
auto prep_kernel(int M, int K) {
    return K <= 2 * 256 * 8   ? (M <= 32 ? act_prep_regs_kernel<KIND, T, PERM8, 2, VEC, true>
                                         : act_prep_regs_kernel<KIND, T, PERM8, 2, VEC, false>)
           : K <= 4 * 256 * 8 ? act_prep_regs_kernel<KIND, T, PERM8, 4, VEC, false>
           : K <= 8 * 256 * 8 ? act_prep_regs_kernel<KIND, T, PERM8, 8, VEC, false>
                              : act_prep_regs_kernel<KIND, T, PERM8, kPrepHold, VEC, false>;
}

template <int KIND, int T, bool PERM8>
int launch_prep(fnn_cuda_ctx *ctx, const QmmArgs &a, int Kp, uint8_t *bq, float *dq, float *rowsum) {
    const int M = (int)a.M, K = (int)a.w->K;
    const bool vec = K % 4 == 0 && (reinterpret_cast<uintptr_t>(a.a) & 15) == 0;
    // same shared-memory carve-out as the main kernel: alternating carve-outs between consecutive
    // kernels makes every SM reconfigure (and drain) twice per call
    auto prep = K > kPrepHold * 256 * 8 ? act_prep_kernel<KIND, T, PERM8>
                : vec                   ? prep_kernel<KIND, T, PERM8, true>(M, K)
                                        : prep_kernel<KIND, T, PERM8, false>(M, K);
    FNN_CUDA_CHECK(cudaFuncSetAttribute(prep, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared),
                   FNN_ERR_DISPATCH);
    FNN_CUDA_CHECK(launch_pdl(prep, M, 256, 0, ctx, a.a, M, K, Kp, bq, dq, rowsum), FNN_ERR_DISPATCH);
    ctx->launches++;
    return FNN_OK;
}

}  // namespace

int tc::launch_act_prep(fnn_cuda_ctx *ctx, const QmmArgs &a, int kind, int terms, bool perm8, int Kp, uint8_t *bq,
                        float *dq, float *rowsum) {
    if (kind == KIND_I8)
        return perm8 ? launch_prep<KIND_I8, 2, true>(ctx, a, Kp, bq, dq, rowsum)
                     : launch_prep<KIND_I8, 2, false>(ctx, a, Kp, bq, dq, rowsum);
    if (kind == KIND_F16) return launch_prep<KIND_F16, 1, false>(ctx, a, Kp, bq, dq, rowsum);
    return terms == 2 ? launch_prep<KIND_F8, 2, false>(ctx, a, Kp, bq, dq, rowsum)
                      : launch_prep<KIND_F8, 3, false>(ctx, a, Kp, bq, dq, rowsum);
}

// Planes of exactly M rows: a tile that reaches past them gets zeros from the copy, so the scratch of a call
// depends on neither the kernel nor the tile height, and grows with M.
tc::PrepLayout tc::prep_layout(int terms, int elem_bytes, size_t M, size_t K) {
    PrepLayout l;
    l.Kp = (K * elem_bytes + 15) & ~(size_t)15;   // TMA strides are multiples of 16 bytes
    l.dq = ((size_t)terms * M * l.Kp + 255) & ~(size_t)255;
    l.rowsum = l.dq + M * 4;
    l.bytes = l.rowsum + M * 4;
    return l;
}

int tc::encode_act_map(CUtensorMap *map, void *planes, const PrepLayout &l, int terms, size_t M, int box_rows, int box_planes) {
    cuuint64_t dims[3] = {(cuuint64_t)l.Kp, (cuuint64_t)M, (cuuint64_t)terms};
    cuuint64_t strides[2] = {(cuuint64_t)l.Kp, (cuuint64_t)(l.Kp * M)};
    cuuint32_t box[3] = {(cuuint32_t)kKBlockBytes, (cuuint32_t)box_rows, (cuuint32_t)box_planes};
    return encode_map(map, planes, 3, dims, strides, box);
}

namespace {

// CTAs (one per SM) that share a tile's K loop as a cluster.  Worth it where the tiles leave SMs idle and K is long;
// the shares meet in distributed shared memory (an earlier form met in global memory behind flags and spent
// 13 us on it).  Costs in microseconds, fitted to chains of one layer: a K block of one CTA, and per extra CTA
// the exchange and the SMs that the next kernel's early blocks no longer find free.  Measured at 1 / 2 / 3 / 4 parts:
// I4 M=64 K=14336 N=4096 32.4 / 21.2 / 19.3 / 20.2, K=4096 N=4096 13.5 / 11.4 / 11.0 / 11.9; I8 M=16 K=11008
// N=4096 19.1 / 15.9 / 14.1 / 13.8; codebook M=64 K=8192 N=2048 53.0 / 28.8 / - / 18.4 and 16.0 at 6.
// A cluster lives inside one GPC, so fewer of the larger ones run at once (74, 45, 33, 26, 22 of 2 .. 6 on a
// B200, and only 15 of 8); a cluster that has to wait for a second round costs more than the split gains
// (48 tiles in 3 parts: 19.9 us against 11.8 in 2).
int split_parts(const fnn_cuda_ctx *ctx, int tiles, int kblocks, int cols, int wf) {
    static const int kActive[] = {0, 148, 74, 45, 33, 26, 22};   // of 148 SMs
    const double t_step = (wf == WF_CB) ? 0.8 : 0.15 + 0.25 * cols / 256.0;
    const double t_part = 0.8 + 0.4 * cols / 128.0;
    const int waves = (tiles + ctx->sm_count - 1) / ctx->sm_count;
    int best = 1;
    double best_cost = waves * kblocks * t_step;
    for (int q = 2; q <= 6 && q <= kblocks; ++q) {
        // (the codebook kernel's 832 threads leave no room beside them: with the last two clusters of three taken a call waits for the
        // SMs that the rewrite is on, M=48 K=2944 N=5732 14.1 us in three parts, 11.3 in two)
        const int spare = wf == WF_CB && q == 3 ? 2 : 0;
        if (tiles > (kActive[q] - spare) * ctx->sm_count / 148) break;
        const bool crowded = 4 * tiles * q > 3 * ctx->sm_count;
        const double cost = (kblocks + q - 1) / q * t_step + t_part * (q - 1) + (crowded ? 1.5 : 0.0);
        if (cost < best_cost) {
            best = q;
            best_cost = cost;
        }
    }
    return best;
}

// TMEM columns of a widened operand tile, and accumulator buffers: two (the next tile's MMAs run under a tile's epilogue)
// where the widened operands of at least four stages fit beside them in the 512 columns, else one.
constexpr int operand_cols(int wf) { return wf == WF_TMA ? 0 : wf == WF_I4 ? 32 : 64; }
int acc_buffers(int cols, int slot_cols) { return 2 * cols + 4 * slot_cols <= 512 ? 2 : 1; }

// Batch rows per tile: T * Mb is the MMA N (multiple of 16, at most 256), tiles of equal height.  The codebook format stops at
// 128: two accumulator buffers then fit beside the widened operands, and the epilogue of a tile runs under the
// next (M=674 K=512 N=8320, where the epilogue is the bound: 34.5 us with one buffer of 256).
int batch_rows(int terms, int M) {
    const int most = terms == 3 ? 80 : 128, tiles = (M + most - 1) / most;
    return ((M + tiles - 1) / tiles + 15) & ~15;
}

// Scratch of one call: the rewritten activations Bq[T][M][Kp], then dq[M] and rowsum[M] (tc::prep_layout).
// `fixed_scratch` null: the context's growable buffer; otherwise a caller-supplied region of
// `fixed_bytes` that must already be large enough (the entry point that may not allocate).
template <int KIND, int T, int WF>
int launch_tc(fnn_cuda_ctx *ctx, const QmmArgs &a, uint8_t *fixed_scratch = nullptr, size_t fixed_bytes = 0) {
    const fnn_cuda_qweight *w = a.w;
    constexpr int ES = (KIND == KIND_F16) ? 2 : 1;  // bytes per operand element
    constexpr int ATOMS = (KIND == KIND_F16) ? 2 : 1;
    const int M = (int)a.M, N = (int)w->N, K = (int)w->K;
    const int Kbytes = K * ES;
    const int Mb = batch_rows(T, M);
    const int m_tiles = (M + Mb - 1) / Mb;
    const PrepLayout lay = prep_layout(T, ES, M, K);
    const int n_tiles = (N + kTileN - 1) / kTileN;
    const int kblocks = (Kbytes + kKBlockBytes * ATOMS - 1) / (kKBlockBytes * ATOMS);
    const int tiles = n_tiles * m_tiles;
    const int parts = split_parts(ctx, tiles, kblocks, T * Mb, WF);
    int rc = FNN_OK;
    uint8_t *bq;
    if (fixed_scratch) {
        FNN_REQUIRE(lay.bytes <= fixed_bytes, FNN_ERR_MEMORY,
                    "qmatmul_noalloc: M=%d, K=%d needs %zu bytes of activation scratch; the built-in "
                    "scratch holds %zu (use fnn_cuda_qmatmul for larger problems)",
                    M, K, lay.bytes, fixed_bytes);
        bq = fixed_scratch;
    } else {
        rc = ensure_scratch(ctx, lay.bytes);
        if (rc != FNN_OK) return rc;
        bq = (uint8_t *)ctx->scratch;
    }
    float *dq = (float *)(bq + lay.dq), *rowsum = (float *)(bq + lay.rowsum);
    rc = launch_act_prep(ctx, a, KIND, T, WF == WF_I4, (int)lay.Kp, bq, dq, rowsum);
    if (rc != FNN_OK) return rc;

    CUtensorMap map_w, map_a, map_s;
    rc = encode_weight_map(&map_w, w);
    if (rc != FNN_OK) return rc;
    rc = encode_act_map(&map_a, bq, lay, T, M, Mb, T);
    if (rc != FNN_OK) return rc;
    if (WF == WF_CB) {
        rc = encode_block_scale_map(&map_s, w);
        if (rc != FNN_OK) return rc;
    } else {
        map_s = map_a;   // unused
    }
    TcParams p{};
    p.scales = (w->fmt == FNN_FMT_I4CB) ? nullptr : w->scales;  // block scales are folded into the operand
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
    p.K = K;
    p.Mb = Mb;
    p.parts = parts;
    p.n_tiles = n_tiles;
    p.m_tiles = m_tiles;
    p.kblocks = kblocks;
    p.a_fmt = (w->fmt == FNN_FMT_F4) ? kFmtE2M1 : kFmtE4M3;
    p.acc_scale = (WF == WF_I4) ? 0.0625f : 1.0f;
    p.epilogue = a.epilogue;
    if (a.allgather) p.ag = *a.allgather;
    const int a_bytes = (WF == WF_TMA) ? ATOMS * kTileN * kKBlockBytes : 0;
    const int b_stride = ATOMS * ((T * Mb * kKBlockBytes + 1023) & ~1023);
    const int raw_bytes = (WF == WF_TMA) ? 0 : kTileN * 64 + (WF == WF_CB ? kTileN * 16 : 0);
    int stages = (int)((200 * 1024) / (size_t)(a_bytes + b_stride + raw_bytes));
    stages = std::max(2, std::min(stages, 8));
    const int slot_cols = operand_cols(WF);
    p.nbuf = acc_buffers(T * Mb, slot_cols);
    if (slot_cols) stages = std::min(stages, (512 - p.nbuf * T * Mb) / slot_cols);
    p.ncols = 32;
    while (p.ncols < p.nbuf * T * Mb + stages * slot_cols) p.ncols <<= 1;
    p.stages = stages;
    const size_t ring = (size_t)stages * (a_bytes + b_stride + raw_bytes);
    // the exchange of a split lies over the drained ring, and the barriers are live right behind the ring
    FNN_REQUIRE(parts == 1 || (size_t)T * Mb * kTileN * 4 <= ring, FNN_ERR_DISPATCH,
                "qmatmul: a ring of %d stages does not hold the partial accumulators of %d columns", stages, T * Mb);
    size_t smem = 1024 + ring + (3 * stages + 5) * 8 + 8 + kTableBytes;
    // A CTA of a split keeps its TMEM until its cluster has met, and the allocation is a wait without a bound: two CTAs
    // of a split on one SM could wait for each other's columns for good.  More than half of an SM's
    // shared memory each keeps them apart (I4 up to 16 rows asks for 98 KB and 512 columns).
    if (parts > 1) smem = std::max(smem, kHalfSmem);
    const int grid = parts > 1 ? tiles * parts : std::min(tiles, ctx->sm_count);
    const int threads = (2 + kEpiWarps + xf_warps(WF)) * 32;
    auto kern = qmm_tc_kernel<KIND, T, WF, 8, true>;
    if constexpr (WF != WF_TMA)
        if (parts == 1) kern = qmm_tc_kernel<KIND, T, WF, 8, false>;
    if constexpr (T < 3)
        if (parts == 1 && Mb > 16) kern = qmm_tc_kernel<KIND, T, WF, 16, false>;
    FNN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   FNN_ERR_DISPATCH);
    if (parts > 1) {
        FNN_CUDA_CHECK(launch_pdl_cluster(kern, grid, parts, threads, smem, ctx, map_w, map_a, map_s, p), FNN_ERR_DISPATCH);
    } else {
        FNN_CUDA_CHECK(launch_pdl(kern, grid, threads, smem, ctx, map_w, map_a, map_s, p), FNN_ERR_DISPATCH);
    }
    ctx->launches++;
    ctx->last_path = fixed_scratch ? "tc-noalloc" : "tc";
    ctx->last_kernel = parts > 1 ? "tc-split" : "tc";
    return FNN_OK;
}

}  // namespace

int dispatch_tc(fnn_cuda_ctx *ctx, const QmmArgs &a, uint8_t *fixed, size_t fixed_bytes);

int tc::tc_terms(int fmt, size_t M) {
    return fmt == FNN_FMT_I4CB ? 1 : (fmt == FNN_FMT_F8 || fmt == FNN_FMT_F4) && M < 128 ? 3 : 2;
}

// Fitted (least squares of the logarithms, 6 to 7 % rms) to chains of one layer with a SiLU: 786 shapes from M=65 on, both
// kernels and up to three tile heights each.
const tc::TileCosts &tc::tile_costs(int fmt, int terms) {
    static const TileCosts i8 = {3.28, 0.283, 0.091, 0.028, 0.53, 1.49, 3.40, 0.110, 0.207, 0.037};
    static const TileCosts i4 = {2.89, 0.135, 0.200, 0.039, 0.0, 1.56, 3.26, 0.194, 0.125, 0.039};
    static const TileCosts f8x3 = {2.53, 0.064, 0.290, 0.043, 2.81, 0.0, 2.78, 0.116, 0.138, 0.042};
    static const TileCosts f8x2 = {3.43, 0.111, 0.267, 0.028, 0.0, 1.70, 3.59, 0.050, 0.293, 0.036};
    static const TileCosts cb = {2.91, 0.450, 0.297, 0.033, 0.0, 2.45, 2.45, 0.699, 0.281, 0.037};
    switch (fmt) {
    case FNN_FMT_I8: return i8;
    case FNN_FMT_I4: return i4;
    case FNN_FMT_I4CB: return cb;
    default: return terms == 3 ? f8x3 : f8x2;
    }
}

size_t qmm_tc_scratch_bytes(const fnn_cuda_qweight *w, size_t M) {
    return prep_layout(tc_terms(w->fmt, M), w->fmt == FNN_FMT_I4CB ? 2 : 1, M, w->K).bytes;
}

double tc_single_cost(const fnn_cuda_ctx *ctx, const fnn_cuda_qweight *w, size_t M) {
    const int terms = tc_terms(w->fmt, M), Mb = batch_rows(terms, (int)M), cols = terms * Mb;
    const int wf = w->fmt == FNN_FMT_I4CB ? WF_CB : w->fmt == FNN_FMT_I4 ? WF_I4 : WF_TMA;
    const int tiles = (int)(div_ceil(w->N, (size_t)kTileN) * div_ceil(M, (size_t)Mb));
    const int kblocks = (int)div_ceil(w->K, (size_t)kKBlockBytes), parts = split_parts(ctx, tiles, kblocks, cols, wf);
    const TileCosts &c = tile_costs(w->fmt, terms);
    const double step = c.step + c.step_256 * cols / 256.0, epilogue = c.row * Mb * (splits_sectors(M, w->N) ? 1.8 : 1.0);
    if (parts > 1)
        return c.fixed + (kblocks + parts - 1) / parts * step + (c.part + c.part_128 * cols / 128.0) * (parts - 1) +
               epilogue / parts;
    return c.fixed + tile_time(tiles, ctx->sm_count, kblocks * step, epilogue, acc_buffers(cols, operand_cols(wf)) == 2);
}

bool qmm_tc_supported(const fnn_cuda_qweight *w, size_t M) {
    (void)M;
    // I8 / FP8 / FP4 codes are operands as stored; I4 and the codebook format are widened on the way.  The codebook format becomes fp16 of block scale x centroid (only when those stay inside
    // the fp16 range) and its block scales travel by TMA, four per row and stage (K a multiple of 128).
    if (w->fmt == FNN_FMT_I4CB && (!w->fp16_ok || w->K % 128 != 0)) return false;
    return w->K >= 128 && w->N >= 1 && w->N < (1u << 30) && w->K < (1u << 29);
}

// Nothing to build: every format is read from the packed rows.
int prepare_qmm_tc(fnn_cuda_ctx *, fnn_cuda_qweight *) { return FNN_OK; }

// Format -> (MMA kind, activation terms, weight path).  `fixed`: caller-supplied scratch or null.
int dispatch_tc(fnn_cuda_ctx *ctx, const QmmArgs &a, uint8_t *fixed, size_t fixed_bytes) {
    switch (a.w->fmt) {
    case FNN_FMT_I8:
        return launch_tc<KIND_I8, 2, WF_TMA>(ctx, a, fixed, fixed_bytes);
    case FNN_FMT_I4:
        return launch_tc<KIND_I8, 2, WF_I4>(ctx, a, fixed, fixed_bytes);
    case FNN_FMT_F8:
    case FNN_FMT_F4:
        // three e4m3 terms keep f32-grade accuracy while the scan of the weights is the bound;
        // two terms (~1e-3 of the output norm) once the tensor core is
        return a.M >= 128 ? launch_tc<KIND_F8, 2, WF_TMA>(ctx, a, fixed, fixed_bytes)
                          : launch_tc<KIND_F8, 3, WF_TMA>(ctx, a, fixed, fixed_bytes);
    case FNN_FMT_I4CB:
        return launch_tc<KIND_F16, 1, WF_CB>(ctx, a, fixed, fixed_bytes);
    }
    return set_error(FNN_ERR_UNSUPPORTED, "qmatmul: tcgen05 path does not cover format %d", a.w->fmt);
}

int launch_qmm_tc(fnn_cuda_ctx *ctx, const QmmArgs &a) {
    FNN_REQUIRE(a.M < (1u << 24), FNN_ERR_DISPATCH, "qmatmul: M=%zu too large for the tcgen05 path", a.M);
    if (!a.allgather && qmm_tc_uses_pair(ctx, a.w, a.M)) return launch_qmm_tc_pair(ctx, a);
    return dispatch_tc(ctx, a, nullptr, 0);
}

}  // namespace fnn

// ---- entry point that allocates nothing ---------------------------------------------------------

namespace {
// Activation scratch of fnn_cuda_qmatmul_noalloc.  Lives in the module image: every GPU that
// loads the library holds these 8 MiB until the process exits.
constexpr size_t kNoAllocScratchBytes = (size_t)8 << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
// In host code the symbol above is only a stand-in; the device address is looked up once per
// device (with that device current) and kept here.
static void *g_noalloc_scratch_addr[64] = {};
}  // namespace

extern "C" int fnn_cuda_qmatmul_noalloc(fnn_cuda_ctx *ctx, fnn_cuda_qweight *w, const float *a_dev,
                                        float *out_dev, const float *bias_dev, size_t M, int epilogue) {
    using namespace fnn;
    clear_error();
    FNN_REQUIRE(ctx && w && a_dev && out_dev, FNN_ERR_DISPATCH, "qmatmul_noalloc: null argument");
    FNN_REQUIRE(w->ctx->device == ctx->device, FNN_ERR_DISPATCH,
                "qmatmul_noalloc: weight lives on device %d, context on %d", w->ctx->device, ctx->device);
    FNN_REQUIRE(ctx->device >= 0 && ctx->device < 64, FNN_ERR_UNSUPPORTED,
                "qmatmul_noalloc: device index %d out of range", ctx->device);
    FNN_REQUIRE(epilogue >= FNN_EPI_NONE && epilogue <= FNN_EPI_SILU, FNN_ERR_DISPATCH,
                "qmatmul_noalloc: unknown epilogue %d", epilogue);
    FNN_REQUIRE(((uintptr_t)a_dev & 15u) == 0 && ((uintptr_t)out_dev & 15u) == 0, FNN_ERR_DISPATCH,
                "qmatmul_noalloc: pointers must be 16-byte aligned");
    FNN_REQUIRE(qmm_tc_supported(w, M), FNN_ERR_UNSUPPORTED,
                "qmatmul_noalloc: format %d / K=%zu is not served by this entry point", w->fmt, w->K);
    FNN_REQUIRE(M < (1u << 24), FNN_ERR_DISPATCH, "qmatmul_noalloc: M=%zu too large", M);
    if (M == 0) return FNN_OK;
    FNN_CUDA_CHECK(cudaSetDevice(ctx->device), FNN_ERR_DISPATCH);
    if (!g_noalloc_scratch_addr[ctx->device]) {
        void *ptr = nullptr;
        FNN_CUDA_CHECK(cudaGetSymbolAddress(&ptr, g_noalloc_scratch), FNN_ERR_MEMORY);
        FNN_REQUIRE(ptr != nullptr, FNN_ERR_MEMORY, "qmatmul_noalloc: scratch symbol has no address");
        g_noalloc_scratch_addr[ctx->device] = ptr;
    }
    uint8_t *scratch = (uint8_t *)g_noalloc_scratch_addr[ctx->device];
    QmmArgs args{w, a_dev, out_dev, bias_dev, M, epilogue};
    return dispatch_tc(ctx, args, scratch, kNoAllocScratchBytes);
}
