// Skinny-M kernel (1 <= M <= 16) on 8-bit tensor-core operands: the HBM scan of the weights with
// almost no instruction per weight.
//
// Same skeleton as the fp16 fragment kernel (fragment-major weights, one block per SM, groups of
// eight warps that split K, a private cp.async ring per lane), but the codes are fed to
// `mma.sync.m16n8k32` as 8-bit operands:
//   I8   -> s8 operands as stored (no decode at all)
//   I4   -> s8 operands holding 16*q: two masks per word of eight codes
//   FP4  -> s8 operands holding 2*|v| through a byte-permute table, positive and negative codes
//           in separate operands (two accumulators, subtracted at the end): no sign arithmetic
//   I4CB -> the 16 centroids as 14-bit fixed point, 128*hi + lo with hi, lo in [0, 127], looked up from
//           two byte-permute tables with the raw index as selector (two operands, two MMAs per
//           32-element scale block); the block scale multiplies the block's exact integer sum in f32
// (FP8 is not served here: `mma.sync` with e4m3 operands measured slower than the fp16 kernel on this
// part) and the f32 activations are rewritten while they are staged, per batch row, as
//   a ~= dq * (128*hi + lo)        (15-bit fixed point, exact int32 accumulation)
// Partial sums are integers, so the split-K reduction is exact in any order.
// Epilogue as everywhere:  out = act(dq*acc*scale[n] + zero[n]*sum_k a[m,k] + bias[n])
// (src/backend/cpu/microkernels/gemm.rs:2048-2087, src/backend/cpu/matmul.rs:61-71).
#include "frag_common.cuh"
#include "tc_common.cuh"

namespace fnn {

namespace {

using frag::cp_async_commit;
using frag::cp_async_wait;
using frag::group_barrier;
using frag::kCbHalf;

constexpr int kW8 = frag::kWarpsPerGroup;   // warps per group
constexpr int kU8 = frag::kChunkBlocks;     // k-blocks per ring chunk
constexpr int kS8 = 3;   // ring stages per lane (two chunks, 96 KB per SM, in flight)
constexpr int kMma8MaxRows = 16;   // four 8-column groups of (term, batch row) columns

template <int FMT>
struct T8 {
    static constexpr bool four_bit = (FMT == FNN_FMT_I4 || FMT == FNN_FMT_F4 || FMT == FNN_FMT_I4CB);
    static constexpr bool codebook = (FMT == FNN_FMT_I4CB);
    static constexpr int KBLK = four_bit ? 128 : 64;       // k per k-block (4 lanes x 16 bytes per row)
    static constexpr int MMAS = four_bit ? 4 : 2;          // m16n8k32 MMAs per k-block
    static constexpr int PAD = four_bit ? 16 : 64;         // activation row padding (bank spread)
};


__device__ __forceinline__ void mma_s8(int *d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// prmt.b32 in its default mode: selector nibble n picks byte n&7 of {a, b}; bit 3 of the nibble
// replaces the byte by its sign bit replicated eight times.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// Contiguous bytes (a multiple of 16, both ends on 16) into shared memory; reports to `bar`.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     tc::smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
                 : "memory");
}

// Eight 4-bit codes of one word -> the two A registers of one m16n8k32 MMA.
//   I4: lo = 16*q of codes 0,2,4,6 ; hi = 16*q of codes 1,3,5,7 (the activations are staged in the
//       matching order 0,2,4,6,1,3,5,7 of each 8-group)
__device__ __forceinline__ void decode_i4(uint32_t w, uint32_t &lo, uint32_t &hi) {
    lo = (w << 4) & 0xF0F0F0F0u;
    hi = w & 0xF0F0F0F0u;
}
//   F4 (sign | 3-bit magnitude code): the magnitudes 0,.5,1,1.5,2,3,4,6 doubled are the bytes of a
//   table that prmt indexes with the raw code.  A code with its sign bit set makes prmt return the
//   replicated top bit of the table byte, i.e. 0 -- so the raw word yields the positive weights
//   (negative ones as 0) and the word with all sign bits flipped yields the negative weights'
//   magnitudes: pos/neg operands in natural element order, seven ALU operations per eight weights.
__device__ __forceinline__ void decode_f4(uint32_t w, uint32_t &plo, uint32_t &phi, uint32_t &nlo,
                                          uint32_t &nhi) {
    const uint32_t t0 = 0x03020100u, t1 = 0x0C080604u;
    const uint32_t f = w ^ 0x88888888u;
    plo = prmt(t0, t1, w);
    phi = prmt(t0, t1, w >> 16);
    nlo = prmt(t0, t1, f);
    nhi = prmt(t0, t1, f >> 16);
}

//   I4CB (index into 16 centroids): every centroid is carried as v = 128*hi + lo, hi and lo in
//   [0, 127], so a table byte never has its top bit set.  Indices 0..7 come out of one prmt on the
//   raw word (indices 8..15 select "replicated top bit" = 0 there), indices 8..15 out of a second
//   prmt on the word with every index's bit 3 flipped (indices 0..7 give 0 there).  The two halves
//   are not merged: each is an operand of its own MMA into the same accumulator, which costs tensor
//   issue slots (idle here) instead of logic instructions (the limiter).
struct CbTables {
    uint32_t hi[4], lo[4];   // bytes of entries 0-3, 4-7, 8-11, 12-15
};
struct CbOperands {
    uint32_t hi_a[2], hi_b[2], lo_a[2], lo_b[2];   // [codes 0..3 | codes 4..7]; _a: indices 0..7, _b: 8..15
};
__device__ __forceinline__ void decode_cb(const CbTables &t, uint32_t w, CbOperands &o) {
    const uint32_t f = w ^ 0x88888888u, w16 = w >> 16, f16 = f >> 16;
    o.hi_a[0] = prmt(t.hi[0], t.hi[1], w);
    o.hi_a[1] = prmt(t.hi[0], t.hi[1], w16);
    o.hi_b[0] = prmt(t.hi[2], t.hi[3], f);
    o.hi_b[1] = prmt(t.hi[2], t.hi[3], f16);
    o.lo_a[0] = prmt(t.lo[0], t.lo[1], w);
    o.lo_a[1] = prmt(t.lo[0], t.lo[1], w16);
    o.lo_b[0] = prmt(t.lo[2], t.lo[3], f);
    o.lo_b[1] = prmt(t.lo[2], t.lo[3], f16);
}

// Staged byte position of activation k inside its row: where its group of eight goes, plus its place
// inside the group.  I4 reorders inside the group (0,2,4,6,1,3,5,7: even codes of a word, then odd);
// the codebook format keeps the group but orders the sixteen groups of a 128-k block by (word c of a
// scale block, scale block b) instead of (b, c), so that the 32 bytes one lane needs for the four MMAs
// of a k-block are contiguous.
template <int FMT>
__device__ __forceinline__ int group_pos8(int k8) {   // k8: a multiple of 8
    if (FMT == FNN_FMT_I4CB) {
        const int r = k8 & 127, b = r >> 5, c = (r >> 3) & 3;
        return (k8 & ~127) + c * 32 + b * 8;
    }
    return k8;
}
template <int FMT>
__device__ __forceinline__ int inner_pos8(int i) {    // i in [0, 8)
    return FMT == FNN_FMT_I4 ? ((i >> 1) + (i & 1) * 4) : i;
}
template <int FMT>
__device__ __forceinline__ int act_pos8(int k) {
    return group_pos8<FMT>(k & ~7) + inner_pos8<FMT>(k & 7);
}

struct P8 {
    const uint4 *frag;
    const float *frag_bs;   // I4CB: block scales in fragment order
    const uint4 *cb_tables; // I4CB: the centroids as fixed point (cb_tables_kernel)
    const float *scales;
    const float *zeros;
    const float *act;
    float *out;
    const float *bias;
    const float *add;   // sum = out + add, where sum is given
    float *sum;
    int M, N, K;
    int KB, ntiles, tiles_per_group;
    int Kc;      // activations staged per pass (multiple of KBLK)
    int epilogue;
    // PLANES: the activations already rewritten (byte planes [2][M][Kp], row factors and sums)
    const uint8_t *planes;
    const float *dq, *rowsum;
    int Kp;
    int *err_flag;
    int gather_on;
    GatherArgs g;
};

// MULTI: more than one batch row (all rows scanned and staged together); the single-row instantiation
// keeps the shortest prologue.  CG 8-column groups hold the (term, batch row) columns: up to 4 * CG rows.
// PLANES: the rows arrive rewritten (p.planes), by bulk copies (kBulk) or by all threads (kThreads, see launch8); instantiations of
// their own, since the branch and the longer code cost the smallest calls 2 %.
// HELD: groups of eight activations a thread keeps of a single row between the scan and the rewrite, so that the row is read
// once (0: never).  A row that is scanned and then read again behind two more block barriers costs 0.8 us (I8 K=11008 N=4096
// 11.5 -> 10.7 us) to 2 us (I4 K=8192 N=2048 7.8 -> 5.6, one warp of byte stores per plane before).  As few groups as cover
// the row: the prologue is straight-line code that every block runs once, and the instructions of groups
// that are not there cost time too (I8 K=1024 N=2048 2.70 with 2, 3.46 with 8).
enum Planes { kNoPlanes, kBulk, kThreads };
template <int FMT, int CG, int kG8, bool MULTI, int PLANES, int BPS, int HELD>
__global__ void __launch_bounds__(kG8 * kW8 * 32, BPS)
qmm_mma8_kernel(P8 p) {
    using TT = T8<FMT>;
    constexpr int KBLK = TT::KBLK, MMAS = TT::MMAS;
    constexpr int NT = kG8 * kW8 * 32, NW = kG8 * kW8;
    constexpr int UNITS = kU8 * 2;
    constexpr int MR = 4 * CG;                 // batch rows this instantiation can hold
    extern __shared__ __align__(16) unsigned char smem[];
    const int RS = p.Kc + TT::PAD;             // bytes per staged activation row
    const int cols = 2 * p.M;                  // (term, batch row) columns in use
    constexpr bool CB = TT::codebook;
    unsigned char *s_ring = smem;                                         // [NW][S][UNITS][32] uint4
    float *s_ring_bs = reinterpret_cast<float *>(s_ring + (size_t)NW * kS8 * UNITS * 512);   // I4CB: [NW][S][UNITS][32]
    unsigned char *s_act = reinterpret_cast<unsigned char *>(s_ring_bs + (CB ? (size_t)NW * kS8 * UNITS * 32 : 0));  // [cols][RS]
    float *s_red = reinterpret_cast<float *>(s_act + (((size_t)cols * RS + 15) & ~(size_t)15));
    float *s_out = s_red + kG8 * 2 * kW8 * CG * 128;                      // [G][tiles_per_group][CG*128]
    float *s_meta = s_out + (size_t)kG8 * p.tiles_per_group * CG * 128;   // [G][tiles_per_group][16][3]
    float *s_part = s_meta + (size_t)kG8 * p.tiles_per_group * 48;        // [NW][MR][2]
    float *s_dq = s_part + NW * MR * 2;                                   // [MR]
    float *s_rs = s_dq + MR;                                              // [MR]
    float *s_mx = s_rs + MR;                                              // [MR]
    // I4CB: -8192 * (sum of the staged bytes of a 32-element block), per block and column
    int *s_boff = reinterpret_cast<int *>(s_mx + MR);                     // [Kc / 32][8 * CG]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int group = warp / kW8, gw = warp % kW8, gtid = tid - group * kW8 * 32;
    const int g = lane >> 2, c = lane & 3;
    const int gg = group * gridDim.x + blockIdx.x, GG = gridDim.x * kG8;
    // the next kernel on the stream may be set up as soon as an SM has room: its own prologue (scales,
    // first weight copies) then runs under this kernel's tail
    pdl_launch_dependents();
    GatherCursor gc{};
    const int tiles_here = gg < p.ntiles ? (p.ntiles - gg + GG - 1) / GG : 0;
    const bool has_zero = p.zeros != nullptr;
    float *my_out = s_out + (size_t)group * p.tiles_per_group * CG * 128;
    float *my_red = s_red + (size_t)group * 2 * kW8 * CG * 128;
    float *my_meta = s_meta + (size_t)group * p.tiles_per_group * 48;
    unsigned char *my_ring = s_ring + (size_t)warp * kS8 * UNITS * 512 + lane * 16;
    float *my_ring_bs = s_ring_bs + (size_t)warp * kS8 * UNITS * 32;

    CbTables cbt{};

    for (int i = gtid; i < tiles_here * 16; i += kW8 * 32) {
        const int n = (gg + (i >> 4) * GG) * 16 + (i & 15);
        const bool in = n < p.N;
        my_meta[i * 3 + 0] = (in && !CB) ? __ldg(p.scales + n) : 1.0f;
        my_meta[i * 3 + 1] = (in && has_zero) ? __ldg(p.zeros + n) : 0.0f;
    }
    for (int i = tid; i < kG8 * p.tiles_per_group * CG * 128; i += NT) s_out[i] = 0.0f;

    // staged row holding batch column (cg*8 + g), or -1
    int brow[CG];
#pragma unroll
    for (int cg = 0; cg < CG; ++cg) brow[cg] = (cg * 8 + g < cols) ? cg * 8 + g : -1;

    int acci[CG][4], accn[FMT == FNN_FMT_F4 ? CG : 1][4];   // accn: FP4's negative-weight sums
    float accf[CB ? CG : 1][4];                              // I4CB: block sums times block scales
#pragma unroll
    for (int cg = 0; cg < CG; ++cg)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            acci[cg][r] = 0;
            if (FMT == FNN_FMT_F4) accn[cg][r] = 0;
            if constexpr (CB) accf[cg][r] = 0.0f;
        }
    int red_buf = 0;

    const bool vec_ok = (p.K % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.act) & 15u) == 0);
    const int Kpad = p.KB * KBLK;
    constexpr int kHeld = HELD;
    constexpr bool kCanHold = kHeld > 0;
    // Long rows (more than 4096 elements of one group's, 8192 of two): a held group is two quads, one round of the block
    // apart, as scan_rows walks a row, so that the sum of a row has the same last bit whether it is held or scanned.  us of
    // groups of eight / of quads: I8 K=8192 N=2048 5.00 / 4.82, K=11008 N=4096 10.3 / 10.4; FP4 K=8192 N=2048 5.26 / 4.91; I4
    // K=14336 N=2048 6.13 / 6.24, K=11008 N=4096 6.76 / 7.10 (scanned and read again: 7.5).
    constexpr bool kQuads = kHeld >= 4 && !CB;   // (the codebook format takes no row sum, and block sums of its own)
    float hv[kCanHold ? kHeld : 1][8];
    bool held = false;
    __shared__ uint64_t s_rows_bar[1];   // kBulk: the rows of a pass have landed
    __shared__ volatile int s_abort[1];
    if (PLANES == kBulk && tid == 0) {
        tc::mbar_init(s_rows_bar, 1);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }   // (published by the barrier ahead of the first pass)
    for (int k0 = 0; k0 < Kpad; k0 += p.Kc) {
        const int kc_len = min(p.Kc, Kpad - k0);
        const int KBc = kc_len / KBLK;
        const int kb0 = k0 / KBLK;
        const int nch = (KBc + kU8 - 1) / kU8;
        const int cpw = (nch + kW8 - 1) / kW8;
        // issue-side cursor: the next item (tile, chunk-of-this-warp) whose copies go into the ring
        int i_tl = 0, i_j = 0, i_st = 0;
        auto issue_next = [&]() {
            const bool valid = i_tl < tiles_here;
            const int ch = gw + i_j * kW8;
            const uint4 *tile_src = p.frag + ((size_t)(gg + i_tl * GG) * p.KB + kb0) * 64 + lane;
#pragma unroll
            for (int u = 0; u < kU8; ++u) {
                const int kb = ch * kU8 + u;
                const bool ok = valid && (kb < KBc);
                const uint4 *src = ok ? tile_src + (size_t)kb * 64 : p.frag;
                frag::cp_async16(my_ring + (size_t)(i_st * UNITS + u * 2) * 512, src, ok ? 16 : 0);
                frag::cp_async16(my_ring + (size_t)(i_st * UNITS + u * 2 + 1) * 512, src + 32, ok ? 16 : 0);
                if (CB) {   // one block scale per 16-byte unit
                    const float *bsrc = p.frag_bs + (ok ? (src - p.frag) : 0);
                    frag::cp_async4(my_ring_bs + (i_st * UNITS + u * 2) * 32 + lane, bsrc, ok ? 4 : 0);
                    frag::cp_async4(my_ring_bs + (i_st * UNITS + u * 2 + 1) * 32 + lane, bsrc + 32, ok ? 4 : 0);
                }
            }
            cp_async_commit();
            if (++i_j == cpw) {
                i_j = 0;
                ++i_tl;
            }
            if (++i_st == kS8) i_st = 0;
        };
#pragma unroll
        for (int i = 0; i < kS8 - 1; ++i) issue_next();

        if (k0 == 0) {   // under the first weight loads: the per-row scan of the activations
            if (CB) {
                const uint4 hi = __ldg(p.cb_tables), lo = __ldg(p.cb_tables + 1);
                cbt.hi[0] = hi.x; cbt.hi[1] = hi.y; cbt.hi[2] = hi.z; cbt.hi[3] = hi.w;
                cbt.lo[0] = lo.x; cbt.lo[1] = lo.y; cbt.lo[2] = lo.z; cbt.lo[3] = lo.w;
            }
            if (CB && kCanHold)   // columns of a single row that hold nothing (its own two are written as it is staged)
                for (int i = tid; i < kc_len / 32 * 8 * CG; i += NT)
                    if ((i & (8 * CG - 1)) >= 2) s_boff[i] = 0;
            // everything above (scales, the first weight copies) is independent of the kernel before
            // this one on the stream; the activations, the bias and the gather counters are not
            pdl_wait();
            if (p.gather_on) gc = gather_begin(p.g, blockIdx.x * NT + tid);
            // ---- per-row step and sum: max |a| over the whole row first ---------------------
            if (PLANES) {
                // written by the kernel before this one: read through L2, after the wait
                if (tid < p.M) {
                    s_dq[tid] = __ldcg(p.dq + tid);
                    s_rs[tid] = __ldcg(p.rowsum + tid);
                }
            } else if (kCanHold && p.K <= NT * 8 * kHeld && kc_len >= Kpad) {
                held = true;
                if constexpr (kCanHold) frag::hold_row<NT, kHeld, kQuads>(p.act, p.K, vec_ok, hv, s_part);
            } else {
                frag::scan_rows<NT, MULTI ? 4 : 1>(p.act, p.M, p.K, vec_ok, s_part, s_mx, s_rs);
            }
            if (!PLANES && !(kCanHold && held) && tid < p.M) {
                const float bm = s_mx[tid];
                s_dq[tid] = (bm > 0.0f && isfinite(bm)) ? bm / 16256.0f : 1.0f;
            }   // (published by the barrier below)

            // the first poll of the previous step's words was issued at the top; its latency is hidden by now
            if (p.gather_on && gc.step > 1u) gather_check_prev(p.g, gc, gridDim.x * NT);
        }

        __syncthreads();  // previous pass fully consumed
        bool landed = true;
        // ---- stage the activation bytes of [k0, k0 + kc_len) --------------------------------
        if (PLANES == kThreads) {
            const int pieces = kc_len / 16;   // of sixteen bytes
            for (int i = tid; i < cols * pieces; i += NT) {
                const int r = i / pieces, k = (i - r * pieces) * 16;   // plane-major rows, as staged
                const bool in = k0 + k < p.Kp;
                frag::cp_async16(s_act + (size_t)r * RS + k, p.planes + (in ? (size_t)r * p.Kp + k0 + k : 0), in ? 16 : 0);
            }
            cp_async_commit();
            cp_async_wait<0>();
        } else if (PLANES) {
            // One bulk copy per rewritten row (plane-major, as staged), issued by the lanes of a warp.  Sixteen bytes at a
            // time through all threads the copies and their index arithmetic took 1.7 us, and waiting for them drained the
            // weights' ring too (I4 M=8 K=4096 N=4096 7.75 -> 6.45 us).  What the last k-block has beyond the planes is cleared.
            const int bytes = min(kc_len, p.Kp - k0);
            if (warp == 0) {
                if (lane == 0) {
                    tc::fence_proxy_async();   // (an earlier pass read these rows)
                    tc::mbar_expect_tx(s_rows_bar, (uint32_t)(cols * bytes));
                }
                __syncwarp();
                if (lane < cols)
                    bulk_load(s_act + (size_t)lane * RS, p.planes + (size_t)lane * p.Kp + k0, (uint32_t)bytes, s_rows_bar);
            }
            if (kc_len > bytes)
                for (int i = tid; i < cols * (kc_len - bytes) / 16; i += NT) {
                    const int pieces = (kc_len - bytes) / 16, r = i / pieces;
                    *reinterpret_cast<uint4 *>(s_act + (size_t)r * RS + bytes + (i - r * pieces) * 16) = make_uint4(0u, 0u, 0u, 0u);
                }
            landed = tc::mbar_wait(s_rows_bar, (uint32_t)(k0 / p.Kc) & 1u, s_abort, p.err_flag, 0x1000);
        } else if (MULTI && vec_ok && (p.K % 8 == 0)) {
            // eight activations of four rows per thread and step: two 16-byte loads per row in flight,
            // one 8-byte store per (row, plane)
            const int n8 = kc_len / 8;
            for (int i8 = tid; i8 < n8; i8 += NT) {
                const bool in = k0 + i8 * 8 < p.K;
                for (int mb = 0; mb < p.M; mb += 4) {
                    float4 v[4][2];
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        v[m][0] = v[m][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (mb + m < p.M && in) {
                            const float4 *src =
                                reinterpret_cast<const float4 *>(p.act + (size_t)(mb + m) * p.K + k0 + i8 * 8);
                            v[m][0] = ld_after_wait(src);
                            v[m][1] = ld_after_wait(src + 1);
                        }
                    }
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        if (mb + m < p.M) {
                            const float inv = 1.0f / s_dq[mb + m];
                            const float e[8] = {v[m][0].x * inv, v[m][0].y * inv, v[m][0].z * inv, v[m][0].w * inv,
                                                v[m][1].x * inv, v[m][1].y * inv, v[m][1].z * inv, v[m][1].w * inv};
                            uint32_t hi[2], lo[2];
                            int8_pairs<FMT == FNN_FMT_I4>(e, hi, lo);   // (inner_pos8)
                            const int gp = group_pos8<FMT>(i8 * 8);
                            *reinterpret_cast<uint2 *>(s_act + (size_t)(mb + m) * RS + gp) = make_uint2(hi[0], hi[1]);
                            *reinterpret_cast<uint2 *>(s_act + (size_t)(p.M + mb + m) * RS + gp) =
                                make_uint2(lo[0], lo[1]);
                        }
                    }
                }
            }
        } else if (kCanHold && held) {
            float bm, bs;
            frag::fold_held<NT>(s_part, bm, bs);
            const float dq0 = (bm > 0.0f && isfinite(bm)) ? bm / 16256.0f : 1.0f;
            if (tid == 0) {   // (published by the barrier below, for the epilogue)
                s_dq[0] = dq0;
                s_rs[0] = bs;
            }
            const float inv = 1.0f / dq0;
#pragma unroll
            for (int j = 0; j < kHeld; ++j) {
                const int g8 = tid + j * NT;
                float e[8];
#pragma unroll
                for (int q8 = 0; q8 < 8; ++q8) e[q8] = hv[j][q8] * inv;
                uint32_t hi[2], lo[2];
                if constexpr (kQuads) {
                    int8_pairs<false>(e, hi, lo);   // a word of each plane per quad
                    if constexpr (FMT == FNN_FMT_I4) {
                        // I4 reorders inside a group of eight (inner_pos8).  The lanes of a pair hold the halves of two groups
                        // and swap one each: the even lane stores the first round's group, the odd one the second's.
                        const bool odd = lane & 1;
                        const uint32_t h = __shfl_xor_sync(0xFFFFFFFFu, odd ? hi[0] : hi[1], 1);
                        const uint32_t l = __shfl_xor_sync(0xFFFFFFFFu, odd ? lo[0] : lo[1], 1);
                        const uint32_t h0 = odd ? h : hi[0], h1 = odd ? hi[1] : h, l0 = odd ? l : lo[0], l1 = odd ? lo[1] : l;
                        const int k8 = ((tid + (2 * j + odd) * NT) >> 1) * 8;
                        if (k8 >= kc_len) continue;
                        *reinterpret_cast<uint2 *>(s_act + k8) = make_uint2(prmt(h0, h1, 0x6420), prmt(h0, h1, 0x7531));
                        *reinterpret_cast<uint2 *>(s_act + (size_t)RS + k8) = make_uint2(prmt(l0, l1, 0x6420), prmt(l0, l1, 0x7531));
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int k4 = (tid + (2 * j + h) * NT) * 4;
                            if (k4 >= kc_len) continue;
                            *reinterpret_cast<uint32_t *>(s_act + k4) = hi[h];
                            *reinterpret_cast<uint32_t *>(s_act + (size_t)RS + k4) = lo[h];
                        }
                    }
                    continue;
                }
                if (g8 * 8 >= kc_len) continue;   // (beyond K the held values are zero: the padding of the last block)
                int8_pairs<FMT == FNN_FMT_I4>(e, hi, lo);   // (inner_pos8)
                const int gp = group_pos8<FMT>(g8 * 8);
                *reinterpret_cast<uint2 *>(s_act + gp) = make_uint2(hi[0], hi[1]);
                *reinterpret_cast<uint2 *>(s_act + (size_t)RS + gp) = make_uint2(lo[0], lo[1]);
                if (CB) {
                    // the block sums of the pass below while the bytes are still in registers: four
                    // consecutive threads hold one 32-element block (whole half-warps are active here)
                    int sh = __dp4a((int)hi[0], 0x01010101, __dp4a((int)hi[1], 0x01010101, 0));
                    int sl = __dp4a((int)lo[0], 0x01010101, __dp4a((int)lo[1], 0x01010101, 0));
                    const unsigned half = 0xFFFFu << (lane & 16);
                    sh += __shfl_xor_sync(half, sh, 1);
                    sl += __shfl_xor_sync(half, sl, 1);
                    sh += __shfl_xor_sync(half, sh, 2);
                    sl += __shfl_xor_sync(half, sl, 2);
                    if ((lane & 3) == 0)
                        *reinterpret_cast<int2 *>(s_boff + (g8 >> 2) * 8 * CG) = make_int2(-kCbHalf * sh, -kCbHalf * sl);
                }
            }
        } else
        for (int m = 0; m < p.M; ++m) {
            const float *row = p.act + (size_t)m * p.K;
            const float inv = 1.0f / s_dq[m];
            auto put = [&](int k, float a) {
                const float x = a * inv;
                const int pos = act_pos8<FMT>(k);
                int q = __float2int_rn(x);
                q = max(-16256, min(16256, q));
                const int hi = (q + 64) >> 7;
                s_act[(size_t)m * RS + pos] = (unsigned char)(signed char)hi;
                s_act[(size_t)(p.M + m) * RS + pos] = (unsigned char)(signed char)(q - hi * 128);
            };
            if (vec_ok) {
                const int n4 = kc_len / 4;
                for (int b4 = 0; b4 < n4; b4 += 2 * NT) {
                    float4 v[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int i4 = b4 + q * NT + tid;
                        v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (i4 < n4 && k0 + i4 * 4 < p.K)
                            v[q] = ld_after_wait(reinterpret_cast<const float4 *>(row + k0 + i4 * 4));
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int i4 = b4 + q * NT + tid;
                        if (i4 < n4) {
                            put(i4 * 4 + 0, v[q].x);
                            put(i4 * 4 + 1, v[q].y);
                            put(i4 * 4 + 2, v[q].z);
                            put(i4 * 4 + 3, v[q].w);
                        }
                    }
                }
            } else {
                for (int k = tid; k < kc_len; k += NT) put(k, (k0 + k < p.K) ? ld_after_wait(row + k0 + k) : 0.0f);
            }
        }
        if (PLANES != kBulk) {
            __syncthreads();
        } else if (!__syncthreads_and(landed)) {
            // The rows have not come: nothing is stored, the residual's slice least of all.  Copies already in flight land
            // before the block's shared memory goes to another.
            cp_async_wait<0>();
            if (tid == 0)
                for (int i = 0; i < 64; ++i) __nanosleep(1000);
            return;
        }
        if (CB && !(kCanHold && held)) {
            // -8192 * sum of each 32-element block of every staged column: the centroids are carried
            // with an offset of 8192, which the second MMA of a block takes back through its C operand
            const int nblk = kc_len / 32;
            for (int i = tid; i < nblk * 8 * CG; i += NT) {
                const int blk = i / (8 * CG), col = i - blk * (8 * CG), kb = blk >> 2, b = blk & 3;
                int sum = 0;
                if (col < cols) {
                    const unsigned char *src = s_act + (size_t)col * RS + kb * 128 + b * 8;
#pragma unroll
                    for (int c4 = 0; c4 < 4; ++c4) {   // the block's eight bytes of each of its four words
                        const uint2 x = *reinterpret_cast<const uint2 *>(src + c4 * 32);
                        sum = __dp4a((int)x.x, 0x01010101, sum);
                        sum = __dp4a((int)x.y, 0x01010101, sum);
                    }
                }
                s_boff[i] = -kCbHalf * sum;
            }
            __syncthreads();
        }

        if (k0 == 0 && p.bias) frag::copy_bias(p.bias, p.N, gtid, tiles_here, gg, GG, my_meta);

        // ---- stream this K range of every tile of the group ----------------------------------
        int c_st = 0;
        for (int tl = 0; tl < tiles_here; ++tl)
        for (int j = 0; j < cpw; ++j) {
            issue_next();
            cp_async_wait<kS8 - 1>();
            const int ch = gw + j * kW8;
#pragma unroll(CB ? 1 : kU8)
            for (int u = 0; u < kU8; ++u) {
                const int slot = c_st * UNITS + u * 2;
                const uint4 wl = *reinterpret_cast<const uint4 *>(my_ring + (size_t)slot * 512);
                const uint4 wh = *reinterpret_cast<const uint4 *>(my_ring + (size_t)(slot + 1) * 512);
                const int kb_s = min(ch * kU8 + u, KBc - 1);
                if constexpr (CB) {
                    // The unit of lane (g, c) holds word c of the four 32-element blocks of this
                    // k-block: block b is two MMAs for the hi bytes of the centroids plus two for the lo
                    // bytes, eight codes of rows g and g + 8 per lane, and its integer sum is scaled by the
                    // block scale of each row, which sits in the ring slot of lane (g, b).
                    const uint32_t wl4[4] = {wl.x, wl.y, wl.z, wl.w}, wh4[4] = {wh.x, wh.y, wh.z, wh.w};
                    const float4 bl4 = *reinterpret_cast<const float4 *>(my_ring_bs + slot * 32 + (lane & ~3));
                    const float4 bh4 = *reinterpret_cast<const float4 *>(my_ring_bs + (slot + 1) * 32 + (lane & ~3));
                    const float bs_lo[4] = {bl4.x, bl4.y, bl4.z, bl4.w}, bs_hi[4] = {bh4.x, bh4.y, bh4.z, bh4.w};
                    const unsigned char *ap[CG];   // this lane's activation bytes: 8 per scale block
                    const int *op[CG];             // -8192 * block sums of its two columns
#pragma unroll
                    for (int cg = 0; cg < CG; ++cg) {
                        ap[cg] = s_act + (size_t)max(brow[cg], 0) * RS + kb_s * 128 + c * 32;
                        op[cg] = s_boff + (size_t)kb_s * 4 * 8 * CG + cg * 8 + 2 * c;
                    }
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        CbOperands rg, rh;   // row g, row g + 8
                        decode_cb(cbt, wl4[b], rg);
                        decode_cb(cbt, wh4[b], rh);
#pragma unroll
                        for (int cg = 0; cg < CG; ++cg) {
                            uint2 bb = *reinterpret_cast<const uint2 *>(ap[cg] + b * 8);
                            if (brow[cg] < 0) bb = make_uint2(0u, 0u);
                            const uint32_t b0 = bb.x, b1 = bb.y;
                            const int2 off = *reinterpret_cast<const int2 *>(op[cg] + b * 8 * CG);
                            int dh[4] = {0, 0, 0, 0};
                            int dl[4] = {off.x, off.y, off.x, off.y};
                            mma_s8(dh, rg.hi_a[0], rh.hi_a[0], rg.hi_a[1], rh.hi_a[1], b0, b1);
                            mma_s8(dh, rg.hi_b[0], rh.hi_b[0], rg.hi_b[1], rh.hi_b[1], b0, b1);
                            mma_s8(dl, rg.lo_a[0], rh.lo_a[0], rg.lo_a[1], rh.lo_a[1], b0, b1);
                            mma_s8(dl, rg.lo_b[0], rh.lo_b[0], rg.lo_b[1], rh.lo_b[1], b0, b1);
                            accf[cg][0] = fmaf(bs_lo[b], (float)(dh[0] * 128 + dl[0]), accf[cg][0]);
                            accf[cg][1] = fmaf(bs_lo[b], (float)(dh[1] * 128 + dl[1]), accf[cg][1]);
                            accf[cg][2] = fmaf(bs_hi[b], (float)(dh[2] * 128 + dl[2]), accf[cg][2]);
                            accf[cg][3] = fmaf(bs_hi[b], (float)(dh[3] * 128 + dl[3]), accf[cg][3]);
                        }
                    }
                    continue;
                }
                // this lane's activation bytes of the k-block: 16 (8-bit codes) or 32 (4-bit)
                const int boff = kb_s * KBLK + c * (KBLK / 4);
#pragma unroll
                for (int v = 0; v < MMAS / 2; ++v) {  // one 16-byte activation vector feeds two MMAs
                    uint32_t a[2][4];                // [mma][a0 a1 a2 a3]
                    uint32_t an[2][4];               // FP4 only: magnitudes of the negative weights
                    if (TT::four_bit) {
                        const uint32_t wl0 = v ? wl.z : wl.x, wl1 = v ? wl.w : wl.y;
                        const uint32_t wh0 = v ? wh.z : wh.x, wh1 = v ? wh.w : wh.y;
                        if (FMT == FNN_FMT_I4) {
                            decode_i4(wl0, a[0][0], a[0][2]);
                            decode_i4(wh0, a[0][1], a[0][3]);
                            decode_i4(wl1, a[1][0], a[1][2]);
                            decode_i4(wh1, a[1][1], a[1][3]);
                        } else {
                            decode_f4(wl0, a[0][0], a[0][2], an[0][0], an[0][2]);
                            decode_f4(wh0, a[0][1], a[0][3], an[0][1], an[0][3]);
                            decode_f4(wl1, a[1][0], a[1][2], an[1][0], an[1][2]);
                            decode_f4(wh1, a[1][1], a[1][3], an[1][1], an[1][3]);
                        }
                    } else {
                        a[0][0] = wl.x; a[0][2] = wl.y; a[0][1] = wh.x; a[0][3] = wh.y;
                        a[1][0] = wl.z; a[1][2] = wl.w; a[1][1] = wh.z; a[1][3] = wh.w;
                    }
#pragma unroll
                    for (int cg = 0; cg < CG; ++cg) {
                        uint4 b = make_uint4(0, 0, 0, 0);
                        if (brow[cg] >= 0)
                            b = *reinterpret_cast<const uint4 *>(s_act + (size_t)brow[cg] * RS + boff + v * 16);
                        mma_s8(acci[cg], a[0][0], a[0][1], a[0][2], a[0][3], b.x, b.y);
                        mma_s8(acci[cg], a[1][0], a[1][1], a[1][2], a[1][3], b.z, b.w);
                        if (FMT == FNN_FMT_F4) {
                            mma_s8(accn[FMT == FNN_FMT_F4 ? cg : 0], an[0][0], an[0][1], an[0][2], an[0][3], b.x, b.y);
                            mma_s8(accn[FMT == FNN_FMT_F4 ? cg : 0], an[1][0], an[1][1], an[1][2], an[1][3], b.z, b.w);
                        }
                    }
                }
            }
            if (++c_st == kS8) c_st = 0;
            if (j == cpw - 1) {
                // last chunk of a tile: fixed-order reduction over the group's warps
                float *red = my_red + (size_t)red_buf * kW8 * CG * 128;
#pragma unroll
                for (int cg = 0; cg < CG; ++cg)
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        red[(gw * CG + cg) * 128 + r * 32 + lane] =
                            CB ? accf[CB ? cg : 0][r]
                               : (float)(FMT == FNN_FMT_F4 ? acci[cg][r] - accn[FMT == FNN_FMT_F4 ? cg : 0][r]
                                                           : acci[cg][r]);
                        acci[cg][r] = 0;
                        if (FMT == FNN_FMT_F4) accn[cg][r] = 0;
                        if constexpr (CB) accf[cg][r] = 0.0f;
                    }
                group_barrier(group);
                for (int e = gtid; e < CG * 128; e += kW8 * 32) {
                    float s = 0.0f;
#pragma unroll
                    for (int w = 0; w < kW8; ++w) s += red[w * CG * 128 + e];
                    my_out[tl * CG * 128 + e] += s;
                }
                red_buf ^= 1;
            }
        }
        cp_async_wait<0>();
    }
    // the residual of this thread's first output is requested ahead of the barrier
    const int total = tiles_here * 16 * p.M;
    auto add_at = [&](int i) -> float {
        const int tl = i / (16 * p.M), rem = i - tl * 16 * p.M, n = (gg + tl * GG) * 16 + (rem & 15);
        return i < total && n < p.N ? ld_after_wait(p.add + (size_t)(rem >> 4) * p.N + n) : 0.0f;
    };
    float first_add = 0.0f;
    if (p.sum) first_add = add_at(gtid);
    __syncthreads();
    const unsigned step = gc.step;

    // ---- epilogue ----------------------------------------------------------------------------
    for (int i = gtid; i < total; i += kW8 * 32) {
        const int tl = i / (16 * p.M);
        const int rem = i - tl * 16 * p.M;
        const int m = rem >> 4, r16 = rem & 15;
        const int n = (gg + tl * GG) * 16 + r16;
        if (n >= p.N) continue;
        auto at = [&](int col) {
            const int cg = col >> 3, cc = col & 7;
            return my_out[tl * CG * 128 + cg * 128 + ((r16 >> 3) * 2 + (cc & 1)) * 32 + (r16 & 7) * 4 + (cc >> 1)];
        };
        float acc = at(m) * 128.0f + at(p.M + m);
        if (FMT == FNN_FMT_I4) acc *= 0.0625f;  // operands carried 16*q
        if (FMT == FNN_FMT_F4) acc *= 0.5f;     // operands carried 2*|v|
        const float *meta = my_meta + (tl * 16 + r16) * 3;
        float v;
        if (CB) {   // no per-row scale or zero point: the block scales are inside acc
            const float dot = acc * s_dq[m] * __ldg(reinterpret_cast<const float *>(p.cb_tables + 2));
            v = apply_act(p.bias ? __fadd_rn(dot, meta[2]) : dot, p.epilogue);
        } else {
            v = finish_output(acc * s_dq[m], meta[0], meta[1], has_zero ? s_rs[m] : 0.0f, p.bias != nullptr,
                              meta[2], p.epilogue);
        }
        if (!p.gather_on) {
            p.out[(size_t)m * p.N + n] = v;
            if (p.sum) p.sum[(size_t)m * p.N + n] = __fadd_rn(v, i == gtid ? first_add : add_at(i));
        } else {
            gather_store(p.g, step, m, n, v);
        }
    }
    if (p.gather_on) gather_finish(p.g, step, p.M, p.N);
}

bool rewritten_once(const QmmArgs &a) {
    const size_t elems = a.M * a.w->K;
    return elems > 16384 || (a.M > 4 && elems >= 8192);
}

template <int FMT, int CG, int kG8, bool MULTI, int BPS = 1, int HELD = 0>
int launch8(fnn_cuda_ctx *ctx, const QmmArgs &a) {
    using TT = T8<FMT>;
    const fnn_cuda_qweight *w = a.w;
    P8 p{};
    p.frag = w->frag;
    p.frag_bs = w->frag_bs;
    p.cb_tables = w->cb_tables;
    p.scales = w->scales;
    p.zeros = w->zeros;
    p.act = a.a;
    p.out = a.out;
    p.bias = a.bias;
    p.add = a.add;
    p.sum = a.sum;
    p.M = (int)a.M;
    p.N = (int)w->N;
    p.K = (int)w->K;
    p.KB = (int)div_ceil(w->K, (size_t)TT::KBLK);
    p.ntiles = (int)div_ceil(w->N, 16);
    p.epilogue = a.epilogue;
    p.gather_on = a.gather != nullptr;
    if (a.gather) p.g = *a.gather;
    // Several rows: every block scans and rewrites all of them, which costs more than a kernel that does it once
    // as soon as there is enough to rewrite (rewritten_once).  us in the blocks / once: I4 K=4096 N=4096 M=2 6.3 / 6.3, M=4 7.3 / 6.7,
    // M=8 10.4 / 7.6; I8 K=11008 N=4096 M=2 13.6 / 12.8, M=4 16.3 / 13.5; I8 K=1024 N=2048 M=4 4.1 / 4.6, M=8 5.7 / 5.0;
    // I4 K=4096 N=28672 M=4 15.3 / 15.8.  (The codebook format stages groups of eight bytes: slower this way.)
    if (MULTI && !TT::codebook && !a.gather && rewritten_once(a)) {
        const tc::PrepLayout lay = tc::prep_layout(2, 1, a.M, w->K);
        // (a capture that finds the scratch buffer too small keeps to the blocks)
        if (ctx->scratch_bytes >= lay.bytes || !stream_capturing(ctx)) {
            int rc = ensure_scratch(ctx, lay.bytes);
            if (rc != FNN_OK) return rc;
            uint8_t *planes = (uint8_t *)ctx->scratch;
            float *dq = (float *)(planes + lay.dq), *rowsum = (float *)(planes + lay.rowsum);
            rc = tc::launch_act_prep(ctx, a, tc::KIND_I8, 2, FMT == FNN_FMT_I4, (int)lay.Kp, planes, dq, rowsum);
            if (rc != FNN_OK) return rc;
            p.planes = planes;
            p.dq = dq;
            p.rowsum = rowsum;
            p.Kp = (int)lay.Kp;
            p.err_flag = ctx->err_flag;
        }
    }
    const int cols = 2 * p.M;   // int8 pairs
    constexpr int MR = 4 * CG;
    const size_t ring = (size_t)kG8 * kW8 * kS8 * kU8 * 2 * (512 + (TT::codebook ? 128 : 0));
    const size_t fixed = ring + (size_t)(kG8 * 2 * kW8 * CG * 128 + kG8 * kW8 * MR * 2 + 3 * MR) * 4 + 64;
    const size_t per_tile = (size_t)kG8 * (CG * 512 + 192);
    frag::FragSizing sz;
    const bool fits = frag::size_frag_launch(
        ctx->sm_count, p.ntiles, kG8, p.KB * TT::KBLK, TT::KBLK, fixed, per_tile,
        [&](int kc) {
            return ((((size_t)cols * (kc + TT::PAD)) + 15) & ~(size_t)15) +
                   (TT::codebook ? (size_t)(kc / 32) * 8 * CG * 4 : 0);
        },
        &sz, BPS);
    if constexpr (BPS > 1)
        if (!fits) return launch8<FMT, CG, kG8, MULTI, 1, HELD>(ctx, a);
    FNN_REQUIRE(fits, FNN_ERR_UNSUPPORTED,
                "qmatmul: shared memory budget exceeded for M=%d on the 8-bit fragment kernel", p.M);
    p.tiles_per_group = sz.tiles_per_group;
    p.Kc = sz.Kc;
    auto kern = qmm_mma8_kernel<FMT, CG, kG8, MULTI, kNoPlanes, BPS, HELD>;
    if constexpr (MULTI && !TT::codebook)
        if (p.planes) kern = qmm_mma8_kernel<FMT, CG, kG8, MULTI, kBulk, BPS, HELD>;
    // Long I8 rows in front of more than a tile per SM: the weights are twice as many bytes, and behind bulk copies they start
    // late.  us by bulk copies / by all threads: M=2 K=11008 N=4096 13.6 / 13.1, M=4 K=8192 N=4096 10.9 / 10.2, N=11008 21.1 /
    // 19.4, M=3 K=8192 N=28672 46.3 / 40.2; but M=4 K=8192 N=2048 7.4 / 8.1, K=5000 N=4096 7.5 / 8.3, K=4104 N=11008 12.6 / 13.0,
    // and of the 4-bit formats I4 M=4 K=11008 N=4096 9.4 / 10.8, M=8 K=4096 N=11008 10.2 / 10.5, FP4 M=4 K=11008 N=2048 8.8 / 10.6.
    if constexpr (MULTI && FMT == FNN_FMT_I8)
        if (p.planes && p.K >= 8192 && p.ntiles > ctx->sm_count) kern = qmm_mma8_kernel<FMT, CG, kG8, MULTI, kThreads, BPS, HELD>;
    FNN_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sz.smem),
                   FNN_ERR_DISPATCH);
    FNN_CUDA_CHECK(launch_pdl(kern, sz.grid, kG8 * kW8 * 32, sz.smem, ctx, p), FNN_ERR_DISPATCH);
    ctx->launches++;
    ctx->last_path = "mma8";
    ctx->last_kernel = p.planes ? "mma8-rewritten" : "mma8";
    return FNN_OK;
}

// A single batch row: groups per block and blocks per SM (the registers of a thread are bounded for that many).  The SMs are
// shared with the blocks of the next kernel on the stream, which prefetch their weights as soon as one fits, so smaller
// blocks win where there are enough of them; every block stages the row, so a long one wants few of them; and up to one
// tile per SM two blocks on an SM would leave another idle.  us, one group x 1 / x 2 / x 3 blocks per SM, two
// groups x 1:
//   up to a tile per SM        I8 K=8192 N=2048 6.18 / 6.72 / 8.35 / 6.57;  FP4 K=8192 N=2048 5.64 / 7.05 / 8.45 / 6.79;
//                              codebook K=8192 N=2048 7.47 / 11.2 / - / 10.4
//   K up to 4096               I4 K=4096 N=4096 - / 4.61 / 5.13 / 4.98;  FP4 K=4096 N=11008 - / 7.80 / 9.84 / 8.41;
//                              I8 K=2048 N=8192 - / 5.05 / 5.65 / 5.70;  codebook K=2048 N=8192 7.77 / 6.60 / - / 7.56
//   and I8 of four tiles a SM  K=4096 N=11008 11.1 / 10.0 / 9.84 / 9.88, N=14336 13.4 / 11.9 / 11.6 / 12.3
//   longer                     I8 K=11008 N=4096 - / 11.1 / 15.8 / 10.7, K=8192 N=28672 - / 37.7 / 41.1 / 37.5; I4 K=14336 N=4096
//                              - / 9.20 / 16.0 / 8.62
//   a little over a tile a SM  FP4 K=4096 N=2560 4.74 / 5.20, N=3584 4.91 / 4.89;  codebook K=4096 N=2560 6.6 / 7.2, N=3072 6.8 /
//                              7.1, K=2048 N=2560 4.65 / 4.77, N=3072 4.76 / 4.61
//   codebook, two to three     K=2048 N=5632 - / 6.5 / - / 5.9;  K=4096 N=6144 - / 9.5 / - / 8.7
//   and by length              K=8192 N=4096 10.8 / - / - / 10.5, N=8192 17.9 / - / - / 17.3, N=28672 48.7 / - / - / 46.9;  K=11008
//                              N=4096 15.0 / 17.4 / - / 15.3;  K=20000 N=4096 (not held) 28.0 / - / - / 25.3
template <int FMT>
int launch8_single(fnn_cuda_ctx *ctx, const QmmArgs &a, int ntiles) {
    const int units = (int)div_ceil(a.w->K, 8), sms = ctx->sm_count;
    bool one = ntiles <= sms;   // a block of one group on an SM
    if (FMT == FNN_FMT_F4 && units > 256 && units <= 512) one = 4 * ntiles < 5 * sms;
    if (T8<FMT>::codebook && units <= 512) one = 4 * ntiles < (units > 256 ? 6 : 5) * sms;
    if (!one) {
        if constexpr (T8<FMT>::codebook) {
            if (units <= 512 ? ntiles > 2 * sms && ntiles <= 3 * sms : units <= 1024)
                return launch8<FMT, 1, 2, false, 1, 2>(ctx, a);
            if (units <= 512) return launch8<FMT, 1, 1, false, 2, 2>(ctx, a);
            if (units > 2048) return launch8<FMT, 1, 2, false>(ctx, a);
        } else {
            if constexpr (FMT == FNN_FMT_I8)
                if (units <= 512 && ntiles >= 4 * sms) return launch8<FMT, 1, 1, false, 3, 2>(ctx, a);
            if (units <= 512) return launch8<FMT, 1, 1, false, 2, 2>(ctx, a);
            return units <= 1024 ? launch8<FMT, 1, 2, false, 1, 2>(ctx, a) : launch8<FMT, 1, 2, false, 1, 4>(ctx, a);
        }
    }
    return units <= 512    ? launch8<FMT, 1, 1, false, 1, 2>(ctx, a)
           : units <= 1024 ? launch8<FMT, 1, 1, false, 1, 4>(ctx, a)
                           : launch8<FMT, 1, 1, false, 1, 8>(ctx, a);
}

// Several batch rows: two groups per block while that still gives (nearly) every SM a block, else one, so that the tiles
// spread over more SMs.  (us with three / two groups: I8 M=4 K=4096 N=11008 12.4 / 12.3, K=2048 N=8192 6.8 / 6.5; I4 M=4 K=4096
// N=11008 9.0 / 8.5, K=8192 N=28672 29.8 / 26.4.)  Three where the block itself scans two or three rows of more than 4096 elements,
// which more threads do faster, and no round of tiles is added: M=2 K=5000 N=13001 I8 14.3 / 14.8, I4 10.4 / 10.8, FP4 13.3 / 13.6;
// M=2 K=8192 N=28672 I8 40.8 / 41.4, I4 24.1 / 24.4; M=3 K=5000 N=13001 I8 15.3 / 15.7, I4 10.8 / 11.6, but FP4 14.7 / 14.2.  With
// as many rounds either way two win again: I8 M=2 K=8192 N=8192 16.7 / 16.2.
template <int FMT, int CG>
int launch8_cg(fnn_cuda_ctx *ctx, const QmmArgs &a) {
    const int ntiles = (int)div_ceil(a.w->N, 16);
    if constexpr (CG == 1)
        if (a.M == 1) return launch8_single<FMT>(ctx, a, ntiles);
    if constexpr (CG == 1 && !T8<FMT>::codebook) {
        auto rounds = [&](int groups) { return div_ceil((size_t)ntiles, (size_t)groups * ctx->sm_count); };
        if (a.w->K > 4096 && !rewritten_once(a) && (FMT != FNN_FMT_F4 || a.M == 2) && rounds(3) < rounds(2))
            return launch8<FMT, 1, 3, true>(ctx, a);
    }
    if ((ntiles + 1) / 2 >= ctx->sm_count * 4 / 5) return launch8<FMT, CG, 2, true>(ctx, a);
    return launch8<FMT, CG, 1, true>(ctx, a);
}

template <int FMT>
int launch8_fmt(fnn_cuda_ctx *ctx, const QmmArgs &a) {
    const int M = (int)a.M;
    FNN_REQUIRE(M >= 1 && M <= kMma8MaxRows, FNN_ERR_UNSUPPORTED,
                "qmatmul: the 8-bit fragment kernel holds up to %d batch rows as int8 pairs (M=%d)",
                kMma8MaxRows, M);
    if (M <= 4) return launch8_cg<FMT, 1>(ctx, a);
    if (M <= 8) return launch8_cg<FMT, 2>(ctx, a);
    return launch8_cg<FMT, 4>(ctx, a);
}

}  // namespace

bool qmm_mma8_supported(const fnn_cuda_qweight *w, size_t M) {
    // Every format whose values are small integers (I8, I4, and FP4 doubled) runs on s8 operands with
    // the activations as exact int8 pairs; `mma.sync` with e4m3 operands runs at a fraction of the
    // fp16 rate on this part, so FP8 stays on the fp16 kernel.
    return (w->fmt == FNN_FMT_I8 || w->fmt == FNN_FMT_I4 || w->fmt == FNN_FMT_F4 || w->fmt == FNN_FMT_I4CB) &&
           M >= 1 &&
           M <= (size_t)kMma8MaxRows &&
           w->N < (1u << 27) &&
           w->K < (1u << 27);
}

// Consumer side of the fused gather: polls (bounded) every word of the last completed step in this
// rank's buffer and, if `out` is given, writes the values as plain f32 [world][rows][n_stride].
__global__ void gather_wait_kernel(const unsigned long long *words, const unsigned *counters, int world,
                                   int n_stride, float *out, int *err_flag) {
    const unsigned step = counters[0];
    const int rows = (int)counters[2];
    if (step == 0u) return;
    const unsigned long long *slot = words + (size_t)(step & 1u) * world * kGatherRows * n_stride;
    const int per_rank = rows * n_stride;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < world * per_rank; i += gridDim.x * blockDim.x) {
        const int r = i / per_rank;
        unsigned long long w;
        if (!wait_word(slot + (size_t)r * kGatherRows * n_stride + (i - r * per_rank), step, w)) {
            raise_error(err_flag, 0x100);
            return;
        }
        if (out) out[i] = __uint_as_float((unsigned)w);
    }
}

int launch_gather_wait(fnn_cuda_ctx *ctx, const unsigned long long *my_words, const unsigned *counters,
                       int world, int n_stride, float *out) {
    const int blocks = (int)div_ceil((size_t)world * kGatherRows * n_stride, 256 * 4);
    gather_wait_kernel<<<blocks < 1 ? 1 : blocks, 256, 0, ctx->stream>>>(my_words, counters, world, n_stride,
                                                                        out, ctx->err_flag);
    FNN_CUDA_CHECK(cudaGetLastError(), FNN_ERR_DISPATCH);
    ctx->launches++;
    return FNN_OK;
}

int launch_qmm_mma8(fnn_cuda_ctx *ctx, const QmmArgs &a) {
    switch (a.w->fmt) {
    case FNN_FMT_I8:
        return launch8_fmt<FNN_FMT_I8>(ctx, a);
    case FNN_FMT_I4:
        return launch8_fmt<FNN_FMT_I4>(ctx, a);
    case FNN_FMT_F4:
        return launch8_fmt<FNN_FMT_F4>(ctx, a);
    case FNN_FMT_I4CB:
        return launch8_fmt<FNN_FMT_I4CB>(ctx, a);
    }
    return set_error(FNN_ERR_UNSUPPORTED, "qmatmul: the 8-bit fragment kernel does not cover format %d",
                     a.w->fmt);
}

}  // namespace fnn
