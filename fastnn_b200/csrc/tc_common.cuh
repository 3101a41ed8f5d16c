// Shared pieces of the tcgen05 kernels: PTX wrappers, operand descriptors, the epilogue arithmetic and the
// host helpers that encode tensor maps and rewrite the activations.
#pragma once

#include "common.cuh"

#include <cuda.h>

namespace fnn {
namespace tc {

constexpr int kTileN = 128;        // weight rows (output channels) per CTA tile = MMA M
constexpr int kKBlockBytes = 128;  // bytes of K per pipeline stage = one 128B swizzle row
constexpr int kEpiWarps = 8;                      // two per TMEM lane quadrant
constexpr long long kWaitCycles = 2000000000LL;  // ~1 s: far beyond any legitimate wait

enum { KIND_I8 = 0, KIND_F8 = 1, KIND_F16 = 2 };
// How the weight tile reaches the MMA: straight from TMA (I8, FP8, FP4), or through the transform
// warps (I4 -> int8, codebook -> fp16).
enum { WF_TMA = 0, WF_I4 = 1, WF_CB = 2 };
// Transform warps: the codebook's table lookups keep twice as many busy as the two masks per word of I4.
__host__ __device__ constexpr int xf_warps(int wf) { return wf == WF_TMA ? 0 : wf == WF_I4 ? 8 : 16; }
constexpr int kFmtE4M3 = 0, kFmtE2M1 = 5;        // operand format codes of kind::f8f6f4

// ---- PTX wrappers -------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
// One lane of the warp.  The single-thread roles (TMA producer, MMA issuer) run under this predicate, not
// under `lane == 0`: the compiler then knows that exactly one thread is active and keeps descriptors in
// uniform registers, which is where the copy and MMA instructions take them from.  Issuing the four MMAs and the
// commit of a step took 339 cycles under `lane == 0` and takes 70 under elect.sync (clock64 around
// them); a step of a small-batch layer went from 580 to 347 cycles, I8 K=4096 N=11008 at M=16 from 15.1 to
// 12.4 us.
__device__ __forceinline__ bool elect_one() {
    uint32_t is_leader;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(is_leader));
    return is_leader != 0;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false (after raising the error flags) if the phase never completes or
// another role has already given up.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                          int *err_flag, int code) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitCycles) {
            *abort_flag = 1;
            raise_error(err_flag, code);
            return false;
        }
    }
}
// The same for a whole warp, with one answer for all of its lanes.  Each lane polls by itself, so one may see the phase
// complete while another sees the abort flag, and what follows is for a converged warp: tcgen05 loads, and the
// arrivals at a cluster barrier, of which every warp owes the same number on every path.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *err_flag,
                                               int code) {
    return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, abort_flag, err_flag, code));
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0,
                                            int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
// Brings a tensor map (a kernel parameter) into the descriptor cache ahead of its first copy.
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap *map, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(map), "r"(c0), "r"(c1),
                 "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0,
                                            int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}
template <int KIND>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
    if (KIND == KIND_I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else if (KIND == KIND_F8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
// The same with the A operand in TMEM (lane = row, a 32-bit column = four 8-bit or two 16-bit k).
template <int KIND>
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
    if (KIND == KIND_I8) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}
// Registers of a thread -> 8 or 16 consecutive columns of its TMEM lane.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
            taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// shared::cluster address of a shared-memory object in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(const void *p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t ld_cluster(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 32 lanes x 16 consecutive 32-bit columns of TMEM -> 16 registers per thread.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes, 128B-swizzled
// (what TMA writes with CU_TENSOR_MAP_SWIZZLE_128B): 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);  // start address / 16
    d |= (uint64_t)1 << 16;                       // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;             // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                       // descriptor version for sm_100
    d |= (uint64_t)2 << 61;                       // layout type: SWIZZLE_128B
    return d;
}

// Instruction descriptor: D format, A/B formats, K-major both, N (>>3) and M (>>4).  `a_fmt`: the
// A operand's format code for kind::f8f6f4 (e4m3 or e2m1); B is e4m3 there.  Format 0 is F16 for
// kind::f16.
__host__ __device__ constexpr uint32_t make_idesc(int kind, int n_cols, int a_fmt, int m_rows) {
    return (kind == KIND_I8 ? (2u << 4) | (1u << 7) | (1u << 10)   // S32 accum, signed 8-bit A and B
                            : (1u << 4) | ((uint32_t)a_fmt << 7) | (0u << 10))  // F32 accum
           | ((uint32_t)(n_cols >> 3) << 17) | ((uint32_t)(m_rows >> 4) << 24);
}
// generic-proxy writes to shared memory -> visible to the async proxy (the tensor core's reads)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// One chunk of outputs: `rows` batch rows of one channel, `pitch` apart from `at` on (a warp writes 32 consecutive channels), and
// where `sum` is given the sums with `add` beside them, eight loads in flight together.
template <int W>
__device__ __forceinline__ void store_chunk(float *out, const float *add, float *sum, size_t at, size_t pitch, int rows,
                                            const float (&v)[W]) {
#pragma unroll
    for (int j = 0; j < W; ++j)
        if (j < rows) out[at + (size_t)j * pitch] = v[j];
    if (!sum) return;
#pragma unroll
    for (int h = 0; h < W; h += 8) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = h + j < rows ? ld_after_wait(add + at + (size_t)(h + j) * pitch) : 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (h + j < rows) sum[at + (size_t)(h + j) * pitch] = __fadd_rn(v[h + j], x[j]);
    }
}

// The epilogue arithmetic of one chunk: W batch rows (8 or 16) of one output channel.  `fac` carries the
// rows' dq (lanes 0 .. W-1) and row sums (lanes 16 ..).  One branch per chunk, on the activation, behind the arithmetic that
// all of them share: a branch per output ran the two warps of a scheduler one after another, and a copy of the whole
// chunk per activation is code that every launch fetches (us with a copy / with one: four I4 decoder layers at 64 rows
// 302.2 / 299.4, six I8 pairs at 16 rows 154.4 / 153.4).
template <int KIND, int T, int W>
__device__ __forceinline__ void finish_chunk(const uint32_t (&r)[T][W], float fac, float scale, float zero, float bias,
                                             bool has_bias, float acc_scale, int epilogue, float (&v)[W]) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const float dq_m = __shfl_sync(0xFFFFFFFFu, fac, j);
        const float rs_m = __shfl_sync(0xFFFFFFFFu, fac, 16 + j);
        float acc;
        if (T == 1)
            acc = __uint_as_float(r[0][j]);
        else if (KIND == KIND_I8)
            acc = ((float)(int)r[0][j] * 128.0f + (float)(int)r[T > 1 ? 1 : 0][j]) * acc_scale;
        else if (T == 3)
            acc = (__uint_as_float(r[0][j]) + __uint_as_float(r[T > 1 ? 1 : 0][j])) + __uint_as_float(r[T - 1][j]);
        else
            acc = __uint_as_float(r[0][j]) + __uint_as_float(r[T > 1 ? 1 : 0][j]);
        // dot*scale + zero*sum(a) with the reference's separate roundings, then act(x + bias)
        const float x = __fadd_rn(__fmul_rn(acc * dq_m, scale), __fmul_rn(zero, rs_m));
        v[j] = has_bias ? __fadd_rn(x, bias) : x;
    }
    switch (epilogue) {
    case FNN_EPI_RELU:
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = apply_act_fast(v[j], FNN_EPI_RELU);
        break;
    case FNN_EPI_GELU:
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = apply_act_fast(v[j], FNN_EPI_GELU);
        break;
    case FNN_EPI_SILU:
#pragma unroll
        for (int j = 0; j < W; ++j) v[j] = apply_act_fast(v[j], FNN_EPI_SILU);
        break;
    default:
        break;
    }
}

// One 16-byte unit of packed nibbles (32 codes of one row) as an MMA operand.
//   I4: 32 int8 holding 16*q, inside every word of eight the even codes, then the odd ones (the
//   activation planes carry the same order inside every group of eight k)
__device__ __forceinline__ void widen_i4(const uint4 &w, uint32_t *o) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        o[2 * j] = (ww[j] << 4) & 0xF0F0F0F0u;
        o[2 * j + 1] = ww[j] & 0xF0F0F0F0u;
    }
}
//   codebook: 32 fp16 of block scale x centroid, one rounding (the unit is one scale block).  Bound by
//   instruction issue: per code a table load, half a packed multiply, half a conversion, and one byte
//   permute that puts the code (times four, masked out of its word for four codes at once) under the
//   upper bytes of the table's 256-byte-aligned address.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ float lds_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void widen_cb(const uint4 &w, float bs, uint32_t table, uint32_t *o) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t even = (ww[j] << 2) & 0x3C3C3C3Cu, odd = (ww[j] >> 2) & 0x3C3C3C3Cu;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float lo = lds_f32(prmt(even, table, 0x7650u + q));
            const float hi = lds_f32(prmt(odd, table, 0x7650u + q));
            asm("{\n\t.reg .b64 c, s;\n\t.reg .f32 x, y;\n\t"
                "mov.b64 c, {%1, %2};\n\tmov.b64 s, {%3, %3};\n\t"
                "mul.rn.f32x2 c, c, s;\n\tmov.b64 {x, y}, c;\n\t"
                "cvt.rn.f16x2.f32 %0, y, x;\n\t}"
                : "=r"(o[4 * j + q])
                : "f"(lo), "f"(hi), "f"(bs));
        }
    }
}
// The 16 centroids' place in shared memory: the next 256-byte boundary of the shared window after `p`.
constexpr int kTableBytes = 64 + 255;
__device__ __forceinline__ float *table_after(void *p) {
    return reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(p) + ((256u - (smem_u32(p) & 255u)) & 255u));
}

// ---- host helpers (qmm_tc.cu) ---------------------------------------------------------------------

constexpr size_t kMaxSmem = 227 * 1024;   // dynamic shared memory a block can have
constexpr size_t kHalfSmem = 114 * 1024;  // no two blocks of this fit an SM's 228 KB (1 KB of each is the system's)
static_assert(2 * (kHalfSmem + 1024) > 228 * 1024 && kHalfSmem <= kMaxSmem, "two blocks would share an SM");

int encode_map(CUtensorMap *map, void *base, int rank, const cuuint64_t *dims, const cuuint64_t *strides,
               const cuuint32_t *box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B,
               CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_UINT8);
int encode_weight_map(CUtensorMap *map, const fnn_cuda_qweight *w);
int encode_block_scale_map(CUtensorMap *map, const fnn_cuda_qweight *w);
// Narrow terms per activation.
int tc_terms(int fmt, size_t M);
// Microseconds of the parts of a call, for the choice between the kernels and of the tile height.
struct TileCosts {
    // single-SM kernel: a call; a K block of 128 (and what 256 columns add); the epilogue of a batch row of a tile; an
    // extra CTA of a K split (and what 128 columns add)
    double fixed, step, step_256, row, part, part_128;
    // two-SM kernel: a call; a K block (and what 256 columns add); a row's epilogue
    double pair_fixed, pair_step, pair_step_256, pair_row;
};
const TileCosts &tile_costs(int fmt, int terms);
// Output rows that start off a 32-byte sector, in a result that L2 does not keep until both halves of a sector are written,
// stretch the epilogues, the single-SM kernel's more (the two SMs of a pair write neighbouring channels at the same
// time).  us single / pair, rows on sectors -> off: FP8 M=1601 K=1920 N=8704 -> 8718 53.4 / 61.4 -> 84.2 / 71.6, M=3165 K=2560
// N=3456 -> 3465 59.1 / 61.2 -> 73.7 / 65.1; of 22 MB (M=900 N=6016 -> 6001) 22.5 / 23.1 -> 24.0 / 23.6.
inline bool splits_sectors(size_t M, size_t N) { return N % 8 != 0 && M * N * 4 > (size_t)32 << 20; }
// Whole tiles in waves over `units` SMs or pairs: the first K loop and the last epilogue are exposed; in between, where the
// accumulators are double-buffered, the longer of both per wave and half of the shorter, which competes for the
// same issue slots and shared memory (half: fitted, 0.43 to 0.62 by format); else both.
inline double tile_time(long long tiles, int units, double main_loop, double epilogue, bool two_buffers) {
    const double waves = (double)((tiles + units - 1) / units);
    const double longer = main_loop > epilogue ? main_loop : epilogue, both = main_loop + epilogue;
    const double wave = two_buffers ? 0.5 * (longer + both) : both;
    return both + (waves - 1) * wave;
}
// Launches the rewrite of the activations as `terms` narrow planes, their row factors and row sums.
int launch_act_prep(fnn_cuda_ctx *ctx, const QmmArgs &a, int kind, int terms, bool perm8, int Kp, uint8_t *bq, float *dq,
                    float *rowsum);
// Where a call's rewritten activations, row factors and row sums lie in its scratch.
struct PrepLayout {
    size_t Kp;            // bytes of a row of a plane
    size_t dq, rowsum;    // byte offsets behind the planes [terms][M][Kp]
    size_t bytes;
};
PrepLayout prep_layout(int terms, int elem_bytes, size_t M, size_t K);
int encode_act_map(CUtensorMap *map, void *planes, const PrepLayout &l, int terms, size_t M, int box_rows, int box_planes);

}  // namespace tc
}  // namespace fnn
