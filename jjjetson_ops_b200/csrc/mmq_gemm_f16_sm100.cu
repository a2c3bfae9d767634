// Prefill-regime multiply with the block scales folded into the operands: both matrices are
// dequantised to fp16 on their way to the tensor core and multiplied by tcgen05.mma.kind::f16 with
// fp32 accumulation in tensor memory, so nothing is drained or rescaled between blocks.
//
// Work to replace: q4_0_q8_1_mat_mul_kernel (reference src/cuda/mm_q4_0_q8_1.cu:164-289) for large
// batches.  The reference adds, per 32-wide block, d4 * (sumi * d8 - 8 * s8) (mm_q4_0_q8_1.cu:92).
// With sumi = sum(q4 * q8) that is
//     sum_i ((q4_i - 8) * d4) * (q8_i * d8)   +   (-8 * d4) * (s8 - d8 * sum_i q8_i)
// The first term is a plain product of two fp16 matrices B[n][k] = (q4 - 8) * d4 and
// A[m][k] = q8 * d8; the second is rank one per block and joins the same accumulator as one more
// MMA per 128 values of K (operands s8 - d8 * sum(q8), computed in fp32, and -8 * d4, exact).  It
// vanishes up to the rounding of s8 when the quantizer stored s = d * sum(q), and carries the
// quantisation residue when it stored the sum of the unquantised values.
//
// Precision.  q4 - 8 and q8 are exact in fp16; their products with the fp16 scales are rounded once
// to fp16 (relative error <= 2^-11 per element), the accumulation is fp32.  The result differs from
// the reference formula by about 3e-4 of the largest output on the configurations this kernel is
// measured on, where the integer kernels differ by 1e-6: it meets the 1e-3 bound against the
// dequantised product but not bit-level parity of the per-block sums; JQ_OPT_PREFILL_EXACT keeps the
// automatic choice, which takes it from 64 columns on, to the integer kernels.  How K is split does
// not show in that error.  Operands must stay inside fp16's range: |x| <= 65504 for the activations, and
// scales whose products are not subnormal (|d| * |q| >= 6.1e-5) keep full precision.
//
// @@DESCRIPTION@@
#include <mutex>
#include <vector>

#include "gemm_f16_plan.h"
#include "tc_common.cuh"

namespace jq {

namespace {

constexpr int HF_ROWS = 128;      // weight rows per CTA: the lanes of its tensor memory
constexpr int HF_W_SLOT_BYTES = HF_ROWS * Q8_BYTES;  // raw weights, two chunks (144 bytes of each row) per slot
static_assert(2 * 4 * Q4_BYTES == Q8_BYTES, "a weight slot is two chunks of 72 bytes per row");
constexpr uint32_t HF_A_COLS = 64;   // tensor-memory columns of a chunk's weights: 128 fp16 values
constexpr uint32_t HF_Z_COLS = 8;    // of -8 * d4 of sixteen blocks
constexpr int HF_TMEM_COLS = 512;
constexpr int HF_EPI_WARPS = 16;     // warps that read the accumulator: four per quarter of the lanes
constexpr int HF_MAX_MATS = 4;

// CG CTAs (one, or two on neighbouring SMs: cta_group::2) share a tile of CG * 128 weight rows and NT activation columns.
template <int CG, int NT>
struct HfTile {
    static constexpr int X_ROWS = NT / CG;               // activation columns that a CTA converts
    static constexpr int X_BOX = X_ROWS * 128;           // bytes of 64 fp16 values of K
    static constexpr int X_BYTES = 2 * X_BOX;            // ... of a chunk
    static constexpr int Z_BYTES = X_ROWS * 32;          // fp16 residues of sixteen blocks
    static constexpr int RAW_BYTES = X_ROWS * Q8_BYTES;  // a chunk's activation blocks as they lie in global memory
    // chunks in flight: what tensor memory (accumulator, weights, rank-one operands) and shared memory hold
    static constexpr int STAGES = NT == 256 ? 3 : CG == 2 ? 5 : 4;
    static constexpr int RAW_SLOTS = NT == 256 ? 3 : CG == 2 ? 5 : 2;
    static constexpr int W_SLOTS = NT == 256 ? 3 : CG == 2 ? 4 : 2;
    // groups of warps that take the chunks in turn, four for the weights and X_WARPS for the activations each
    static constexpr int GROUPS = CG == 2 && NT == 128 ? 3 : 2;
    static constexpr int X_WARPS = X_ROWS / 32;
    static constexpr int W_WARPS_ALL = 4 * GROUPS, X_WARPS_ALL = X_WARPS * GROUPS;
    static constexpr int MMA_WARP = W_WARPS_ALL + X_WARPS_ALL, COPY_X_WARP = MMA_WARP + 1, COPY_W_WARP = MMA_WARP + 2;
    static constexpr int THREADS = (MMA_WARP + 3) * 32;
    static constexpr uint32_t A_COL = NT, Z_COL = NT + STAGES * HF_A_COLS;
    static constexpr int Z_OFF = STAGES * X_BYTES;
    static constexpr int RAW_OFF = Z_OFF + 2 * Z_BYTES;
    static constexpr int W_OFF = RAW_OFF + RAW_SLOTS * RAW_BYTES;
    static constexpr int BAR_OFF = W_OFF + W_SLOTS * HF_W_SLOT_BYTES;
    static constexpr int SMEM_BYTES = BAR_OFF + 256;
    static constexpr int BLOCKS = NT / 32 / (HF_EPI_WARPS / 4);  // 32 x 32 output blocks per warp
    static_assert(W_WARPS_ALL + X_WARPS_ALL >= HF_EPI_WARPS, "too few warps for the epilogue");
    static_assert(Z_COL + 2 * HF_Z_COLS <= HF_TMEM_COLS, "tensor memory too small");
    static_assert(SMEM_BYTES <= 227 * 1024, "rings do not fit in shared memory");
    static_assert(X_BOX % 1024 == 0 && RAW_OFF % 128 == 0 && RAW_BYTES % 128 == 0 && W_OFF % 128 == 0, "boxes start on whole patterns");
    static_assert(HF_EPI_WARPS * BLOCKS * 4096 <= BAR_OFF, "partial tiles do not fit in shared memory");
};

// fp16 constants, two per word
constexpr uint32_t H2_MAGIC_BYTES = 0x64646464u;  // high byte of 1024 + v for an 8-bit v
constexpr uint32_t H2_1032 = 0x64086408u;
constexpr uint32_t H2_1152 = 0x64806480u;
constexpr uint32_t H2_SIXTEENTH = 0x2C002C00u;
constexpr uint32_t H2_MINUS_72 = 0xD480D480u;

// D(fp32, TMEM) (+)= A(fp16, TMEM: lane = row, two values of K per column) x B(fp16 tile in shared memory)^T, K = 16
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}

// ---- the same for a pair of CTAs: A's 256 rows are 128 in each CTA, B's rows half in each, at the same addresses -------------
__device__ __forceinline__ void tc_mma_f16_ts_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
// completion of this thread's tensor-core operations arrives on the barrier at this offset in both CTAs (`first`: the cluster
// rank of the pair's first CTA)
__device__ __forceinline__ void tc_commit_pair(uint64_t *bar, int first) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)(3 << first))
                 : "memory");
}
// arrive on the barrier at this offset in the pair's first CTA (which issues the MMAs)
__device__ __forceinline__ void mbar_arrive_leader(uint64_t *bar, int first) {
    asm volatile(
        "{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %0, %1;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [remote];\n\t}" ::"r"(smem_u32(bar)), "r"(first)
        : "memory");
}
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint64_t *bar, uint32_t parity, int *fault, uint32_t limit = (1u << 22)) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    report_fault(fault, 1);
    return false;
}

__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }

// (v - offset) * scale: the subtraction is exact, the product is rounded once
__device__ __forceinline__ uint32_t h2_sub_scale(uint32_t v, uint32_t offset, __half2 scale) {
    return as_u32(__hmul2(__hsub2(as_h2(v), as_h2(offset)), scale));
}
// (v / 16 - 72) * scale for v = 1024 + 16 * q: the fma is exact (q - 8), the product is rounded once
__device__ __forceinline__ uint32_t h2_high_scale(uint32_t v, __half2 scale) {
    return as_u32(__hmul2(__hfma2(as_h2(v), as_h2(H2_SIXTEENTH), as_h2(H2_MINUS_72)), scale));
}

template <int MATS>
struct HfMaps {
    CUtensorMap w[MATS];
    CUtensorMap x;
};

// The kernel has an instance for one matrix and one for up to four, and takes these by value: a look-up by matrix needs
// them addressable (__grid_constant__), and then fields are read again in every turn of the conversion loop.
template <int MATS>
struct HfParams {
    // Up to four weight matrices that share K and the activations: the CTAs with blockIdx.x in [tile_begin[i],
    // tile_begin[i + 1]) have 128 rows each of matrix i (whole pairs of CTAs, if they work in pairs), which goes to y[i],
    // an [M][rows[i]] array.
    float *y[MATS];
    int64_t rows[MATS];
    int tile_begin[MATS + 1];
    int n_mats;
    int *fault;
#ifdef JQ_BOUNDS_CHECK
    Extent ext_y[MATS];  // range-checked debug build (the operand loads are tensor copies: their maps bound them)
#endif
    int64_t M;
    int n_chunks;        // K / 128
    int order;
    // Split K (few output tiles): the CTAs of a tile, blockIdx.z of k_splits, are a cluster and take the chunks
    // [z * chunks_per_split, ...) each; their partial tiles meet in shared memory.
    int k_splits, chunks_per_split;
    int static_weights;  // the weight copies may start before the previous kernel in the stream has finished
};

__device__ __forceinline__ void sts_v2(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st2_nowait(uint32_t taddr, uint32_t a, uint32_t b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st4_nowait(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Two blocks (64 values of K) of one weight row -> 32 words (q4 - 8) * d4: (values, of word t) 4t, 4t + 2 | 4t + 16, 4t + 18 |
// 4t + 1, 4t + 3 | 4t + 17, 4t + 19, as the nibbles come out of the word without moving bytes.
__device__ __forceinline__ void convert_two_blocks(const uint32_t (&ww)[18], int jj, uint32_t (&o)[32], uint32_t *dpair) {
    constexpr uint32_t LOW = 0x000F000Fu, HIGH = 0x00F000F0u, MAGIC = 0x64006400u;
    uint32_t db[2];
#pragma unroll
    for (int j2 = 0; j2 < 2; ++j2) {
        uint32_t q[4];
        q4_chunk_block(ww, 2 * jj + j2, q, &db[j2]);
        const __half2 d2 = as_h2(db[j2] | (db[j2] << 16));
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t u = q[t] >> 8;
            o[16 * j2 + 4 * t] = h2_sub_scale((q[t] & LOW) | MAGIC, H2_1032, d2);
            o[16 * j2 + 4 * t + 1] = h2_high_scale((q[t] & HIGH) | MAGIC, d2);
            o[16 * j2 + 4 * t + 2] = h2_sub_scale((u & LOW) | MAGIC, H2_1032, d2);
            o[16 * j2 + 4 * t + 3] = h2_high_scale((u & HIGH) | MAGIC, d2);
        }
    }
    *dpair = db[0] | (db[1] << 16);
}

// One block of an activation column -> four chunks of eight scaled fp16 values in the weights' order, each 16 bytes of the
// column's row in the swizzled tile; returns s8 - d8 * sum(q8) (d8 * the sum is exact in fp32).  `at`: the row's address with its
// number modulo 8 in the chunk bits.
__device__ __forceinline__ float convert_activation_block(const uint4 &lo, const uint4 &hi, uint32_t ds, uint32_t at, int chunk0) {
    const uint32_t dbits = ds & 0xFFFFu;
    const __half2 d2 = as_h2(dbits | (dbits << 16));
    const uint32_t w0[4] = {lo.x, lo.y, lo.z, lo.w}, w4[4] = {hi.x, hi.y, hi.z, hi.w};
    int isum = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        isum = __dp4a((int)w4[t], 0x01010101, __dp4a((int)w0[t], 0x01010101, isum));
        const uint32_t u0 = w0[t] ^ 0x80808080u, u4 = w4[t] ^ 0x80808080u;  // q + 128 in 1..255
        sts_v4(at ^ (uint32_t)((chunk0 + t) << 4),
               make_uint4(h2_sub_scale(__byte_perm(u0, H2_MAGIC_BYTES, 0x4240), H2_1152, d2), h2_sub_scale(__byte_perm(u4, H2_MAGIC_BYTES, 0x4240), H2_1152, d2),
                          h2_sub_scale(__byte_perm(u0, H2_MAGIC_BYTES, 0x4341), H2_1152, d2), h2_sub_scale(__byte_perm(u4, H2_MAGIC_BYTES, 0x4341), H2_1152, d2)));
    }
    return fmaf(-half_bits_to_float(dbits), (float)isum, half_bits_to_float(ds >> 16));
}

// the matrix this CTA works on
template <int MATS>
__device__ __forceinline__ int hf_matrix(const HfParams<MATS> &p) {
    int mat = 0;
    if (MATS > 1) {
        while (mat + 1 < p.n_mats && (int)blockIdx.x >= p.tile_begin[mat + 1]) ++mat;
    }
    return mat;
}

template <int CG, int NT, bool SPLIT, int MATS>
__global__ void __launch_bounds__((HfTile<CG, NT>::THREADS), 1)
gemm_q4_0_q8_1_f16_kernel(const HfParams<MATS> p, const __grid_constant__ HfMaps<MATS> maps) {
    using T = HfTile<CG, NT>;
    constexpr bool PAIR = CG == 2;
    constexpr int NS = T::STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + T::BAR_OFF);
    uint64_t *stage_full = bars;            // [NS] converted: weights in tensor memory, activations in shared memory
    uint64_t *stage_empty = bars + NS;      // [NS] the stage's MMAs are done: it may be filled again
    uint64_t *x_full = bars + 2 * NS;       // [RAW_SLOTS] raw activations have landed
    uint64_t *x_empty = x_full + T::RAW_SLOTS;
    uint64_t *w_full = x_empty + T::RAW_SLOTS;  // [W_SLOTS] raw weights have landed
    uint64_t *w_empty = w_full + T::W_SLOTS;
    uint64_t *acc_full = w_empty + T::W_SLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    static_assert((2 * NS + 2 * T::RAW_SLOTS + 2 * T::W_SLOTS + 1) * 8 + 4 <= 256, "barrier block too small");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = PAIR ? (int)(blockIdx.x & 1u) : 0;
    const int first = SPLIT && PAIR ? 2 * (int)blockIdx.z : 0;  // cluster rank of the pair's first CTA
    const int mat = hf_matrix(p);
    const int64_t n0 = (int64_t)((int)blockIdx.x - (MATS > 1 ? p.tile_begin[mat] : 0)) * HF_ROWS;  // this CTA's weight rows
    const int64_t m0 = (int64_t)blockIdx.y * NT;  // the tile's activation columns; this CTA converts X_ROWS from m0 + rank * X_ROWS
    const int c0 = SPLIT ? (int)blockIdx.z * p.chunks_per_split : 0;
    const int n_chunks = SPLIT ? min(p.chunks_per_split, p.n_chunks - c0) : p.n_chunks;  // even

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&stage_full[s], (4 + T::X_WARPS) * CG);
            mbar_init(&stage_empty[s], 1);
        }
        for (int i = 0; i < T::RAW_SLOTS; ++i) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], T::X_WARPS);
        }
        for (int i = 0; i < T::W_SLOTS; ++i) {
            mbar_init(&w_full[i], 1);
            mbar_init(&w_empty[i], 8);  // four warps for each of two chunks
        }
        mbar_init(acc_full, 1);
        fence_mbar_init();
    }
    if (warp == T::MMA_WARP) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(HF_TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(HF_TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();  // both CTAs' barriers are set up before the other arrives on them
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
    // Programmatic dependent launch: everything above ran while the previous kernel (the activation quantizer, as a
    // rule) was still finishing; the activations are read, and the outputs written, only after it has.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    bool finished = false;  // this epilogue warp has seen the tile complete

    if (warp < T::MMA_WARP) {
        bool alive = true;
        if (warp < T::W_WARPS_ALL) {
            // =============================== weights -> tensor memory =========================
            const int gw = warp & 3;
            const uint32_t lanes = tmem + ((uint32_t)(gw * 32) << 16);
#pragma unroll 1
            for (int c = warp >> 2; c < n_chunks; c += T::GROUPS) {
                const int s = c % NS, ws = (c >> 1) % T::W_SLOTS;
                const uint32_t round = (uint32_t)(c / NS);
                alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&w_full[ws], (uint32_t)((c >> 1) / T::W_SLOTS) & 1u, p.fault)) != 0;
                if (!alive) break;
                uint32_t ww[18];
                load_q4_chunk(ww, sbase + T::W_OFF + ws * HF_W_SLOT_BYTES + (uint32_t)((gw * 32 + lane) * Q8_BYTES), (c & 1) != 0);
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_empty[ws]);
                uint32_t o[32], z0, z1;
                convert_two_blocks(ww, 0, o, &z0);
                if (round > 0) {
                    alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&stage_empty[s], (round - 1) & 1u, p.fault)) != 0;
                    if (!alive) break;
                }
                tc_fence_after();
                const uint32_t a = lanes + T::A_COL + (uint32_t)s * HF_A_COLS;
                tmem_st32_nowait(a, o);
                convert_two_blocks(ww, 1, o, &z1);
                tmem_st32_nowait(a + 32, o);
                // -8 * d4 as fp16 (exact: a power of two; finite unless |d4| > 8188); columns without a chunk stay zero
                const __half2 m8 = __float2half2_rn(-8.0f);
                const uint32_t zt = lanes + T::Z_COL + (uint32_t)((c >> 2) & 1) * HF_Z_COLS;
                tmem_st2_nowait(zt + 2 * (c & 3), as_u32(__hmul2(as_h2(z0), m8)), as_u32(__hmul2(as_h2(z1), m8)));
                if (c == n_chunks - 1 && (c & 3) == 1) tmem_st4_nowait(zt + 4, 0u, 0u, 0u, 0u);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR)
                        mbar_arrive_leader(&stage_full[s], first);
                    else
                        mbar_arrive(&stage_full[s]);
                }
            }
        } else {
            // =============================== activations -> shared memory =====================
            const int xw = warp - T::W_WARPS_ALL;
            const int row = (xw % T::X_WARPS) * 32 + lane;
#pragma unroll 1
            for (int c = xw / T::X_WARPS; c < n_chunks; c += T::GROUPS) {
                const int s = c % NS, rs = c % T::RAW_SLOTS;
                const uint32_t round = (uint32_t)(c / NS);
                alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&x_full[rs], (uint32_t)(c / T::RAW_SLOTS) & 1u, p.fault)) != 0;
                if (!alive) break;
                uint4 v[9];
                const uint32_t raw = sbase + T::RAW_OFF + rs * T::RAW_BYTES + (uint32_t)(row * Q8_BYTES);
#pragma unroll
                for (int i = 0; i < 9; ++i) v[i] = lds_v4(raw + 16 * i);
                __syncwarp();
                if (lane == 0) mbar_arrive(&x_empty[rs]);
                if (round > 0) {
                    alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&stage_empty[s], (round - 1) & 1u, p.fault)) != 0;
                    if (!alive) break;
                }
                const uint32_t at = sbase + s * T::X_BYTES + (uint32_t)(row * 128 + ((row & 7) << 4));
                const float r0 = convert_activation_block(v[1], v[2], v[0].x, at, 0);
                const float r1 = convert_activation_block(v[3], v[4], v[0].y, at, 4);
                const float r2 = convert_activation_block(v[5], v[6], v[0].z, at + T::X_BOX, 0);
                const float r3 = convert_activation_block(v[7], v[8], v[0].w, at + T::X_BOX, 4);
                // the rank-one operand: sixteen residues per column, four of each chunk; those without a chunk stay zero
                const uint32_t zx = sbase + T::Z_OFF + ((c >> 2) & 1) * T::Z_BYTES + tile_off(row, 0);
                sts_v2(zx + ((c & 2) >> 1) * TC_LBO + (c & 1) * 8, as_u32(__floats2half2_rn(r0, r1)), as_u32(__floats2half2_rn(r2, r3)));
                if (c == n_chunks - 1 && (c & 3) == 1) sts_v4(zx + TC_LBO, make_uint4(0u, 0u, 0u, 0u));
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // tiles are read by the tensor core
                __syncwarp();
                if (lane == 0) {
                    if (PAIR)
                        mbar_arrive_leader(&stage_full[s], first);
                    else
                        mbar_arrive(&stage_full[s]);
                }
            }
        }

        // epilogue: a lane is a weight row, a column an activation column: 128 contiguous bytes of an output row per store
        if (warp < HF_EPI_WARPS && alive && __all_sync(0xFFFFFFFFu, mbar_wait_bounded(acc_full, 0u, p.fault))) {
            const int gw = warp & 3;
            const uint32_t lanes = tmem + ((uint32_t)(gw * 32) << 16);
            tc_fence_after();
            asm volatile("griddepcontrol.wait;" ::: "memory");  // (long past: orders the stores to y after the previous kernel)
            finished = true;
            const int out = hf_matrix(p);
            float *const y = p.y[out];
            const int64_t N = p.rows[out], n = n0 + gw * 32 + lane;
#pragma unroll
            for (int blk = 0; blk < T::BLOCKS; ++blk) {
                const int col = ((warp >> 2) * T::BLOCKS + blk) * 32;
                uint32_t v[32];
                tmem_ld32_nowait(lanes + (uint32_t)col, v);
                tmem_ld_wait();
                if (SPLIT) {
                    const uint32_t part = sbase + (uint32_t)((warp * T::BLOCKS + blk) * 4096 + lane * 4);
#pragma unroll
                    for (int j = 0; j < 32; ++j) sts_f32(part + j * 128, __uint_as_float(v[j]));
                } else {
                    float *at = y + (m0 + col) * N + n;
#pragma unroll
                    for (int j = 0; j < 32; ++j, at += N) {
                        if (m0 + col + j < p.M && n < N && JQ_IN_EXTENT(p.ext_y[out], at, sizeof(float), p.fault)) *at = __uint_as_float(v[j]);
                    }
                }
            }
        }
    } else if (warp == T::COPY_X_WARP) {
        // =============================== raw activations ======================================
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const int64_t col = m0 + rank * T::X_ROWS;
            for (int c = 0; c < n_chunks; ++c) {
                const int rs = c % T::RAW_SLOTS;
                const uint32_t round = (uint32_t)(c / T::RAW_SLOTS);
                if (round > 0 && !mbar_wait_bounded(&x_empty[rs], (round - 1) & 1u, p.fault)) break;
                mbar_arrive_expect_tx(&x_full[rs], T::RAW_BYTES);
                const uint32_t dst = sbase + T::RAW_OFF + rs * T::RAW_BYTES;
                if (p.order == JQ_ORDER_KSUPER_COL)  // the tensor is [n_super * M blocks][144 bytes]
                    tma_load_2d(dst, &maps.x, 0, (int)((int64_t)(c0 + c) * p.M + col), &x_full[rs]);
                else                                 // the tensor is [M columns][n_super * 144 bytes]
                    tma_load_2d(dst, &maps.x, (c0 + c) * Q8_BYTES, (int)col, &x_full[rs]);
            }
        }
    } else if (warp == T::COPY_W_WARP) {
        // =============================== raw weights ==========================================
        if (lane == 0) {
            if (!p.static_weights) asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int pr = 0; pr < n_chunks / 2; ++pr) {
                const int ws = pr % T::W_SLOTS;
                const uint32_t round = (uint32_t)(pr / T::W_SLOTS);
                if (round > 0 && !mbar_wait_bounded(&w_empty[ws], (round - 1) & 1u, p.fault)) break;
                mbar_arrive_expect_tx(&w_full[ws], HF_W_SLOT_BYTES);
                tma_load_2d(sbase + T::W_OFF + ws * HF_W_SLOT_BYTES, &maps.w[mat], ((c0 >> 1) + pr) * Q8_BYTES, (int)n0, &w_full[ws]);
            }
        }
    } else if (lane == 0 && rank == 0) {
        // =============================== MMA issuer (of a pair: the first CTA's, for both) =====
        const uint32_t idesc = tc_idesc_f16(CG * HF_ROWS, NT);
        bool alive = true;
        for (int c = 0; c < n_chunks; ++c) {
            const int s = c % NS;
            const uint32_t parity = (uint32_t)(c / NS) & 1u;
            if (!(PAIR ? mbar_wait_bounded_cluster(&stage_full[s], parity, p.fault) : mbar_wait_bounded(&stage_full[s], parity, p.fault))) {
                alive = false;
                break;
            }
            tc_fence_after();
            const uint32_t a = tmem + T::A_COL + (uint32_t)s * HF_A_COLS, x = sbase + s * T::X_BYTES;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const uint64_t db = tc_desc_sw128(x + (t >> 2) * T::X_BOX + (t & 3) * 32);
                const uint32_t more = c > 0 || t > 0 ? 1u : 0u;
                if (PAIR)
                    tc_mma_f16_ts_pair(tmem, a + t * 8, db, idesc, more);
                else
                    tc_mma_f16_ts(tmem, a + t * 8, db, idesc, more);
            }
            if ((c & 3) == 3 || c == n_chunks - 1) {  // the rank-one terms of sixteen blocks
                const uint32_t z = (uint32_t)((c >> 2) & 1);
                const uint64_t db = tc_desc(sbase + T::Z_OFF + z * T::Z_BYTES);
                if (PAIR)
                    tc_mma_f16_ts_pair(tmem, tmem + T::Z_COL + z * HF_Z_COLS, db, idesc, 1u);
                else
                    tc_mma_f16_ts(tmem, tmem + T::Z_COL + z * HF_Z_COLS, db, idesc, 1u);
            }
            // the stage may be overwritten once these MMAs have read it
            if (PAIR)
                tc_commit_pair(&stage_empty[s], first);
            else
                tc_commit(&stage_empty[s]);
        }
        if (alive) {
            if (PAIR)
                tc_commit_pair(acc_full, first);
            else
                tc_commit(acc_full);
        }
    }

    if (SPLIT) {
        // The parts of K: every CTA of the cluster has its partial tile in shared memory and adds up its share of the columns
        // over all parts, in the order of z (the same bits every time).
        const int parts = p.k_splits, z = (int)blockIdx.z;
        cluster_sync();
        if (finished) {
            const int gw = warp & 3;
            const int out = hf_matrix(p);
            float *const y = p.y[out];
            const int64_t N = p.rows[out], n = n0 + gw * 32 + lane;
            const int end = 32 * (z + 1) / parts;
#pragma unroll
            for (int blk = 0; blk < T::BLOCKS; ++blk) {
                const uint32_t part0 = sbase + (uint32_t)((warp * T::BLOCKS + blk) * 4096 + lane * 4);
#pragma unroll 1
                for (int j0 = 32 * z / parts; j0 < end; j0 += 4) {
                    float part[4][HF_MAX_SPLITS];
#pragma unroll
                    for (int q = 0; q < HF_MAX_SPLITS; ++q) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            part[u][q] = 0.0f;
                            if (q < parts && j0 + u < end) part[u][q] = lds_f32_of(part0 + (j0 + u) * 128, CG * q + rank);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float v = part[u][0];
#pragma unroll
                        for (int q = 1; q < HF_MAX_SPLITS; ++q) v += part[u][q];
                        const int64_t m = m0 + ((warp >> 2) * T::BLOCKS + blk) * 32 + j0 + u;
                        if (j0 + u < end && m < p.M && n < N && JQ_IN_EXTENT(p.ext_y[out], y + m * N + n, sizeof(float), p.fault)) y[m * N + n] = v;
                    }
                }
            }
        }
        cluster_sync();  // nobody leaves while another still reads its part
    }

    // common exit: nobody touches tensor memory any more, release it
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync();  // nor does the other CTA, which may still arrive on this one's barriers until here
    if (warp == T::MMA_WARP) {
        __syncwarp();
        if (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(HF_TMEM_COLS) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(HF_TMEM_COLS) : "memory");
    }
}

template <int CG, int NT, bool SPLIT, int MATS>
int launch_kernel(cudaStream_t st, dim3 grid, const HfParams<MATS> &p, const HfMaps<MATS> &maps) {
    using T = HfTile<CG, NT>;
    const auto kernel = gemm_q4_0_q8_1_f16_kernel<CG, NT, SPLIT, MATS>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), T::SMEM_BYTES)) return rc;
    (void)cudaGetLastError();  // a stale error of an earlier, unrelated call must not be taken for this launch's
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(T::THREADS);
    cfg.dynamicSmemBytes = T::SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CG;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)p.k_splits;
    cfg.attrs = attr;
    cfg.numAttrs = CG > 1 || SPLIT ? 2 : 1;
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, maps));
    return JQ_OK;
}
// Clusters of CG CTAs by z along K of this kernel that the current device runs at a time (0: none).  The instances for several
// matrices have the same threads and shared memory.  `answered` is cleared when the query failed for another reason than the size
// of the cluster.
template <int CG, int NT, bool SPLIT>
int clusters_at_a_time(unsigned z, int *out, bool *answered) {
    using T = HfTile<CG, NT>;
    const auto kernel = gemm_q4_0_q8_1_f16_kernel<CG, NT, SPLIT, 1>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), T::SMEM_BYTES)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CG, 1, z);
    cfg.blockDim = dim3(T::THREADS);
    cfg.dynamicSmemBytes = T::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CG;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = z;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(out, kernel, &cfg);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        *out = 0;
        if (e != cudaErrorInvalidClusterSize && e != cudaErrorInvalidConfiguration) *answered = false;
    }
    return JQ_OK;
}
// ... for every form, asked once per device that answers
int form_widths(const DeviceCaps &caps, GemmF16Widths *out) {
    struct Entry {
        int dev;
        GemmF16Widths width;
    };
    static std::vector<Entry> table;
    static std::mutex table_mutex;
    int dev = 0;
    JQ_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(table_mutex);
    for (const Entry &e : table) {
        if (e.dev == dev) {
            *out = e.width;
            return JQ_OK;
        }
    }
    GemmF16Widths w{};
    w.splits[1] = caps.sm_count;
    bool answered = true;
    for (int s = 2; s <= HF_MAX_SPLITS; ++s)
        if (int rc = clusters_at_a_time<1, 128, true>((unsigned)s, &w.splits[s], &answered)) return rc;
    if (int rc = clusters_at_a_time<2, 256, false>(1, &w.pairs, &answered)) return rc;
    if (int rc = clusters_at_a_time<2, 128, false>(1, &w.narrow[1], &answered)) return rc;
    for (int s = 2; s <= HF_MAX_NARROW_SPLITS; ++s)
        if (int rc = clusters_at_a_time<2, 128, true>((unsigned)s, &w.narrow[s], &answered)) return rc;
    if (answered) table.push_back(Entry{dev, w});
    *out = w;
    return JQ_OK;
}
template <int MATS>
int launch_form(cudaStream_t st, int cg, int nt, dim3 grid, const HfParams<MATS> &p, const HfMaps<MATS> &maps) {
    const bool split = p.k_splits > 1;
    if (cg == 1) return split ? launch_kernel<1, 128, true, MATS>(st, grid, p, maps) : launch_kernel<1, 128, false, MATS>(st, grid, p, maps);
    if (nt == 128) return split ? launch_kernel<2, 128, true, MATS>(st, grid, p, maps) : launch_kernel<2, 128, false, MATS>(st, grid, p, maps);
    return launch_kernel<2, 256, false, MATS>(st, grid, p, maps);
}

}  // namespace

int launch_gemm_f16(cudaStream_t st, const void *d_w, const void *d_xq, float *d_y, int64_t K, int64_t N, int64_t M,
                    int order, const MultiMat *multi) {
    // a weight row's pitch, K / 32 * 18 bytes, must be a multiple of 16 for the tensor copies
    if (K % (2 * SUPER) != 0) return set_error(JQ_ERR_UNSUPPORTED, "fp16-operand tcgen05 GEMM needs K %% 256 == 0 (K = %lld)", (long long)K);
    const void *w[HF_MAX_MATS] = {};
    HfParams<HF_MAX_MATS> p{};
    p.n_mats = multi != nullptr ? multi->n : 1;
    if (p.n_mats < 1 || p.n_mats > HF_MAX_MATS) return set_error(JQ_ERR_INVALID_ARG, "1 to %d weight matrices per launch", HF_MAX_MATS);
    uintptr_t bits = (uintptr_t)d_xq;
    int64_t gx = 0, pair_gx = 0;  // CTAs along the weight rows, on their own and in pairs
    for (int i = 0; i < p.n_mats; ++i) {
        w[i] = multi != nullptr ? multi->w[i] : d_w;
        p.y[i] = multi != nullptr ? multi->y[i] : d_y;
        p.rows[i] = multi != nullptr ? multi->rows[i] : N;
        bits |= (uintptr_t)w[i];
        gx += (p.rows[i] + HF_ROWS - 1) / HF_ROWS;
        pair_gx += (p.rows[i] + 2 * HF_ROWS - 1) / (2 * HF_ROWS) * 2;
    }
    if ((bits & 15u) != 0) return set_error(JQ_ERR_UNSUPPORTED, "fp16-operand tcgen05 GEMM needs 16-byte aligned operands");
    if (N == 0 || M == 0) return JQ_OK;
    DeviceCaps caps;
    if (int rc = device_caps(&caps)) return rc;
    if (caps.cc / 10 != 10) return set_error(JQ_ERR_UNSUPPORTED, "tcgen05 needs an sm_100-class device");
    const int64_t gy = (M + 127) / 128, pair_gy = (M + 255) / 256;
    if (gy > 65535 || K > (1 << 24) || (K / SUPER) * M >= ((int64_t)1 << 31) || N >= ((int64_t)1 << 31))
        return set_error(JQ_ERR_UNSUPPORTED, "shape too large for the tcgen05 GEMM");
    p.fault = device_fault_ptr();
    p.M = M;
    p.n_chunks = (int)(K / SUPER);
    p.order = order;
    p.static_weights = option_value(JQ_OPT_STATIC_WEIGHTS) != 0 ? 1 : 0;
    GemmF16Widths width;
    if (int rc = form_widths(caps, &width)) return rc;
    const GemmF16Plan plan = plan_gemm_f16(p.n_chunks, gx * gy, pair_gx / 2 * pair_gy, width, pair_gx / 2 * gy);
    int cg = plan.pair || plan.narrow ? 2 : 1, nt = plan.pair ? 256 : 128;
    p.k_splits = plan.k_splits;
    p.chunks_per_split = plan.chunks_per_split;
#ifdef HF_FORCE
    if (const char *f = getenv("HF_FORM")) {
        sscanf(f, "%d,%d,%d", &cg, &nt, &p.k_splits);
        p.chunks_per_split = ((p.n_chunks + p.k_splits - 1) / p.k_splits + 1) / 2 * 2;
        if ((p.n_chunks + p.chunks_per_split - 1) / p.chunks_per_split != p.k_splits) return set_error(JQ_ERR_UNSUPPORTED, "no such split");
    }
#endif
    const uint32_t row_bytes = (uint32_t)(K / QK * Q4_BYTES);
    HfMaps<HF_MAX_MATS> maps{};
    p.tile_begin[0] = 0;
    for (int i = 0; i < p.n_mats; ++i) {
        p.tile_begin[i + 1] = p.tile_begin[i] + (int)((p.rows[i] + cg * HF_ROWS - 1) / (cg * HF_ROWS) * cg);
        if (int rc = encode_byte_map(&maps.w[i], w[i], row_bytes, (uint64_t)p.rows[i], row_bytes, Q8_BYTES, HF_ROWS)) return rc;
#ifdef JQ_BOUNDS_CHECK
        p.ext_y[i] = make_extent(p.y[i], (unsigned long long)M * (unsigned long long)p.rows[i] * sizeof(float));
#endif
    }
    const int64_t n_super = K / SUPER;
    const uint64_t x_row = (uint64_t)n_super * Q8_BYTES;
    const uint32_t x_rows = (uint32_t)(nt / cg);
    if (int rc = order == JQ_ORDER_KSUPER_COL
                     ? encode_byte_map(&maps.x, d_xq, Q8_BYTES, (uint64_t)n_super * (uint64_t)M, Q8_BYTES, Q8_BYTES, x_rows)
                     : encode_byte_map(&maps.x, d_xq, x_row, (uint64_t)M, x_row, Q8_BYTES, x_rows))
        return rc;
    const dim3 grid((unsigned)p.tile_begin[p.n_mats], (unsigned)(nt == 256 ? pair_gy : gy), (unsigned)p.k_splits);
    if (p.n_mats > 1) return launch_form(st, cg, nt, grid, p, maps);
    HfParams<1> p1{};
    p1.y[0] = p.y[0];
    p1.rows[0] = p.rows[0];
    p1.n_mats = 1;
    p1.fault = p.fault;
#ifdef JQ_BOUNDS_CHECK
    p1.ext_y[0] = p.ext_y[0];
#endif
    p1.M = p.M;
    p1.n_chunks = p.n_chunks;
    p1.order = p.order;
    p1.k_splits = p.k_splits;
    p1.chunks_per_split = p.chunks_per_split;
    p1.static_weights = p.static_weights;
    HfMaps<1> maps1{};
    maps1.w[0] = maps.w[0];
    maps1.x = maps.x;
    return launch_form(st, cg, nt, grid, p1, maps1);
}

}  // namespace jq
