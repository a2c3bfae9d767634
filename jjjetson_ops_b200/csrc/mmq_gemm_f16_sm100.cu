// Prefill-regime multiply with the block scales folded into the operands: both matrices are
// dequantised to fp16 on their way to the tensor core and multiplied by tcgen05.mma.kind::f16 with
// fp32 accumulation in tensor memory, so nothing is drained or rescaled between blocks.
//
// Work to replace: q4_0_q8_1_mat_mul_kernel (reference src/cuda/mm_q4_0_q8_1.cu:164-289) for large
// batches.  The reference adds, per 32-wide block, d4 * (sumi * d8 - 8 * s8) (mm_q4_0_q8_1.cu:92).
// With sumi = sum(q4 * q8) that is
//     sum_i ((q4_i - 8) * d4) * (q8_i * d8)   +   (-8 * d4) * (s8 - d8 * sum_i q8_i)
// The first term is a plain product of two fp16 matrices A[n][k] = (q4 - 8) * d4 and
// B[m][k] = q8 * d8; the second is rank one per block and joins the same accumulator as one more
// MMA per 512 values of K (operands -8 * d4, exact, and s8 - d8 * sum(q8), computed in fp32).  It
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
// A CTA owns 128 weight rows x 128 activation columns of Y, or two CTAs on neighbouring SMs own 256 x 256: each converts 128 rows
// and 128 columns, and cta_group::2 MMAs, issued by the first, multiply all with all, so that a converted operand is used twice as
// often.  K advances in chunks of 128 values (one Q8_1 block per column, four Q4_0 blocks per row):
//   raw rings       the quantized bytes as they lie in global memory, brought in by the copy engine, one tiled tensor copy per chunk
//                   for the activation blocks and one per two chunks for 144 bytes of each weight row.  (A per-thread load of "its"
//                   row touches 32 cache lines per warp instruction.)  A slot is handed back as soon as its words are in registers.
//   operand stages  the weights are the MMA's A operand and lie in tensor memory, lane = weight row, 64 columns holding the 128
//                   values of a chunk; the activations are B, in shared memory with the 128-byte swizzle.  So the tile comes out
//                   with the weight rows in the lanes, and a register of the accumulator is 128 contiguous bytes of an output row:
//                   stored as it is, where activations in the lanes took a turn through shared memory.
//   order of K      inside a block of 32 both operands take the values in the order in which a word's nibbles come out under a mask
//                   (0, 2 | 16, 18 | 1, 3 | 17, 19 of each four): 13 instructions for eight weights, no bytes moved.
//   rank-one terms  those of four chunks are one MMA of K = 16.
// Warps: groups of four for the weights (a row per thread: nibbles become fp16 by the magic-number trick, 0x6400 | q is 1024 + q;
// then one exact subtraction and one rounded multiplication by the scale) and four for the activations (a column per thread, int8
// the same way) take the chunks in turn; one thread issues the MMAs, one copies activations, one weights.
// Every mbarrier wait is a bounded poll; a wait that runs out sets the device fault word, and every warp still reaches the common
// exit where tensor memory is released.
//
// What bounds it.  Per chunk of a 256 x 256 pair (K = 8192, N = 28672, M = 2048, with two groups: 1.0 us): the MMAs alone (everything
// else left out) 0.6, the conversion alone 0.8, the copies alone 0.8, the hand-overs between warps alone 0.33.  The multiply, before
// (activations in tensor memory, weights in shared memory, two groups) / now: 1010 / 890 us; K = 4096, N = 11008, M = 512 79.1 / 66.9 us;
// K = N = 4096, M = 512 27.7 / 26.2 us (35.2 / 29.6 us in another process: the card's clock), M = 128 13.1 / 12.4 us; K = 11008,
// N = 4096, M = 128 23.9 / 22.4 us.  Over 110 shapes 0.924 of the time, none slower.
// Dropped: pairs on 256 x 128 (each converts 64 columns), 0.25 % over those shapes; all of a chunk converted in registers before its
// stage is free, 1023 against 961 us; one lane polling for its warp, 982 us; polls that suspend the warp longer, or not at all, or
// with a pause in between, no better.
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

constexpr int HF_X_ROWS = 128;    // activation columns that a CTA converts
constexpr int HF_X_BOX = HF_X_ROWS * 128;           // bytes of 64 fp16 values of K
constexpr int HF_X_BYTES = 2 * HF_X_BOX;            // ... of a chunk
constexpr int HF_Z_BYTES = HF_X_ROWS * 32;          // fp16 residues of sixteen blocks
constexpr int HF_RAW_BYTES = HF_X_ROWS * Q8_BYTES;  // a chunk's activation blocks as they lie in global memory
constexpr int HF_STAGES = 3;      // chunks of converted operands: what tensor memory (256 columns of accumulator) and shared memory hold
constexpr int HF_RAW_SLOTS = 3, HF_W_SLOTS = 3;
// Groups of warps that take the chunks in turn, four for the weights and four for the activations each.  Three groups of 72 registers
// a thread, against two of 104: 877 / 928 us on 256 x 256 (K = 8192, N = 28672, M = 2048), 27.1 / 28.3 us on 128 x 128 (K = N = 4096,
// M = 512): a group waits for its barriers and its stores to tensor memory as long as it converts.
constexpr int HF_GROUPS = 3;
constexpr int HF_W_WARPS = 4 * HF_GROUPS, HF_X_WARPS = 4 * HF_GROUPS;
constexpr int HF_MMA_WARP = HF_W_WARPS + HF_X_WARPS, HF_COPY_X_WARP = HF_MMA_WARP + 1, HF_COPY_W_WARP = HF_MMA_WARP + 2;
constexpr int HF_THREADS = (HF_MMA_WARP + 3) * 32;
constexpr int HF_Z_OFF = HF_STAGES * HF_X_BYTES;
constexpr int HF_RAW_OFF = HF_Z_OFF + 2 * HF_Z_BYTES;
constexpr int HF_W_OFF = HF_RAW_OFF + HF_RAW_SLOTS * HF_RAW_BYTES;
constexpr int HF_BAR_OFF = HF_W_OFF + HF_W_SLOTS * HF_W_SLOT_BYTES;
constexpr int HF_SMEM_BYTES = HF_BAR_OFF + 256;
static_assert(HF_SMEM_BYTES <= 227 * 1024, "rings do not fit in shared memory");
static_assert(HF_X_BOX % 1024 == 0 && HF_RAW_OFF % 128 == 0 && HF_RAW_BYTES % 128 == 0 && HF_W_OFF % 128 == 0, "boxes start on whole patterns");
// A wait by parity is only right while the phase before the awaited one is known to be over.  A raw activation slot belongs to one
// group, which has waited for each of its phases; what a weight slot held before has been used by the MMAs of chunk
// c - HF_GROUPS - HF_STAGES or an earlier one, which are over when a group comes to chunk c.
static_assert(HF_RAW_SLOTS % HF_GROUPS == 0, "another group would use the slot in between");
static_assert(HF_GROUPS + HF_STAGES <= 2 * HF_W_SLOTS, "the slot's last contents may not have landed");

// A CTA on 128 weight rows x NT = 128 activation columns, or a pair (cta_group::2) on 256 x 256
template <bool PAIR>
struct HfTile {
    static constexpr int NT = PAIR ? 256 : 128;
    static constexpr uint32_t A_COL = NT, Z_COL = NT + HF_STAGES * HF_A_COLS;  // tensor memory: accumulator, weights, rank-one operands
    static constexpr int BLOCKS = NT / 32 / (HF_EPI_WARPS / 4);                // 32 x 32 output blocks per warp
    static_assert(Z_COL + 2 * HF_Z_COLS <= HF_TMEM_COLS, "tensor memory too small");
    static_assert(HF_EPI_WARPS * BLOCKS * 4096 <= HF_BAR_OFF, "partial tiles do not fit in shared memory");
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
// completion of this thread's tensor-core operations arrives on the barrier at this offset in both CTAs
__device__ __forceinline__ void tc_commit_pair(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
// arrive on the barrier at this offset in the pair's first CTA (which issues the MMAs)
__device__ __forceinline__ void mbar_arrive_leader(uint64_t *bar) {
    asm volatile(
        "{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %0, 0;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [remote];\n\t}" ::"r"(smem_u32(bar))
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

// The kernel has an instance for one matrix and one for up to four.  What is looked up by matrix is addressable (__grid_constant__:
// by value, such a look-up takes a copy in local memory, 128 bytes per thread of the instances for several matrices) ...
template <int MATS>
struct HfMats {
    // Up to four weight matrices that share K and the activations: the CTAs with blockIdx.x in [tile_begin[i],
    // tile_begin[i + 1]) have 128 rows each of matrix i (whole pairs of CTAs, if they work in pairs), which goes to y[i],
    // an [M][rows[i]] array.
    CUtensorMap w[MATS];
    CUtensorMap x;
    float *y[MATS];
    int64_t rows[MATS];
    int tile_begin[MATS + 1];
    int n_mats;
#ifdef JQ_BOUNDS_CHECK
    Extent ext_y[MATS];  // range-checked debug build (the operand loads are tensor copies: their maps bound them)
#endif
};

// ... and the rest is not: fields of an addressable parameter are read again in every turn of the conversion loop, and when they are
// needed (K = 256, N = 74, M = 809 4.19 us with the one matrix's output by value, 4.25 without).
struct HfParams {
    float *y0;      // where there is one matrix: y[0], rows[0]
    int64_t rows0;
    int *fault;
    int64_t M;
    int n_chunks;        // K / 128
    int order;
    // Split K (few output tiles): the CTAs of a tile, blockIdx.z of k_splits, are a cluster and take the chunks
    // [z * chunks_per_split, ...) each; their partial tiles meet in shared memory.
    int k_splits, chunks_per_split;
    int static_weights;  // the weight copies may start before the previous kernel in the stream has finished
    unsigned long long *trace;  // tracing aid (or nullptr): SM clock stamps of the first CTA, rows of 8
};
// TRACE: an instance of its own, so that the others have neither the test nor the registers
template <bool TRACE>
__device__ __forceinline__ void hf_stamp(const HfParams &p, int who, int c, int slot) {
    if (TRACE && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && c < 64) p.trace[(who * 64 + c) * 8 + slot] = (unsigned long long)clock64();
}

__device__ __forceinline__ void sts_v2(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st2_nowait(uint32_t taddr, uint32_t a, uint32_t b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(taddr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void tmem_st4_nowait(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// A weight row's 72 bytes of a 128-value chunk from a raw slot, where two chunks of 128 rows lie 144 bytes apart: four 16-byte
// words (conflict-free at that pitch) and one of 8, which comes last in an even chunk and first in an odd one.
__device__ __forceinline__ void load_q4_chunk(uint32_t (&ww)[18], uint32_t raw, bool odd) {
    if (!odd) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 v = lds_v4(raw + 16 * i);
            ww[4 * i] = v.x;
            ww[4 * i + 1] = v.y;
            ww[4 * i + 2] = v.z;
            ww[4 * i + 3] = v.w;
        }
        const uint2 e = lds_v2(raw + 64);
        ww[16] = e.x;
        ww[17] = e.y;
    } else {
        const uint2 e = lds_v2(raw + 72);
        ww[0] = e.x;
        ww[1] = e.y;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint4 v = lds_v4(raw + 80 + 16 * i);
            ww[2 + 4 * i] = v.x;
            ww[3 + 4 * i] = v.y;
            ww[4 + 4 * i] = v.z;
            ww[5 + 4 * i] = v.w;
        }
    }
}

// The sixteen quant bytes and the scale of block j of a 72-byte chunk
__device__ __forceinline__ void q4_chunk_block(const uint32_t (&ww)[18], int j, uint32_t (&q)[4], uint32_t *dbits) {
    if ((j & 1) == 0) {  // starts on a word boundary: [d | q0 q1] [q2..q5] ...
        const int w0 = (j / 2) * 9;
        *dbits = ww[w0] & 0xFFFFu;
#pragma unroll
        for (int t = 0; t < 4; ++t) q[t] = __funnelshift_r(ww[w0 + t], ww[w0 + t + 1], 16);
    } else {  // starts in the middle of a word
        const int w0 = (j / 2) * 9 + 4;
        *dbits = ww[w0] >> 16;
#pragma unroll
        for (int t = 0; t < 4; ++t) q[t] = ww[w0 + 1 + t];
    }
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
__device__ __forceinline__ int hf_matrix(const HfMats<MATS> &mats) {
    int mat = 0;
    if (MATS > 1) {
        while (mat + 1 < mats.n_mats && (int)blockIdx.x >= mats.tile_begin[mat + 1]) ++mat;
    }
    return mat;
}

template <bool PAIR, bool SPLIT, int MATS, bool TRACE = false>
__global__ void __launch_bounds__(HF_THREADS, 1)
gemm_q4_0_q8_1_f16_kernel(const HfParams p, const __grid_constant__ HfMats<MATS> mats) {
    using T = HfTile<PAIR>;
    constexpr int NS = HF_STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + HF_BAR_OFF);
    uint64_t *stage_full = bars;            // [NS] converted: weights in tensor memory, activations in shared memory
    uint64_t *stage_empty = bars + NS;      // [NS] the stage's MMAs are done: it may be filled again
    uint64_t *x_full = bars + 2 * NS;       // [RAW_SLOTS] raw activations have landed
    uint64_t *x_empty = x_full + HF_RAW_SLOTS;
    uint64_t *w_full = x_empty + HF_RAW_SLOTS;  // [W_SLOTS] raw weights have landed
    uint64_t *w_empty = w_full + HF_W_SLOTS;
    uint64_t *acc_full = w_empty + HF_W_SLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    static_assert((2 * NS + 2 * HF_RAW_SLOTS + 2 * HF_W_SLOTS + 1) * 8 + 4 <= 256, "barrier block too small");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = PAIR ? (int)(blockIdx.x & 1u) : 0;
    const int mat = hf_matrix(mats);
    const int64_t n0 = (int64_t)((int)blockIdx.x - (MATS > 1 ? mats.tile_begin[mat] : 0)) * HF_ROWS;  // this CTA's weight rows
    const int64_t m0 = (int64_t)blockIdx.y * T::NT;  // the tile's activation columns; this CTA converts X_ROWS from m0 + rank * X_ROWS
    const int c0 = SPLIT ? (int)blockIdx.z * p.chunks_per_split : 0;
    const int n_chunks = SPLIT ? min(p.chunks_per_split, p.n_chunks - c0) : p.n_chunks;  // even

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&stage_full[s], PAIR ? 16 : 8);  // four warps for each operand, of each CTA
            mbar_init(&stage_empty[s], 1);
        }
        for (int i = 0; i < HF_RAW_SLOTS; ++i) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], 4);
        }
        for (int i = 0; i < HF_W_SLOTS; ++i) {
            mbar_init(&w_full[i], 1);
            mbar_init(&w_empty[i], 8);  // four warps for each of two chunks
        }
        mbar_init(acc_full, 1);
        fence_mbar_init();
    }
    if (warp == HF_MMA_WARP) {
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

    if (warp < HF_MMA_WARP) {
        bool alive = true;
        if (warp < HF_W_WARPS) {
            // =============================== weights -> tensor memory =========================
            const int gw = warp & 3;
            const uint32_t lanes = tmem + ((uint32_t)(gw * 32) << 16);
#pragma unroll 1
            for (int c = warp >> 2; c < n_chunks; c += HF_GROUPS) {
                const int s = c % NS, ws = (c >> 1) % HF_W_SLOTS;
                const uint32_t round = (uint32_t)(c / NS);
                const bool stamps = TRACE && tid == 0;
                if (stamps) hf_stamp<TRACE>(p, 0, c, 0);
                alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&w_full[ws], (uint32_t)((c >> 1) / HF_W_SLOTS) & 1u, p.fault)) != 0;
                if (!alive) break;
                if (stamps) hf_stamp<TRACE>(p, 0, c, 1);
                uint32_t ww[18];
                load_q4_chunk(ww, sbase + HF_W_OFF + ws * HF_W_SLOT_BYTES + (uint32_t)((gw * 32 + lane) * Q8_BYTES), (c & 1) != 0);
                __syncwarp();
                if (lane == 0) mbar_arrive(&w_empty[ws]);
                uint32_t o[32], z0, z1;
                convert_two_blocks(ww, 0, o, &z0);
                if (round > 0) {
                    alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&stage_empty[s], (round - 1) & 1u, p.fault)) != 0;
                    if (!alive) break;
                }
                if (stamps) hf_stamp<TRACE>(p, 0, c, 3);
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
                if (stamps) hf_stamp<TRACE>(p, 0, c, 4);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (PAIR)
                        mbar_arrive_leader(&stage_full[s]);
                    else
                        mbar_arrive(&stage_full[s]);
                }
                if (stamps) hf_stamp<TRACE>(p, 0, c, 5);
            }
        } else {
            // =============================== activations -> shared memory =====================
            const int xw = warp - HF_W_WARPS;
            const int row = (xw & 3) * 32 + lane;
#pragma unroll 1
            for (int c = xw >> 2; c < n_chunks; c += HF_GROUPS) {
                const int s = c % NS, rs = c % HF_RAW_SLOTS;
                const uint32_t round = (uint32_t)(c / NS);
                const bool stamps = TRACE && tid == HF_W_WARPS * 32;
                if (stamps) hf_stamp<TRACE>(p, 1, c, 0);
                alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&x_full[rs], (uint32_t)(c / HF_RAW_SLOTS) & 1u, p.fault)) != 0;
                if (!alive) break;
                if (stamps) hf_stamp<TRACE>(p, 1, c, 1);
                uint4 v[9];
                const uint32_t raw = sbase + HF_RAW_OFF + rs * HF_RAW_BYTES + (uint32_t)(row * Q8_BYTES);
#pragma unroll
                for (int i = 0; i < 9; ++i) v[i] = lds_v4(raw + 16 * i);
                __syncwarp();
                if (lane == 0) mbar_arrive(&x_empty[rs]);
                if (round > 0) {
                    alive = __all_sync(0xFFFFFFFFu, mbar_wait_bounded(&stage_empty[s], (round - 1) & 1u, p.fault)) != 0;
                    if (!alive) break;
                }
                if (stamps) hf_stamp<TRACE>(p, 1, c, 3);
                const uint32_t at = sbase + s * HF_X_BYTES + (uint32_t)(row * 128 + ((row & 7) << 4));
                const float r0 = convert_activation_block(v[1], v[2], v[0].x, at, 0);
                const float r1 = convert_activation_block(v[3], v[4], v[0].y, at, 4);
                const float r2 = convert_activation_block(v[5], v[6], v[0].z, at + HF_X_BOX, 0);
                const float r3 = convert_activation_block(v[7], v[8], v[0].w, at + HF_X_BOX, 4);
                // the rank-one operand: sixteen residues per column, four of each chunk; those without a chunk stay zero
                const uint32_t zx = sbase + HF_Z_OFF + ((c >> 2) & 1) * HF_Z_BYTES + tile_off(row, 0);
                sts_v2(zx + ((c & 2) >> 1) * TC_LBO + (c & 1) * 8, as_u32(__floats2half2_rn(r0, r1)), as_u32(__floats2half2_rn(r2, r3)));
                if (c == n_chunks - 1 && (c & 3) == 1) sts_v4(zx + TC_LBO, make_uint4(0u, 0u, 0u, 0u));
                if (stamps) hf_stamp<TRACE>(p, 1, c, 4);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // tiles are read by the tensor core
                __syncwarp();
                if (lane == 0) {
                    if (PAIR)
                        mbar_arrive_leader(&stage_full[s]);
                    else
                        mbar_arrive(&stage_full[s]);
                }
                if (stamps) hf_stamp<TRACE>(p, 1, c, 5);
            }
        }

        // epilogue: a lane is a weight row, a column an activation column: 128 contiguous bytes of an output row per store
        if (warp < HF_EPI_WARPS && alive && __all_sync(0xFFFFFFFFu, mbar_wait_bounded(acc_full, 0u, p.fault))) {
            const int gw = warp & 3;
            const uint32_t lanes = tmem + ((uint32_t)(gw * 32) << 16);
            tc_fence_after();
            asm volatile("griddepcontrol.wait;" ::: "memory");  // (long past: orders the stores to y after the previous kernel)
            finished = true;
            const int out = hf_matrix(mats);
            float *const y = MATS == 1 ? p.y0 : mats.y[out];
            const int64_t N = MATS == 1 ? p.rows0 : mats.rows[out], n = n0 + gw * 32 + lane;
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
                        if (m0 + col + j < p.M && n < N && JQ_IN_EXTENT(mats.ext_y[out], at, sizeof(float), p.fault)) *at = __uint_as_float(v[j]);
                    }
                }
            }
        }
    } else if (warp == HF_COPY_X_WARP) {
        // =============================== raw activations ======================================
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            const int64_t col = m0 + rank * HF_X_ROWS;
            for (int c = 0; c < n_chunks; ++c) {
                const int rs = c % HF_RAW_SLOTS;
                const uint32_t round = (uint32_t)(c / HF_RAW_SLOTS);
                if (round > 0 && !mbar_wait_bounded(&x_empty[rs], (round - 1) & 1u, p.fault)) break;
                mbar_arrive_expect_tx(&x_full[rs], HF_RAW_BYTES);
                const uint32_t dst = sbase + HF_RAW_OFF + rs * HF_RAW_BYTES;
                if (p.order == JQ_ORDER_KSUPER_COL)  // the tensor is [n_super * M blocks][144 bytes]
                    tma_load_2d(dst, &mats.x, 0, (int)((int64_t)(c0 + c) * p.M + col), &x_full[rs]);
                else                                 // the tensor is [M columns][n_super * 144 bytes]
                    tma_load_2d(dst, &mats.x, (c0 + c) * Q8_BYTES, (int)col, &x_full[rs]);
            }
        }
    } else if (warp == HF_COPY_W_WARP) {
        // =============================== raw weights ==========================================
        if (lane == 0) {
            if (!p.static_weights) asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int pr = 0; pr < n_chunks / 2; ++pr) {
                const int ws = pr % HF_W_SLOTS;
                const uint32_t round = (uint32_t)(pr / HF_W_SLOTS);
                if (round > 0 && !mbar_wait_bounded(&w_empty[ws], (round - 1) & 1u, p.fault)) break;
                mbar_arrive_expect_tx(&w_full[ws], HF_W_SLOT_BYTES);
                tma_load_2d(sbase + HF_W_OFF + ws * HF_W_SLOT_BYTES, &mats.w[mat], ((c0 >> 1) + pr) * Q8_BYTES, (int)n0, &w_full[ws]);
            }
        }
    } else if (lane == 0 && rank == 0) {
        // =============================== MMA issuer (of a pair: the first CTA's, for both) =====
        const uint32_t idesc = tc_idesc_f16(PAIR ? 2 * HF_ROWS : HF_ROWS, T::NT);
        bool alive = true;
        for (int c = 0; c < n_chunks; ++c) {
            const int s = c % NS;
            const uint32_t parity = (uint32_t)(c / NS) & 1u;
            if (!(PAIR ? mbar_wait_bounded_cluster(&stage_full[s], parity, p.fault) : mbar_wait_bounded(&stage_full[s], parity, p.fault))) {
                alive = false;
                break;
            }
            hf_stamp<TRACE>(p, 2, c, 0);
            tc_fence_after();
            const uint32_t a = tmem + T::A_COL + (uint32_t)s * HF_A_COLS, x = sbase + s * HF_X_BYTES;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const uint64_t db = tc_desc_sw128(x + (t >> 2) * HF_X_BOX + (t & 3) * 32);
                const uint32_t more = c > 0 || t > 0 ? 1u : 0u;
                if (PAIR)
                    tc_mma_f16_ts_pair(tmem, a + t * 8, db, idesc, more);
                else
                    tc_mma_f16_ts(tmem, a + t * 8, db, idesc, more);
            }
            if ((c & 3) == 3 || c == n_chunks - 1) {  // the rank-one terms of sixteen blocks
                const uint32_t z = (uint32_t)((c >> 2) & 1);
                const uint64_t db = tc_desc(sbase + HF_Z_OFF + z * HF_Z_BYTES);
                if (PAIR)
                    tc_mma_f16_ts_pair(tmem, tmem + T::Z_COL + z * HF_Z_COLS, db, idesc, 1u);
                else
                    tc_mma_f16_ts(tmem, tmem + T::Z_COL + z * HF_Z_COLS, db, idesc, 1u);
            }
            // the stage may be overwritten once these MMAs have read it
            if (PAIR)
                tc_commit_pair(&stage_empty[s]);
            else
                tc_commit(&stage_empty[s]);
            hf_stamp<TRACE>(p, 2, c, 1);
        }
        if (alive) {
            if (PAIR)
                tc_commit_pair(acc_full);
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
            const int out = hf_matrix(mats);
            float *const y = MATS == 1 ? p.y0 : mats.y[out];
            const int64_t N = MATS == 1 ? p.rows0 : mats.rows[out], n = n0 + gw * 32 + lane;
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
                            if (q < parts && j0 + u < end) part[u][q] = lds_f32_of(part0 + (j0 + u) * 128, q);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        float v = part[u][0];
#pragma unroll
                        for (int q = 1; q < HF_MAX_SPLITS; ++q) v += part[u][q];
                        const int64_t m = m0 + ((warp >> 2) * T::BLOCKS + blk) * 32 + j0 + u;
                        if (j0 + u < end && m < p.M && n < N && JQ_IN_EXTENT(mats.ext_y[out], y + m * N + n, sizeof(float), p.fault)) y[m * N + n] = v;
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
    if (warp == HF_MMA_WARP) {
        __syncwarp();
        if (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(HF_TMEM_COLS) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(HF_TMEM_COLS) : "memory");
    }
}

template <bool PAIR, bool SPLIT, int MATS>
int launch_kernel(cudaStream_t st, dim3 grid, const HfParams &p, const HfMats<MATS> &mats) {
    const auto kernel = p.trace != nullptr ? gemm_q4_0_q8_1_f16_kernel<PAIR, SPLIT, MATS, true> : gemm_q4_0_q8_1_f16_kernel<PAIR, SPLIT, MATS>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), HF_SMEM_BYTES)) return rc;
    (void)cudaGetLastError();  // a stale error of an earlier, unrelated call must not be taken for this launch's
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(HF_THREADS);
    cfg.dynamicSmemBytes = HF_SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = PAIR ? 2 : 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)p.k_splits;
    cfg.attrs = attr;
    cfg.numAttrs = PAIR || SPLIT ? 2 : 1;
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, mats));
    return JQ_OK;
}
// Clusters of z CTAs along K, or of a pair of CTAs, of this kernel that the current device runs at a time (0: none).  The instances
// for several matrices have the same threads and shared memory.  `answered` is cleared when the query failed for another reason than
// the size of the cluster.
template <bool PAIR, bool SPLIT>
int clusters_at_a_time(unsigned z, int *out, bool *answered) {
    const auto kernel = gemm_q4_0_q8_1_f16_kernel<PAIR, SPLIT, 1>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), HF_SMEM_BYTES)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(PAIR ? 2 : 1, 1, z);
    cfg.blockDim = dim3(HF_THREADS);
    cfg.dynamicSmemBytes = HF_SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = PAIR ? 2 : 1;
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
        if (int rc = clusters_at_a_time<false, true>((unsigned)s, &w.splits[s], &answered)) return rc;
    if (int rc = clusters_at_a_time<true, false>(1, &w.pairs, &answered)) return rc;
    if (answered) table.push_back(Entry{dev, w});
    *out = w;
    return JQ_OK;
}
// form: 0 pairs of CTAs, 1 split K, 2 neither
template <int MATS>
int launch_form(cudaStream_t st, int form, dim3 grid, const HfParams &p, const HfMats<MATS> &mats) {
    if (form == 0) return launch_kernel<true, false, MATS>(st, grid, p, mats);
    if (form == 1) return launch_kernel<false, true, MATS>(st, grid, p, mats);
    return launch_kernel<false, false, MATS>(st, grid, p, mats);
}

}  // namespace

int launch_gemm_f16(cudaStream_t st, const void *d_w, const void *d_xq, float *d_y, int64_t K, int64_t N, int64_t M,
                    int order, const MultiMat *multi) {
    // a weight row's pitch, K / 32 * 18 bytes, must be a multiple of 16 for the tensor copies
    if (K % (2 * SUPER) != 0) return set_error(JQ_ERR_UNSUPPORTED, "fp16-operand tcgen05 GEMM needs K %% 256 == 0 (K = %lld)", (long long)K);
    const void *w[HF_MAX_MATS] = {};
    HfParams p{};
    HfMats<HF_MAX_MATS> mats{};
    mats.n_mats = multi != nullptr ? multi->n : 1;
    if (mats.n_mats < 1 || mats.n_mats > HF_MAX_MATS) return set_error(JQ_ERR_INVALID_ARG, "1 to %d weight matrices per launch", HF_MAX_MATS);
    uintptr_t bits = (uintptr_t)d_xq;
    int64_t gx = 0, pair_gx = 0;  // CTAs along the weight rows, on their own and in pairs
    for (int i = 0; i < mats.n_mats; ++i) {
        w[i] = multi != nullptr ? multi->w[i] : d_w;
        mats.y[i] = multi != nullptr ? multi->y[i] : d_y;
        mats.rows[i] = multi != nullptr ? multi->rows[i] : N;
        bits |= (uintptr_t)w[i];
        gx += (mats.rows[i] + HF_ROWS - 1) / HF_ROWS;
        pair_gx += (mats.rows[i] + 2 * HF_ROWS - 1) / (2 * HF_ROWS) * 2;
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
    p.trace = static_cast<unsigned long long *>(next_trace_slot());
    GemmF16Widths width;
    if (int rc = form_widths(caps, &width)) return rc;
    const GemmF16Plan plan = plan_gemm_f16(p.n_chunks, gx * gy, pair_gx / 2 * pair_gy, width);
    const bool pair = plan.pair;
    p.k_splits = plan.k_splits;
    p.chunks_per_split = plan.chunks_per_split;
    const uint32_t row_bytes = (uint32_t)(K / QK * Q4_BYTES);
    mats.tile_begin[0] = 0;
    for (int i = 0; i < mats.n_mats; ++i) {
        const int64_t per = pair ? 2 : 1;
        mats.tile_begin[i + 1] = mats.tile_begin[i] + (int)((mats.rows[i] + per * HF_ROWS - 1) / (per * HF_ROWS) * per);
        if (int rc = encode_byte_map(&mats.w[i], w[i], row_bytes, (uint64_t)mats.rows[i], row_bytes, Q8_BYTES, HF_ROWS)) return rc;
#ifdef JQ_BOUNDS_CHECK
        mats.ext_y[i] = make_extent(mats.y[i], (unsigned long long)M * (unsigned long long)mats.rows[i] * sizeof(float));
#endif
    }
    const int64_t n_super = K / SUPER;
    const uint64_t x_row = (uint64_t)n_super * Q8_BYTES;
    if (int rc = order == JQ_ORDER_KSUPER_COL
                     ? encode_byte_map(&mats.x, d_xq, Q8_BYTES, (uint64_t)n_super * (uint64_t)M, Q8_BYTES, Q8_BYTES, HF_X_ROWS)
                     : encode_byte_map(&mats.x, d_xq, x_row, (uint64_t)M, x_row, Q8_BYTES, HF_X_ROWS))
        return rc;
    const int form = pair ? 0 : p.k_splits > 1 ? 1 : 2;
    const dim3 grid((unsigned)mats.tile_begin[mats.n_mats], (unsigned)(pair ? pair_gy : gy), (unsigned)p.k_splits);
    if (mats.n_mats > 1) return launch_form(st, form, grid, p, mats);
    p.y0 = mats.y[0];
    p.rows0 = mats.rows[0];
    HfMats<1> one{};
    one.w[0] = mats.w[0];
    one.x = mats.x;
    one.y[0] = mats.y[0];
    one.rows[0] = mats.rows[0];
    one.n_mats = 1;
#ifdef JQ_BOUNDS_CHECK
    one.ext_y[0] = mats.ext_y[0];
#endif
    return launch_form(st, form, grid, p, one);
}

}  // namespace jq
