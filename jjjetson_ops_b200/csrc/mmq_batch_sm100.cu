// Batches of a few to a few dozen columns on the 5th-generation tensor cores: exact int32 block sums by tcgen05.mma.kind::i8.
//
// Work to replace: q4_0_q8_1_mat_mul_kernel (reference src/cuda/mm_q4_0_q8_1.cu:164-289) for batched decode.
#include <algorithm>

#include "tc_common.cuh"

namespace jq {

namespace {

constexpr int SB_ROWS = 128;   // weight rows per CTA: the lanes of its tensor memory
constexpr int SB_COLS = 16;    // activation columns per CTA
constexpr int SB_CHAINS = 4;   // running sums over K per output and CTA
constexpr int SB_W_SLOTS = 4, SB_X_SLOTS = 4, SB_T_SLOTS = 4;
constexpr int SB_W_SLOT_BYTES = SB_ROWS * Q8_BYTES;  // two chunks (144 bytes) of each row
constexpr int SB_Q_BYTES = SB_COLS * SUPER;          // a chunk's int8 values, 128-byte swizzle
constexpr int SB_H_BYTES = SB_COLS * 16;             // ... (d, s) pairs
constexpr int SB_D4_BYTES = SB_ROWS * 16;            // scales of a chunk's four blocks per row, fp32
constexpr int SB_C_BYTES = 4 * (SB_COLS / 2) * 16;   // per block and pair of columns: d8 of both, -8 * s8 of both
constexpr int SB_T_BYTES = SB_D4_BYTES + SB_C_BYTES;
constexpr int SB_W_OFF = SB_X_SLOTS * SB_Q_BYTES;
constexpr int SB_H_OFF = SB_W_OFF + SB_W_SLOTS * SB_W_SLOT_BYTES;
constexpr int SB_T_OFF = SB_H_OFF + SB_X_SLOTS * SB_H_BYTES;
constexpr int SB_BIAS_OFF = SB_T_OFF + SB_T_SLOTS * SB_T_BYTES;
constexpr int SB_BAR_OFF = SB_BIAS_OFF + SB_COLS * 32;
constexpr int SB_SUMS_OFF = SB_BAR_OFF + 256;
constexpr int SB_SUM_BYTES = SB_ROWS * 4;            // one column of a chain
// Tensor memory: two chunks of four integer tiles, two chunks of weights, the constant tile
constexpr uint32_t SB_D_CHUNK = 4 * SB_COLS, SB_A_COL = 2 * SB_D_CHUNK, SB_A_CHUNK = 32, SB_64_COL = SB_A_COL + 2 * SB_A_CHUNK;
constexpr int SB_TMEM_COLS = 256;
constexpr int SB_MAX_MATS = 4, SB_MAX_PARTS = 4;

// SETS groups of four drain warps (a quarter of the rows each) take eight columns each.
template <int SETS>
struct SbTile {
    static constexpr int DRAIN_WARPS = 4 * SETS, CONV_WARP = DRAIN_WARPS, HEAD_WARP = CONV_WARP + 4, MMA_WARP = HEAD_WARP + 1, COPY_W_WARP = HEAD_WARP + 2;
    static constexpr int THREADS = (HEAD_WARP + 4) * 32;
    // the chains' sums: on their own for eight columns, where a chain may end early, else where the weights were
    static constexpr int SUMS_OFF = SETS == 1 ? SB_SUMS_OFF : SB_W_OFF;
    static constexpr int SMEM_BYTES = SB_SUMS_OFF + (SETS == 1 ? SB_CHAINS * 8 * SB_SUM_BYTES : 0);
    static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs do not share an SM");
    static_assert(SB_CHAINS * 8 * SETS * SB_SUM_BYTES <= SB_W_SLOTS * SB_W_SLOT_BYTES, "the sums do not fit in shared memory");
};
static_assert(SB_W_OFF % 1024 == 0 && SB_H_OFF % 128 == 0 && SB_T_BYTES % 128 == 0 && SB_BAR_OFF % 128 == 0, "copies land on whole patterns");
static_assert(SB_64_COL + 8 <= SB_TMEM_COLS, "tensor memory too small");

struct SbMaps {
    CUtensorMap w[SB_MAX_MATS];
    CUtensorMap q, h;
};
struct SbParams {
    // Up to four weight matrices that share K and the activations: the CTAs with blockIdx.x in [tile_begin[i],
    // tile_begin[i + 1]) have 128 rows each of matrix i, which goes to y[i], an [M][rows[i]] array.
    float *y[SB_MAX_MATS];
    int64_t rows[SB_MAX_MATS];
    int tile_begin[SB_MAX_MATS + 1];
    int n_mats;
    int *fault;
#ifdef JQ_BOUNDS_CHECK
    Extent ext_y[SB_MAX_MATS];  // the tensor copies are bounded by their maps
#endif
    int64_t M;
    int n_pairs;         // K / 256
    int parts;           // CTAs along K: a cluster
    int pairs_per_part;  // of part z: these from z * pairs_per_part on, or, 0, every parts-th from z on
    int chain_chunks;    // (neighbouring pairs) chunks per chain
    int order, static_weights;
    uint32_t poll_limit;
};

// D(s32) (+)= A(s8, TMEM: lane = row, four values of K per column) x B(s8 tile in shared memory)^T, K = 32
__device__ __forceinline__ void sb_mma_i8(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void sb_tmem_st8(uint32_t taddr, uint32_t v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(v) : "memory");
}
__device__ __forceinline__ void sb_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
                 "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void sb_tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ float2 sb_add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<uint64_t &>(d)) : "l"(reinterpret_cast<const uint64_t &>(a)), "l"(reinterpret_cast<const uint64_t &>(b)));
    return d;
}
__device__ __forceinline__ float2 sb_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t &>(d))
        : "l"(reinterpret_cast<const uint64_t &>(a)), "l"(reinterpret_cast<const uint64_t &>(b)), "l"(reinterpret_cast<const uint64_t &>(c)));
    return d;
}
__device__ __forceinline__ bool sb_wait(uint64_t *bar, uint32_t parity, const SbParams &p) {
    return __all_sync(0xFFFFFFFFu, mbar_wait_bounded(bar, parity, p.fault, p.poll_limit)) != 0;
}

// One block of eight columns and 32 rows: acc += d4 * (sumi * d8 - 8 * s8), with sumi read from tensor memory as 2^17 + sumi, a
// (subnormal) multiple of 2^-149 as a float.  The powers of two in the scales cancel, so every rounding is that of the plain formula.
__device__ __forceinline__ void sb_add_block(float2 (&acc)[4], const uint32_t (&v)[8], float d4, uint32_t scales) {
    const float2 bias = make_float2(-__uint_as_float(1u << 17), -__uint_as_float(1u << 17)), d42 = make_float2(d4, d4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint4 k = lds_v4(scales + i * 16);
        const float2 x = sb_add2(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), bias);  // exact
        const float2 t = sb_fma2(x, make_float2(__uint_as_float(k.x), __uint_as_float(k.y)), make_float2(__uint_as_float(k.z), __uint_as_float(k.w)));
        acc[i] = sb_fma2(d42, t, acc[i]);
    }
}

// NEIGHBOURS: a chain is some neighbouring chunks of K; else the chains take the pairs of blocks in turn
template <int SETS, bool NEIGHBOURS>
__global__ void __launch_bounds__(SbTile<SETS>::THREADS, 2) mmq_batch_kernel(const __grid_constant__ SbParams p, const __grid_constant__ SbMaps maps) {
    using T = SbTile<SETS>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    uint64_t *w_full = reinterpret_cast<uint64_t *>(smem + SB_BAR_OFF);  // raw weights have landed
    uint64_t *w_empty = w_full + SB_W_SLOTS;
    uint64_t *x_full = w_empty + SB_W_SLOTS;   // activations have landed
    uint64_t *x_empty = x_full + SB_X_SLOTS;   // ... used by the MMAs and by the header warp
    uint64_t *t_full = x_empty + SB_X_SLOTS;   // a chunk's weights are in tensor memory, its tables in shared memory
    uint64_t *t_empty = t_full + SB_T_SLOTS;   // ... drained
    uint64_t *d_full = t_empty + SB_T_SLOTS;   // [2] a chunk's MMAs are done
    uint64_t *d_empty = d_full + 2;            // [2] its integer tiles have been read
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(d_empty + 2);
    static_assert((2 * (SB_W_SLOTS + SB_X_SLOTS + SB_T_SLOTS) + 4) * 8 + 4 <= 256, "barrier block too small");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int mat = 0;
    while (mat + 1 < p.n_mats && (int)blockIdx.x >= p.tile_begin[mat + 1]) ++mat;
    const int64_t n0 = (int64_t)((int)blockIdx.x - p.tile_begin[mat]) * SB_ROWS, m0 = (int64_t)blockIdx.y * SB_COLS;
    // this CTA's pairs of chunks: first, first + step, ...
    const int first = NEIGHBOURS ? (int)blockIdx.z * p.pairs_per_part : (int)blockIdx.z, step = NEIGHBOURS ? 1 : p.parts;
    const int n_pairs = NEIGHBOURS ? max(0, min(p.pairs_per_part, p.n_pairs - first)) : (p.n_pairs - first + step - 1) / step;
    const int n_chunks = 2 * n_pairs;

    if (tid == 0) {
        for (int i = 0; i < SB_W_SLOTS; ++i) {
            mbar_init(&w_full[i], 1);
            mbar_init(&w_empty[i], 8);  // four warps for each of two chunks
        }
        for (int i = 0; i < SB_X_SLOTS; ++i) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], 2);
        }
        for (int i = 0; i < SB_T_SLOTS; ++i) {
            mbar_init(&t_full[i], 5);
            mbar_init(&t_empty[i], T::DRAIN_WARPS);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&d_full[i], 1);
            mbar_init(&d_empty[i], T::DRAIN_WARPS);
        }
        fence_mbar_init();
    }
    if (tid < SB_COLS * 2) {  // the constant tile: every value 64
        sts_v4(sbase + SB_BIAS_OFF + tid * 16, make_uint4(0x40404040u, 0x40404040u, 0x40404040u, 0x40404040u));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == T::MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(SB_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp < T::DRAIN_WARPS) {
        // =============================== integer tiles -> scaled sums ========================
        const int gw = warp & 3, set = warp >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(gw * 32) << 16) + (uint32_t)(set * 8);
        const uint32_t sums = sbase + T::SUMS_OFF + (uint32_t)(set * 8 * SB_SUM_BYTES + (gw * 32 + lane) * 4);
        constexpr int ACCS = NEIGHBOURS ? 1 : SB_CHAINS;
        float2 acc[ACCS][4];
#pragma unroll
        for (int h = 0; h < ACCS; ++h)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[h][i] = make_float2(0.0f, 0.0f);
        const auto store_chain = [&](int chain, const float2(&a)[4]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sts_f32(sums + (uint32_t)((chain * 8 * SETS + 2 * i) * SB_SUM_BYTES), a[i].x);
                sts_f32(sums + (uint32_t)((chain * 8 * SETS + 2 * i + 1) * SB_SUM_BYTES), a[i].y);
            }
        };
        int chain = 0, in_chain = 0;
#pragma unroll 1
        for (int c0 = 0; c0 < n_chunks; c0 += 2) {
            bool alive = true;
#pragma unroll
            for (int par = 0; par < 2; ++par) {
                const int c = c0 + par, ts = c % SB_T_SLOTS;
                alive = sb_wait(&t_full[ts], (uint32_t)(c / SB_T_SLOTS) & 1u, p) && sb_wait(&d_full[par], (uint32_t)(c >> 1) & 1u, p);
                if (!alive) break;
                tc_fence_after();
                const uint32_t tile = lanes + (uint32_t)par * SB_D_CHUNK, table = sbase + SB_T_OFF + ts * SB_T_BYTES;
                const uint32_t scales = table + SB_D4_BYTES + (uint32_t)(set * 4 * 16);
                constexpr uint32_t BLOCK = (SB_COLS / 2) * 16;
                const uint4 d4 = lds_v4(table + (uint32_t)(gw * 32 + lane) * 16);
                float2(&a)[4] = acc[NEIGHBOURS ? 0 : 2 * par], (&e)[4] = acc[NEIGHBOURS ? 0 : 2 * par + 1];
                uint32_t v[4][8];
                sb_tmem_ld8(tile, v[0]);
                sb_tmem_ld8(tile + SB_COLS, v[1]);
                if (SETS == 1) {
                    sb_tmem_ld8(tile + 2 * SB_COLS, v[2]);
                    sb_tmem_ld8(tile + 3 * SB_COLS, v[3]);
                }
                tmem_ld_wait();
                if (SETS == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&d_empty[par]);
                }
                sb_add_block(a, v[0], __uint_as_float(d4.x), scales);
                sb_add_block(a, v[1], __uint_as_float(d4.y), scales + BLOCK);
                if (SETS > 1) {  // (64 registers: two blocks at a time)
                    sb_tmem_ld8(tile + 2 * SB_COLS, v[2]);
                    sb_tmem_ld8(tile + 3 * SB_COLS, v[3]);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&d_empty[par]);
                }
                sb_add_block(e, v[2], __uint_as_float(d4.z), scales + 2 * BLOCK);
                sb_add_block(e, v[3], __uint_as_float(d4.w), scales + 3 * BLOCK);
                __syncwarp();
                if (lane == 0) mbar_arrive(&t_empty[ts]);
                if (NEIGHBOURS && ++in_chain == p.chain_chunks) {
                    store_chain(chain++, acc[0]);
                    in_chain = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[0][i] = make_float2(0.0f, 0.0f);
                }
            }
            if (!alive) break;
        }
        if (NEIGHBOURS) {
            for (; chain < SB_CHAINS; ++chain) {  // one that K ends in, and those behind it
                store_chain(chain, acc[0]);
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[0][i] = make_float2(0.0f, 0.0f);
            }
        } else {
#pragma unroll
            for (int h = 0; h < ACCS; ++h) store_chain(h, acc[h]);
        }
    } else if (warp < T::HEAD_WARP) {
        // =============================== weights -> tensor memory, scales -> table ============
        const int gw = warp & 3;  // the quarter of the lanes it can reach
        const int row = gw * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(gw * 32) << 16);
        sb_tmem_st8(lanes + SB_64_COL, 0x40404040u);
        bool alive = true;
#pragma unroll 1
        for (int c = 0; c < n_chunks; ++c) {
            const int ws = (c >> 1) % SB_W_SLOTS, ts = c % SB_T_SLOTS, b = c & 1;
            if (!sb_wait(&w_full[ws], (uint32_t)((c >> 1) / SB_W_SLOTS) & 1u, p)) break;
            uint32_t ww[18];
            load_q4_chunk(ww, sbase + SB_W_OFF + ws * SB_W_SLOT_BYTES + (uint32_t)(row * Q8_BYTES), b != 0);
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_empty[ws]);
            float d4[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t o[16];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    uint32_t q[4], dbits;
                    q4_chunk_block(ww, 2 * h + u, q, &dbits);
                    d4[2 * h + u] = half_bits_to_float(dbits);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {  // byte i: value i (low nibble) and value i + 16 (high nibble)
                        o[8 * u + t] = q[t] & 0x0F0F0F0Fu;
                        o[8 * u + 4 + t] = (q[t] >> 4) & 0x0F0F0F0Fu;
                    }
                }
                if (h == 0) {
                    // the weights of chunk c - 2 have been multiplied, the tables of chunk c - SB_T_SLOTS used
                    alive = (c < 2 || sb_wait(&d_full[b], (uint32_t)((c >> 1) - 1) & 1u, p)) &&
                            (c < SB_T_SLOTS || sb_wait(&t_empty[ts], (uint32_t)(c / SB_T_SLOTS - 1) & 1u, p));
                    if (!alive) break;
                    tc_fence_after();
                }
                sb_tmem_st16(lanes + SB_A_COL + (uint32_t)b * SB_A_CHUNK + (uint32_t)(16 * h), o);
            }
            if (!alive) break;
            constexpr float TWO49 = 562949953421312.0f;
            sts_v4(sbase + SB_T_OFF + ts * SB_T_BYTES + (uint32_t)row * 16,
                   make_uint4(__float_as_uint(d4[0] * TWO49), __float_as_uint(d4[1] * TWO49), __float_as_uint(d4[2] * TWO49), __float_as_uint(d4[3] * TWO49)));
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_full[ts]);
        }
    } else if (warp == T::HEAD_WARP) {
        // =============================== scales of the activations -> table ===================
        const int col = lane & 15;
#pragma unroll 1
        for (int c = 0; c < n_chunks; ++c) {
            const int xs = c % SB_X_SLOTS, ts = c % SB_T_SLOTS;
            if (!sb_wait(&x_full[xs], (uint32_t)(c / SB_X_SLOTS) & 1u, p)) break;
            const uint2 ds = lds_v2(sbase + SB_H_OFF + xs * SB_H_BYTES + (uint32_t)(col * 16 + (lane >> 4) * 8));
            const uint32_t dsw[2] = {ds.x, ds.y};
            __syncwarp();
            if (lane == 0) mbar_arrive(&x_empty[xs]);
            if (c >= SB_T_SLOTS && !sb_wait(&t_empty[ts], (uint32_t)(c / SB_T_SLOTS - 1) & 1u, p)) break;
            constexpr float TWO100 = 1267650600228229401496703205376.0f, M8_TWO_MINUS49 = -1.4210854715202004e-14f;  // -8 * 2^-49 = -2^-46
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j = 2 * (lane >> 4) + u;
                const uint32_t at = sbase + SB_T_OFF + ts * SB_T_BYTES + SB_D4_BYTES + (uint32_t)((j * (SB_COLS / 2) + (col >> 1)) * 16 + (col & 1) * 4);
                sts_f32(at, half_bits_to_float(dsw[u] & 0xFFFFu) * TWO100);
                sts_f32(at + 8, half_bits_to_float(dsw[u] >> 16) * M8_TWO_MINUS49);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&t_full[ts]);
        }
    } else if (warp == T::MMA_WARP) {
        // =============================== MMA issuer ==========================================
        if (lane == 0) {
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(SB_COLS >> 3) << 17) | ((uint32_t)(SB_ROWS >> 4) << 24);
            const uint64_t bias = tc_desc(sbase + SB_BIAS_OFF);
            for (int c = 0; c < n_chunks; ++c) {
                const int xs = c % SB_X_SLOTS, ts = c % SB_T_SLOTS, b = c & 1;
                if (!mbar_wait_bounded(&t_full[ts], (uint32_t)(c / SB_T_SLOTS) & 1u, p.fault, p.poll_limit)) break;
                if (!mbar_wait_bounded(&x_full[xs], (uint32_t)(c / SB_X_SLOTS) & 1u, p.fault, p.poll_limit)) break;
                if (c >= 2 && !mbar_wait_bounded(&d_empty[b], (uint32_t)((c >> 1) - 1) & 1u, p.fault, p.poll_limit)) break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)b * SB_D_CHUNK, a = tmem + SB_A_COL + (uint32_t)b * SB_A_CHUNK, q = sbase + xs * SB_Q_BYTES;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sb_mma_i8(d + j * SB_COLS, tmem + SB_64_COL, bias, idesc, 0u);  // 32 * 64 * 64 = 2^17
                    sb_mma_i8(d + j * SB_COLS, a + j * 8, tc_desc_sw128(q + j * 32), idesc, 1u);
                }
                tc_commit(&x_empty[xs]);
                tc_commit(&d_full[b]);
            }
        }
    } else if (warp == T::COPY_W_WARP) {
        if (lane == 0) {
            if (!p.static_weights) asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int pr = 0; pr < n_pairs; ++pr) {
                const int ws = pr % SB_W_SLOTS;
                if (pr >= SB_W_SLOTS && !mbar_wait_bounded(&w_empty[ws], (uint32_t)(pr / SB_W_SLOTS - 1) & 1u, p.fault, p.poll_limit)) break;
                mbar_arrive_expect_tx(&w_full[ws], SB_W_SLOT_BYTES);
                tma_load_2d(sbase + SB_W_OFF + ws * SB_W_SLOT_BYTES, &maps.w[mat], (first + pr * step) * Q8_BYTES, (int)n0, &w_full[ws]);
            }
        }
    } else {
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int c = 0; c < n_chunks; ++c) {
                const int xs = c % SB_X_SLOTS, chunk = 2 * (first + (c >> 1) * step) + (c & 1);
                if (c >= SB_X_SLOTS && !mbar_wait_bounded(&x_empty[xs], (uint32_t)(c / SB_X_SLOTS - 1) & 1u, p.fault, p.poll_limit)) break;
                mbar_arrive_expect_tx(&x_full[xs], SB_Q_BYTES + SB_H_BYTES);
                const bool by_super = p.order == JQ_ORDER_KSUPER_COL;  // the tensor is [n_super * M blocks][144 bytes], else [M][n_super * 144]
                const int x = by_super ? 0 : chunk * Q8_BYTES, y = by_super ? (int)((int64_t)chunk * p.M + m0) : (int)m0;
                tma_load_2d(sbase + xs * SB_Q_BYTES, &maps.q, x + Q8_QS_OFFSET, y, &x_full[xs]);
                tma_load_2d(sbase + SB_H_OFF + xs * SB_H_BYTES, &maps.h, x, y, &x_full[xs]);
            }
        }
    }

    // Every CTA of the cluster adds up its share of the outputs over all chains, in their order.
    cluster_sync();
    asm volatile("griddepcontrol.wait;" ::: "memory");  // (long past: orders the stores to y after the previous kernel)
    {
        const int z = (int)blockIdx.z, parts = p.parts;
        const int64_t N = p.rows[mat];
        float *const y = p.y[mat];
        constexpr int OUTPUTS = 8 * SETS * SB_ROWS;
        for (int e = OUTPUTS * z / parts + tid, end = OUTPUTS * (z + 1) / parts; e < end; e += T::THREADS) {
            float v[SB_MAX_PARTS][SB_CHAINS];
#pragma unroll
            for (int q = 0; q < SB_MAX_PARTS; ++q)
#pragma unroll
                for (int h = 0; h < SB_CHAINS; ++h)
                    v[q][h] = q < parts ? lds_f32_of(sbase + T::SUMS_OFF + (uint32_t)(h * OUTPUTS + e) * 4, q) : 0.0f;
            float sum = 0.0f;
#pragma unroll
            for (int q = 0; q < SB_MAX_PARTS; ++q)
#pragma unroll
                for (int h = 0; h < SB_CHAINS; ++h) sum += v[q][h];
            const int64_t m = m0 + e / SB_ROWS, n = n0 + e % SB_ROWS;
            if (m < p.M && n < N && JQ_IN_EXTENT(p.ext_y[mat], y + m * N + n, sizeof(float), p.fault)) y[m * N + n] = sum;
        }
    }
    cluster_sync();  // nobody leaves while another still reads its sums

    tc_fence_before();
    __syncthreads();
    if (warp == T::MMA_WARP) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(SB_TMEM_COLS) : "memory");
    }
}

int sb_byte_map(CUtensorMap *map, const void *base, uint64_t row_len, uint64_t rows, uint64_t pitch, uint32_t box_bytes, uint32_t box_rows,
                CUtensorMapSwizzle swizzle) {
    const EncodeTiledFn encode = tensor_map_encoder();
    if (encode == nullptr) return set_error(JQ_ERR_UNSUPPORTED, "the driver does not export cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {row_len, rows};
    const cuuint64_t strides[1] = {pitch};
    const cuuint32_t box[2] = {box_bytes, box_rows};
    const cuuint32_t elem_strides[2] = {1u, 1u};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, elem_strides,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(JQ_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return JQ_OK;
}

template <int SETS, bool NEIGHBOURS>
int sb_launch(cudaStream_t st, dim3 grid, const SbParams &p, const SbMaps &maps) {
    using T = SbTile<SETS>;
    const auto kernel = mmq_batch_kernel<SETS, NEIGHBOURS>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), T::SMEM_BYTES, true)) return rc;
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
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)p.parts;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, maps));
    return JQ_OK;
}

}  // namespace

int launch_mmq_batch(cudaStream_t st, const void *d_w, const void *d_xq, float *d_y, int64_t K, int64_t N, int64_t M, int order,
                     const MultiMat *multi) {
    if (K % (2 * SUPER) != 0) return set_error(JQ_ERR_UNSUPPORTED, "tcgen05 batch kernel needs K %% 256 == 0 (K = %lld)", (long long)K);
    const void *w[SB_MAX_MATS] = {};
    SbParams p{};
    p.n_mats = multi != nullptr ? multi->n : 1;
    if (p.n_mats < 1 || p.n_mats > SB_MAX_MATS) return set_error(JQ_ERR_INVALID_ARG, "1 to %d weight matrices per launch", SB_MAX_MATS);
    uintptr_t bits = (uintptr_t)d_xq;
    int64_t tiles32 = 0, tiles64 = 0;
    for (int i = 0; i < p.n_mats; ++i) {
        w[i] = multi != nullptr ? multi->w[i] : d_w;
        p.y[i] = multi != nullptr ? multi->y[i] : d_y;
        p.rows[i] = multi != nullptr ? multi->rows[i] : N;
        bits |= (uintptr_t)w[i];
        tiles32 += (p.rows[i] + 31) / 32;
        tiles64 += (p.rows[i] + 63) / 64;
    }
    if ((bits & 15u) != 0) return set_error(JQ_ERR_UNSUPPORTED, "tcgen05 batch kernel needs 16-byte aligned operands");
    if (N == 0 || M == 0) return JQ_OK;
    DeviceCaps caps;
    if (int rc = device_caps(&caps)) return rc;
    if (caps.cc / 10 != 10) return set_error(JQ_ERR_UNSUPPORTED, "tcgen05 needs an sm_100-class device");
    const int64_t gy = (M + SB_COLS - 1) / SB_COLS;
    if (gy > 65535 || K > (1 << 24) || (K / SUPER) * M >= ((int64_t)1 << 31) || N >= ((int64_t)1 << 31))
        return set_error(JQ_ERR_UNSUPPORTED, "shape too large for the tcgen05 batch kernel");
    p.fault = device_fault_ptr();
    p.M = M;
    p.n_pairs = (int)(K / (2 * SUPER));
    p.order = order;
    p.static_weights = option_value(JQ_OPT_STATIC_WEIGHTS) != 0 ? 1 : 0;
    p.poll_limit = copy_wait_poll_limit();
    // How K is summed (@@RULE@@)
    const bool neighbours = M <= 8 && K <= 6144;
    if (neighbours) {
        p.chain_chunks = K <= 4096 ? 2 : 3;
        p.pairs_per_part = SB_CHAINS * p.chain_chunks / 2;
        p.parts = (p.n_pairs + p.pairs_per_part - 1) / p.pairs_per_part;
    } else {
        const int64_t groups = (M + 31) / 32, columns = (M + groups - 1) / groups;
        const bool wide = columns > 16 && tiles64 * groups >= caps.sm_count;
        p.parts = wide ? 1 : tiles32 * groups <= caps.sm_count ? 4 : 2;
    }
    SbMaps maps{};
    const uint32_t row_bytes = (uint32_t)(K / QK * Q4_BYTES);
    p.tile_begin[0] = 0;
    for (int i = 0; i < p.n_mats; ++i) {
        p.tile_begin[i + 1] = p.tile_begin[i] + (int)((p.rows[i] + SB_ROWS - 1) / SB_ROWS);
        if (int rc = encode_byte_map(&maps.w[i], w[i], row_bytes, (uint64_t)p.rows[i], row_bytes, Q8_BYTES, SB_ROWS)) return rc;
#ifdef JQ_BOUNDS_CHECK
        p.ext_y[i] = make_extent(p.y[i], (unsigned long long)M * (unsigned long long)p.rows[i] * sizeof(float));
#endif
    }
    const uint64_t n_super = (uint64_t)K / SUPER, x_row = n_super * Q8_BYTES;
    const bool by_super = order == JQ_ORDER_KSUPER_COL;
    const uint64_t len = by_super ? Q8_BYTES : x_row, rows = by_super ? n_super * (uint64_t)M : (uint64_t)M;
    if (int rc = sb_byte_map(&maps.q, d_xq, len, rows, len, SUPER, SB_COLS, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    if (int rc = sb_byte_map(&maps.h, d_xq, len, rows, len, 16, SB_COLS, CU_TENSOR_MAP_SWIZZLE_NONE)) return rc;
    const dim3 grid((unsigned)p.tile_begin[p.n_mats], (unsigned)gy, (unsigned)p.parts);
    if (neighbours) return sb_launch<1, true>(st, grid, p, maps);
    return M <= 8 ? sb_launch<1, false>(st, grid, p, maps) : sb_launch<2, false>(st, grid, p, maps);
}

}  // namespace jq
