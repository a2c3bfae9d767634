// Small-batch multiply (a few to a few dozen activation columns): an int8 tensor-core kernel that reads every weight
// once per 32 columns (up to 63 where that makes one wave of CTAs) and keeps the memory system busy while it does.
//
// Work to replace: q4_0_q8_1_mat_mul_kernel (reference src/cuda/mm_q4_0_q8_1.cu:164-289) for batched decode.  The
// cost is the weight stream as long as the arithmetic hides behind it, so the kernel is organised around that:
//
//   * A CTA owns 32 * WR weight rows and 8 * CT columns for all of K.  Weights and activations of a K stage arrive by
//     tiled tensor copies in a ring of up to eight stages, as much as shared memory holds: about 200 KB in flight per SM.  Where the
//     rows can be dealt out so that each SM has one CTA, it has one; otherwise two or three CTAs of eight consumer warps share an
//     SM and one's start and end lie behind the others' streams.
//   * The consumer warps split K, not the tile: each takes one pair of 32-value blocks per stage for all rows
//     of its row group and all columns.  So a weight is unpacked once and an activation fragment is read once (WR
//     times) per CTA, the least shared-memory traffic there is, and the activations need no registers between
//     stages, which is what bounds K in the register-resident decode kernels.  The warps' partial tiles are added
//     in a fixed order at the end.
//   * Rows land 144 bytes apart (16 x odd): eight rows x four neighbouring words touch 32 banks.
//   * Per block and 16 x 8 tile one mma.m16n8k32 (u8 nibbles x s8) onto the integer 0x4B400000: read back as a float
//     and less 1.5 * 2^23 it is the block sum exactly (a conversion instruction runs at half the rate), then the
//     reference's acc += d4 * (sumi * d8 - 8 * s8) (mm_q4_0_q8_1.cu:92) in packed fma.
//
// What bounds it: the copies, on the most loaded SM.  Rows of 144 bytes, 256 values of a weight row or 128 of a column, arrive at
// about eight cycles each per SM, so K = 4096, 96 weight rows and 24 columns on an SM are 9.6 us, two CTAs of 64 rows and 24 columns
// 15.  Hence one CTA of many rows instead of several of few: the activations of an SM are then copied once, and no SM has twice the
// rows of another.  K = 4096, N = 11008, which is 344 tiles of 32 rows, 172 of 64 and 115 of 96: M = 12 12.8 -> 10.8 us, M = 24
// 16.9 -> 13.1, M = 32 21.1 -> 16.3, M = 40 24.7 -> 18.8; its weights alone are 3.8 us at the copy bandwidth of the memory.  From some 40
// columns on the arithmetic: 70 warp instructions per 16 x 32 weights and 24 columns.
// Measured and dropped: 16-byte cp.async by two producer warps instead of the tensor copies, 15.2 us at M = 8 there (13.1) and 22.5
// against 18.0 at M = 24; untiled bulk copies of a column's or a row's part of a stage, one per lane, to padded places: 16.9 -> 22.2 us
// for the columns, 42 for the rows; weights of four or eight stages ahead of the previous kernel's end instead of two, no difference.
//
// Rounding.  K % 256 == 0: a warp keeps one running sum over all of its blocks and the warps' parts are added one after the other,
// 1.0 to 1.4 times the error against 64 bits of the kernels that took these shapes up to 32 columns (8e-8 to 12e-8 of the result)
// and a seventh to a half of the integer GEMM's beyond.  An odd multiple of 128 replaces the generic kernel, whose 32 lanes round off
// little (7.3e-8): there the same sums were 1.2 to 1.55 times as far off, so they are kept short.  The two blocks of a pair are added
// to each other first, unless sixteen warps share K; up to eight columns, where registers are left, each of eight warps sums in two
// levels; the parts are added as a tree; beyond K = 2048 a CTA keeps to 32 rows (eight warps along K, not four) and adds the parts of
// eight warps with the rounded-off remainders.  That is 0.93 to 1.06 times the generic kernel's error on average over each group of
// shapes, for 0.98 to 1.06 of the time (at most 1.18: K = 4224, N = 32000, M = 24, where the generic kernel takes eight times as long).
// The same for K % 256 == 0 was measured (1.00 to 1.05 of the time, the former kernels' error) and left out: a decode step turns a
// last bit into a step of the int8 quantizer here and there, up to 4e-3 of its logits, for no gain in their own error (6.2e-3 against
// a chain in 64 bits either way).
//
// A tensor copy wants a row pitch of whole 16-byte units, which K % 256 == 0 gives.  When K is an odd multiple of 128 a
// row is 8 bytes short of that but two rows are not: the even rows are one tensor and the odd rows another (its base 8
// bytes before the first odd row, so that it is aligned), each with the pitch of two rows; the even rows of a group of 32
// become its first m16 tile, the odd ones the second.
#include "tc_common.cuh"

namespace jq {

namespace {

constexpr int SK_MAX_STAGES = 8;
// Consumer warps with several CTAs per SM, and with 32 rows and one CTA per SM, for grids that would leave the second place empty
// anyway (K = 11008, N = 4096, M = 8 17.6 -> 10.6 us, whole linears of K = N = 4096: M = 24 12 -> 9.5 us)
constexpr int SK_WARPS = 8, SK_WARPS_ALONE = 16;
constexpr int SK_BAR_BYTES = 256;       // full[8], empty[8], meet[2]
constexpr int SK_PITCH = 144;           // bytes of a weight row per 256 values of K, of an activation column per 128
constexpr int SK_ODD_PITCH = 160;       // the same for the odd rows of an odd K, which start 8 bytes into their 160
constexpr int SK_MAX_MATS = 4;
constexpr int SK_RED_PITCH = 36;        // floats between two columns of a warp's partial tile: 2 * 36 = 8 mod 32 banks
constexpr int SK_COLUMNS = 32;          // most columns a CTA takes, unless choose_shape gives it all of them
constexpr int SK_FLUSH = 4;             // stages per running sum
constexpr int SK_SHORT_SUPERS = 16;     // K up to 2048: short running sums
constexpr uint32_t SK_MASK4 = 0x0F0F0F0Fu;

struct StreamMaps {
    CUtensorMap w[SK_MAX_MATS];
    CUtensorMap w_odd[SK_MAX_MATS];  // odd rows (K an odd multiple of 128)
    CUtensorMap x;
};

struct StreamParams {
    // Up to four weight matrices that share K and the activations: the row tiles [tile_begin[i], tile_begin[i + 1])
    // are those of matrix i, which writes to y[i], an [M][rows[i]] array.
    float *y[SK_MAX_MATS];
    int64_t rows[SK_MAX_MATS];
    int tile_begin[SK_MAX_MATS + 1];
    int n_mats;
    int64_t M;
    int n_super;         // K / 128
    int order;
    int stages;
    int early_stages;    // stages whose weights may be requested before the preceding kernel in the stream has finished
    int *fault;
    uint32_t poll_limit;
#ifdef JQ_BOUNDS_CHECK
    Extent ext_y[SK_MAX_MATS];  // the tensor copies are bounded by their maps
#endif
};

template <int CT, int WR, bool ODD, int WARPS>
struct StreamTile {
    static constexpr int ROWS = 32 * WR, COLS = 8 * CT;
    // the blocks of a pair are added before they join the running sum (sixteen warps' are short without that: it then only
    // stays where the copies hide it)
    static constexpr bool PAIR_FIRST = ODD && (WARPS == SK_WARPS || CT <= 2);
    static constexpr bool LEVELS = ODD && WARPS == SK_WARPS && CT == 1;  // running sums of SK_FLUSH stages, and one of those
    static constexpr int KW = WARPS / WR;  // warps along K = pairs of blocks per stage
    static constexpr int SUPERS = KW / 2;     // 128-value groups per stage
    // weights of 256 values of K: ROWS rows, or ROWS / 2 even ones and ROWS / 2 odd ones
    static constexpr int HALF_BYTES = ODD ? ROWS / 2 * (SK_PITCH + SK_ODD_PITCH) : ROWS * SK_PITCH;
    static constexpr int SUPER_BYTES = COLS * SK_PITCH;  // activations of 128 values of K
    static constexpr int W_BYTES = (SUPERS / 2) * HALF_BYTES;
    static constexpr int STAGE_BYTES = W_BYTES + SUPERS * SUPER_BYTES;
    static constexpr int RED_BYTES = WARPS * COLS * SK_RED_PITCH * 4;
    static_assert(HALF_BYTES % 128 == 0 && SUPER_BYTES % 128 == 0, "tensor copies land on 128-byte boundaries");
    static_assert(ROWS / 2 * SK_PITCH % 128 == 0, "tensor copies land on 128-byte boundaries");
};

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<uint64_t &>(d))
        : "l"(reinterpret_cast<const uint64_t &>(a)), "l"(reinterpret_cast<const uint64_t &>(b)));
    return d;
}
// Sums of the warps' parts, in an order that is always the same: one after the other, as a tree, or with what each addition
// rounds off added up as well (Knuth's two-sum), so that only the result is rounded.
template <int N>
__device__ __forceinline__ float sum_in_order(const float (&v)[N]) {
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < N; ++k) sum += v[k];
    return sum;
}
template <int N>
__device__ __forceinline__ float sum_tree(float (&v)[N]) {
#pragma unroll
    for (int step = 1; step < N; step *= 2) {
#pragma unroll
        for (int k = 0; k < N; k += 2 * step) v[k] += v[k + step];
    }
    return v[0];
}
template <int N>
__device__ __forceinline__ float sum_compensated(const float (&v)[N]) {
    float sum = v[0], lost = 0.0f;
#pragma unroll
    for (int k = 1; k < N; ++k) {
        const float s = sum + v[k], got = s - sum;
        lost += (sum - (s - got)) + (v[k] - got);
        sum = s;
    }
    return isfinite(sum) ? sum + lost : sum;
}

// sumi * d8 - 8 * s8 of one block for the rows g and g + 8 and two columns
__device__ __forceinline__ void block_terms(float2 (&t)[2], const uint32_t (&a)[4], const uint32_t (&b)[2], float2 d8, float2 m8s) {
    const int magic4[4] = {MAGIC_I, MAGIC_I, MAGIC_I, MAGIC_I};
    const float2 minus = make_float2(-MAGIC_F, -MAGIC_F);
    int c[4];
    mma_u8s8_16832(c, a, b, magic4);
    t[0] = fma2(add2(make_float2(__int_as_float(c[0]), __int_as_float(c[1])), minus), d8, m8s);  // the sum is exact
    t[1] = fma2(add2(make_float2(__int_as_float(c[2]), __int_as_float(c[3])), minus), d8, m8s);
}

// The consumer warps meet on an mbarrier with a bounded wait: a warp whose wait for a stage ran out has left.
__device__ __forceinline__ bool stream_meet(uint64_t *bar, int lane, int *fault, uint32_t limit) {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar);
    return mbar_wait_bounded(bar, 0u, fault, limit);
}

// Weights of stage c (one thread).
template <int CT, int WR, bool ODD, int WARPS>
__device__ __forceinline__ void stream_load_weights(const StreamParams &p, const StreamMaps &maps, int mat, int64_t n0, int c, uint32_t stage,
                                                    uint64_t *full) {
    using T = StreamTile<CT, WR, ODD, WARPS>;
#pragma unroll
    for (int h = 0; h < T::SUPERS / 2; ++h) {
        const int ks = c * T::SUPERS + 2 * h;  // first 128-value group of this half
        if (ks >= p.n_super) break;
        const uint32_t dst = stage + h * T::HALF_BYTES;
        if (ODD) {  // n0 is a multiple of 32
            tma_load_2d(dst, &maps.w[mat], (ks >> 1) * SK_PITCH, (int)(n0 >> 1), full);
            tma_load_2d(dst + T::ROWS / 2 * SK_PITCH, &maps.w_odd[mat], (ks >> 1) * SK_PITCH, (int)(n0 >> 1), full);
        } else {
            tma_load_2d(dst, &maps.w[mat], (ks >> 1) * SK_PITCH, (int)n0, full);
        }
    }
}

// Activations of stage c (lane 0).
template <int CT, int WR, bool ODD, int WARPS>
__device__ __forceinline__ void stream_load_activations(const StreamParams &p, const CUtensorMap *map, int64_t m0, int c, uint32_t stage,
                                                        uint64_t *full) {
    using T = StreamTile<CT, WR, ODD, WARPS>;
#pragma unroll
    for (int i = 0; i < T::SUPERS; ++i) {
        const int ks = c * T::SUPERS + i;
        if (ks >= p.n_super) break;
        const uint32_t dst = stage + T::W_BYTES + i * T::SUPER_BYTES;
        if (p.order == JQ_ORDER_KSUPER_COL)  // the tensor is [n_super * M blocks][144 bytes]
            tma_load_2d(dst, map, 0, (int)((int64_t)ks * p.M + m0), full);
        else                                 // the tensor is [M columns][n_super * 144 bytes]
            tma_load_2d(dst, map, ks * SK_PITCH, (int)m0, full);
    }
}

// PLACES: CTAs per SM
template <int CT, int WR, bool ODD, int WARPS, int PLACES>
__global__ void __launch_bounds__((WARPS + 1) * 32, PLACES) mmq_stream_kernel(const __grid_constant__ StreamParams p, const __grid_constant__ StreamMaps maps) {
    using T = StreamTile<CT, WR, ODD, WARPS>;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem);
    uint64_t *empty = full + SK_MAX_STAGES;
    uint64_t *meet = empty + SK_MAX_STAGES;
    const uint32_t smem_base = smem_u32(smem), ring = smem_base + SK_BAR_BYTES;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], WARPS);
        }
        mbar_init(&meet[0], WARPS);
        mbar_init(&meet[1], WARPS);
        fence_mbar_init();
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    int mat = 0;
    while (mat + 1 < p.n_mats && (int)blockIdx.x >= p.tile_begin[mat + 1]) ++mat;
    const int64_t n0 = (int64_t)((int)blockIdx.x - p.tile_begin[mat]) * T::ROWS;
    const int64_t m0 = (int64_t)blockIdx.y * T::COLS;
    const int n_chunks = (p.n_super + T::SUPERS - 1) / T::SUPERS;

    if (warp == WARPS) {
        // ---- producer: the weights of the first stages may be on their way before the previous kernel is done ------
        if (lane != 0) return;
        const int early = min(p.early_stages, n_chunks);  // at most `stages`: no slot is waited for below
        const auto arm = [&](int c, int s) {
            const int supers = min(T::SUPERS, p.n_super - c * T::SUPERS);
            mbar_arrive_expect_tx(&full[s], (uint32_t)(supers * T::SUPER_BYTES + (supers + 1) / 2 * T::HALF_BYTES));
            stream_load_weights<CT, WR, ODD, WARPS>(p, maps, mat, n0, c, ring + (uint32_t)s * T::STAGE_BYTES, &full[s]);
        };
        for (int c = 0; c < early; ++c) arm(c, c);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        int s = 0;
        uint32_t round = 0;
        for (int c = 0; c < n_chunks; ++c) {
            if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1u, p.fault, p.poll_limit)) return;
            if (c >= early) arm(c, s);
            stream_load_activations<CT, WR, ODD, WARPS>(p, &maps.x, m0, c, ring + (uint32_t)s * T::STAGE_BYTES, &full[s]);
            if (++s == p.stages) {
                s = 0;
                ++round;
            }
        }
        return;
    }

    // ---- consumers: warp (wr, kw) multiplies pair kw of every stage for the 32 rows of row group wr --------------
    const int wr = warp / T::KW, kw = warp % T::KW;
    const int g = lane >> 2, t = lane & 3;
    const int n_pairs = 2 * p.n_super;
    // the warp's m16 tiles of weight rows: 32 neighbouring rows, or (ODD) 16 even and 16 odd ones of them
    const uint32_t w_pair = (uint32_t)((kw >> 2) * T::HALF_BYTES + (kw & 3) * (2 * Q4_BYTES));
    const uint32_t w_off[2] = {w_pair + (uint32_t)((wr * (ODD ? 16 : 32) + g) * SK_PITCH),
                               ODD ? w_pair + (uint32_t)(T::ROWS / 2 * SK_PITCH + (wr * 16 + g) * SK_ODD_PITCH + 8)
                                   : w_pair + (uint32_t)((wr * 32 + 16 + g) * SK_PITCH)};
    const uint32_t x_head = (uint32_t)(T::W_BYTES + (kw >> 1) * T::SUPER_BYTES + (kw & 1) * 8 + 2 * t * SK_PITCH);
    const uint32_t x_off = (uint32_t)(T::W_BYTES + (kw >> 1) * T::SUPER_BYTES + g * SK_PITCH + Q8_QS_OFFSET + (kw & 1) * 2 * QK + 4 * t);
    float2 acc[2][CT][2], sum[2][CT][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) acc[i][j][0] = acc[i][j][1] = sum[i][j][0] = sum[i][j][1] = make_float2(0.0f, 0.0f);

    int s = 0;
    uint32_t parity = 0;
    for (int c = 0; c < n_chunks; ++c) {
        if (!mbar_wait_bounded(&full[s], parity, p.fault, p.poll_limit)) return;
        if (c * T::KW + kw < n_pairs) {
            const uint32_t stage = ring + (uint32_t)s * T::STAGE_BYTES;
            uint32_t a_e[2][4], a_o[2][4];
            float d_e[2][2], d_o[2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t pr = stage + w_off[i] + (uint32_t)(h * 8 * (ODD && i == 1 ? SK_ODD_PITCH : SK_PITCH));
                    const uint32_t u0 = lds_u32(pr + 4 * t), u1 = lds_u32(pr + 4 * t + 4), u2 = lds_u32(pr + 4 * t + 20);
                    const uint32_t we = __funnelshift_r(u0, u1, 16);  // word t of the even block
                    a_e[i][h] = we & SK_MASK4;                        // weights 4t .. 4t + 3
                    a_e[i][2 + h] = (we >> 4) & SK_MASK4;             // weights 16 + 4t ..
                    a_o[i][h] = u2 & SK_MASK4;
                    a_o[i][2 + h] = (u2 >> 4) & SK_MASK4;
                    d_e[i][h] = half_bits_to_float(lds_u16(pr));
                    d_o[i][h] = half_bits_to_float(lds_u16(pr + Q4_BYTES));
                }
            }
#pragma unroll
            for (int j = 0; j < CT; ++j) {
                const uint32_t xb = stage + x_off + (uint32_t)(j * 8 * SK_PITCH);
                const uint32_t b_e[2] = {lds_u32(xb), lds_u32(xb + 16)}, b_o[2] = {lds_u32(xb + 32), lds_u32(xb + 48)};
                const uint32_t sb = stage + x_head + (uint32_t)(j * 8 * SK_PITCH);
                const uint2 s0 = lds_v2(sb), s1 = lds_v2(sb + SK_PITCH);  // columns 2t, 2t + 1: (d, s) of both blocks
                const float2 de = make_float2(half_bits_to_float(s0.x & 0xFFFFu), half_bits_to_float(s1.x & 0xFFFFu));
                const float2 dq = make_float2(half_bits_to_float(s0.y & 0xFFFFu), half_bits_to_float(s1.y & 0xFFFFu));
                const float2 me = make_float2(-8.0f * half_bits_to_float(s0.x >> 16), -8.0f * half_bits_to_float(s1.x >> 16));
                const float2 mo = make_float2(-8.0f * half_bits_to_float(s0.y >> 16), -8.0f * half_bits_to_float(s1.y >> 16));
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float2 te[2], to[2];
                    block_terms(te, a_e[i], b_e, de, me);
                    block_terms(to, a_o[i], b_o, dq, mo);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float2 de2 = make_float2(d_e[i][h], d_e[i][h]), do2 = make_float2(d_o[i][h], d_o[i][h]);
                        if (T::PAIR_FIRST)
                            acc[i][j][h] = add2(acc[i][j][h], fma2(de2, te[h], mul2(do2, to[h])));
                        else
                            acc[i][j][h] = fma2(do2, to[h], fma2(de2, te[h], acc[i][j][h]));
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (T::LEVELS && (c % SK_FLUSH == SK_FLUSH - 1 || c == n_chunks - 1)) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
#pragma unroll
                for (int j = 0; j < CT; ++j) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        sum[i][j][h] = add2(sum[i][j][h], acc[i][j][h]);
                        acc[i][j][h] = make_float2(0.0f, 0.0f);
                    }
                }
            }
        }
        if (++s == p.stages) {
            s = 0;
            parity ^= 1u;
        }
    }

    // ---- partial tiles -> shared memory (the ring is free by now) -> sums in the order of kw -> y ------------------
    if (!stream_meet(&meet[0], lane, p.fault, p.poll_limit)) return;
    const uint32_t mine = ring + (uint32_t)(warp * T::COLS * SK_RED_PITCH * 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int j = 0; j < CT; ++j) {
            const uint32_t at = mine + (uint32_t)(((j * 8 + 2 * t) * SK_RED_PITCH + i * 16 + g) * 4);
            const float2(&out)[2] = T::LEVELS ? sum[i][j] : acc[i][j];
            sts_f32(at, out[0].x);
            sts_f32(at + SK_RED_PITCH * 4, out[0].y);
            sts_f32(at + 32, out[1].x);
            sts_f32(at + SK_RED_PITCH * 4 + 32, out[1].y);
        }
    }
    if (!stream_meet(&meet[1], lane, p.fault, p.poll_limit)) return;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // (long past: orders the stores to y after the previous kernel)
    // warp (wr, kw) takes the columns kw, kw + KW, ... of its row group, a lane per row
    const int64_t n = n0 + wr * 32 + (ODD ? 2 * (lane & 15) + (lane >> 4) : lane);
    const int64_t rows = p.rows[mat];
#pragma unroll
    for (int col = kw; col < T::COLS; col += T::KW) {
        float v[T::KW];
#pragma unroll
        for (int k = 0; k < T::KW; ++k)
            v[k] = __uint_as_float(lds_u32(ring + (uint32_t)((((wr * T::KW + k) * T::COLS + col) * SK_RED_PITCH + lane) * 4)));
        const float total = !ODD ? sum_in_order(v) : WARPS == SK_WARPS && p.n_super > SK_SHORT_SUPERS ? sum_compensated(v) : sum_tree(v);
        const int64_t m = m0 + col;
        if (n < rows && m < p.M && JQ_IN_EXTENT(p.ext_y[mat], p.y[mat] + m * rows + n, sizeof(float), p.fault)) p.y[mat][m * rows + n] = total;
    }
}

template <int CT, int WR, bool ODD, int WARPS, int PLACES = WARPS == SK_WARPS ? 2 : 1>
int run_stream(cudaStream_t st, StreamParams &p, const StreamMaps &maps, const DeviceCaps &caps) {
    using T = StreamTile<CT, WR, ODD, WARPS>;
    const int budget = min(caps.smem_optin, caps.smem_per_sm / PLACES - 1024);  // 1 KB of an SM's is reserved per CTA
    p.stages = min(SK_MAX_STAGES, (budget - SK_BAR_BYTES) / T::STAGE_BYTES);
    if (p.stages < 2 || p.stages * T::STAGE_BYTES < T::RED_BYTES)
        return set_error(JQ_ERR_UNSUPPORTED, "the stages of the small-batch kernel do not fit in shared memory");
    p.early_stages = min(p.early_stages, p.stages);
    const int bytes = SK_BAR_BYTES + p.stages * T::STAGE_BYTES;
    p.tile_begin[0] = 0;
    for (int i = 0; i < p.n_mats; ++i) p.tile_begin[i + 1] = p.tile_begin[i] + (int)((p.rows[i] + T::ROWS - 1) / T::ROWS);
    const int64_t gy = (p.M + T::COLS - 1) / T::COLS;
    if (gy > 65535) return set_error(JQ_ERR_UNSUPPORTED, "too many columns for the small-batch kernel");
    auto kernel = mmq_stream_kernel<CT, WR, ODD, WARPS, PLACES>;
    if (int rc = ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), bytes, true)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.tile_begin[p.n_mats], (unsigned)gy);
    cfg.blockDim = dim3((WARPS + 1) * 32);
    cfg.dynamicSmemBytes = (size_t)bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    (void)cudaGetLastError();  // a stale error of an earlier, unrelated call must not be taken for this launch's
    JQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, p, maps));
    return JQ_OK;
}

// What a CTA takes.
struct StreamShape {
    int wr;     // groups of 32 rows
    int warps;
    int ct;     // groups of 8 columns
    int places = 2;  // CTAs per SM, of eight consumer warps
};

// One wave, one CTA per SM, with as few rows per CTA as that allows: K = 4096, M = 24, N = 14208 (148 CTAs of 96 rows) 17.1 -> 13.3 us,
// N = 14300 (112 of 128) 17.1 -> 16.3, N = 18944 (148 of 128) 18.4 -> 16.7; N = 19200 (150 of 128) would be two waves and stays with
// two CTAs of 64 rows per SM, 24.5.  From three column tiles on, tiles of 64 rows that fill the SMs are given four warps along K;
// everything else eight or, where tiles of 32 rows do not fill them, sixteen, so that enough warps are at work: K = 11008, N =
// 8192, M = 24 (128 CTAs of 64 rows, sixteen warps, instead of 256 of 32) 23.1 -> 21.4 us, K = 3072, N = 8192, M = 48 (two groups of
// columns, so 2 x 128 tiles of 64 rows; 2 x 64 of 128) 13.5 -> 12.7.  How many warps share K decides how the sum is rounded, and
// does not depend on how rows and columns are dealt out beyond that.
//
// 33 to 63 columns are two groups, unless one CTA of all columns makes one wave of what otherwise is more: K = 4096, N = 11008 (115 CTAs of
// 96 rows instead of 2 x 172 of 64) M = 40 24.7 -> 18.8 us, M = 48 24.9 -> 22.4, M = 60 30.9 -> 29.0.  With 128 rows the limit
// is six column tiles, for which the registers lack 44 bytes a thread (96 rows, seven or eight tiles: 56): N = 18944, M = 36 33.5 -> 25.2
// us, M = 48 32.5 -> 31.2; the other side, M = 60, 40.4 in two groups, 59.6 in one.
//
// Up to 4096 values of K the sixteen warps of a CTA of 64 rows have little to do before their sums meet, and with 32 columns many
// sums: K = 1792, M = 28, N = 4800 (150 tiles of 32 rows) 6.9 us in CTAs of 32 rows, 7.2 in 64; K = 512 3.8 / 4.1; with 12 columns N = 4800
// 4.8 / 5.1, N = 5440 (170) 5.4 / 5.2, N = 9472 5.8 / 5.2; K = 4096, M = 28 N = 4800 12.2 / 12.0.
//
// Tiles of 32 rows that are two waves of two CTAs per SM stay that, beyond three share an SM up to two column tiles (then the registers do not
// reach).  K = 4096, M = 16, two / three: 570 tiles 17.4 / 19.2 us, 590 18.1 / 19.3, 600 20.9 / 19.3, 1000 29.2 / 26.6; K = 1024 590
// 7.3 / 7.5, 600 8.8 / 7.5; K = 8192, M = 4 590 25.1 / 26.8, 600 31.6 / 27.0.
//
// An odd K keeps to the shapes that its rounding was settled for, 32 rows only beyond K = 2048.
StreamShape choose_shape(const int64_t (&tiles)[5], int64_t *groups, int64_t M, bool odd, int n_super, int sm_count) {
    *groups = (M + SK_COLUMNS - 1) / SK_COLUMNS;  // columns in equal groups of at most 32
    const int ct = (int)(((M + *groups - 1) / *groups + 7) / 8);
    const auto one_wave = [&](int wr, int64_t n_groups) { return tiles[wr] * n_groups <= sm_count; };
    const bool narrow = odd && n_super > SK_SHORT_SUPERS;
    const bool four_along_k = !narrow && ct >= 3 && tiles[2] * *groups >= sm_count;
    if (!four_along_k) {
        if (one_wave(1, *groups)) return {1, SK_WARPS_ALONE, ct};
        const bool long_k = n_super >= 4096 / SUPER;
        if (!odd && one_wave(2, *groups) && (long_k || (ct < 4 && 10 * tiles[1] * *groups > 11 * sm_count))) return {2, 16, ct};
        // (at most two column tiles below: from three on 64 rows are one wave here)
        if (!odd && !one_wave(2, *groups) && one_wave(3, *groups)) return {3, 24, ct};
        return {1, SK_WARPS, ct, !odd && tiles[1] * *groups > 4 * sm_count ? 3 : 2};
    }
    if (!odd && !one_wave(2, *groups)) {
        if (one_wave(3, *groups)) return {3, 12, ct};
        if (one_wave(4, *groups)) return {4, 16, ct};
        const int all = (int)((M + 7) / 8);
        const int wr = *groups != 2 ? 0 : one_wave(3, 1) ? 3 : one_wave(4, 1) && all <= 6 ? 4 : 0;
        if (wr != 0) {
            *groups = 1;
            return {wr, 4 * wr, all};
        }
    }
    return {2, SK_WARPS, ct};
}

template <int CT>
int run_stream_columns(cudaStream_t st, StreamParams &p, const StreamMaps &maps, const DeviceCaps &caps, StreamShape f, bool odd) {
    if constexpr (CT > 4) {
        if constexpr (CT <= 6) {
            if (f.wr == 4) return run_stream<CT, 4, false, 16>(st, p, maps, caps);
        }
        return run_stream<CT, 3, false, 12>(st, p, maps, caps);
    } else {
        if (odd) {
            if (f.warps == SK_WARPS_ALONE) return run_stream<CT, 1, true, SK_WARPS_ALONE>(st, p, maps, caps);
            if constexpr (CT >= 3) {
                if (f.wr == 2) return run_stream<CT, 2, true, SK_WARPS>(st, p, maps, caps);
            }
            return run_stream<CT, 1, true, SK_WARPS>(st, p, maps, caps);
        }
        if (f.wr == 1 && f.warps == SK_WARPS_ALONE) return run_stream<CT, 1, false, SK_WARPS_ALONE>(st, p, maps, caps);
        if (f.wr == 2 && f.warps == 16) return run_stream<CT, 2, false, 16>(st, p, maps, caps);
        if constexpr (CT <= 2) {
            if (f.wr == 3) return run_stream<CT, 3, false, 24>(st, p, maps, caps);
            if (f.places == 3) return run_stream<CT, 1, false, SK_WARPS, 3>(st, p, maps, caps);
            return run_stream<CT, 1, false, SK_WARPS>(st, p, maps, caps);
        } else {
            if (f.wr == 1) return run_stream<CT, 1, false, SK_WARPS>(st, p, maps, caps);
            if (f.wr == 3) return run_stream<CT, 3, false, 12>(st, p, maps, caps);
            if (f.wr == 4) return run_stream<CT, 4, false, 16>(st, p, maps, caps);
            return run_stream<CT, 2, false, SK_WARPS>(st, p, maps, caps);
        }
    }
}

// The maps of one weight matrix.  Row pitch (of two rows, if odd) and bases are multiples of 16 bytes, and no map covers
// a byte outside the matrix but the 8 before each odd row, which end the even row ahead of it.
int encode_weight_maps(CUtensorMap *even, CUtensorMap *odd_rows, const void *d_w, int64_t rows, uint32_t row_bytes, int tile_rows, bool odd) {
    const uint8_t *w = static_cast<const uint8_t *>(d_w);
    if (!odd) return encode_byte_map(even, w, row_bytes, (uint64_t)rows, row_bytes, SK_PITCH, (uint32_t)tile_rows);
    if (int rc = encode_byte_map(even, w, row_bytes, (uint64_t)(rows + 1) / 2, 2ull * row_bytes, SK_PITCH, (uint32_t)tile_rows / 2)) return rc;
    // a single row has no odd one: a map of the even row in its place, whose bytes only reach outputs that are not stored
    if (rows < 2) return encode_byte_map(odd_rows, w, row_bytes, 1, 2ull * row_bytes, SK_ODD_PITCH, (uint32_t)tile_rows / 2);
    return encode_byte_map(odd_rows, w + row_bytes - 8, row_bytes + 8, (uint64_t)rows / 2, 2ull * row_bytes, SK_ODD_PITCH, (uint32_t)tile_rows / 2);
}

}  // namespace

int launch_mmq_stream(cudaStream_t st, const void *d_w, const void *d_xq, float *d_y, int64_t K, int64_t N, int64_t M, int order,
                      const MultiMat *multi) {
    if (K % SUPER != 0) return set_error(JQ_ERR_UNSUPPORTED, "small-batch kernel needs K %% 128 == 0 (K = %lld)", (long long)K);
    if (N == 0 || M == 0 || K == 0) return JQ_OK;
    const int64_t n_super = K / SUPER;
    if (K > (1 << 24) || N > (int64_t)1 << 31 || n_super * M >= (int64_t)1 << 31)
        return set_error(JQ_ERR_UNSUPPORTED, "shape too large for the small-batch kernel");
    if (((uintptr_t)d_xq & 15u) != 0) return set_error(JQ_ERR_UNSUPPORTED, "small-batch kernel needs 16-byte aligned Q8_1 blocks");
    DeviceCaps caps;
    if (int rc = device_caps(&caps)) return rc;
    StreamParams p{};
    p.n_mats = multi != nullptr ? multi->n : 1;
    if (p.n_mats < 1 || p.n_mats > SK_MAX_MATS) return set_error(JQ_ERR_INVALID_ARG, "1 to %d weight matrices per launch", SK_MAX_MATS);
    const void *w[SK_MAX_MATS] = {};
    uintptr_t bits = 0;
    int64_t tiles[5] = {};  // of 32, 64, 96 and 128 rows
    const uint32_t row_bytes = (uint32_t)(K / QK * Q4_BYTES);
    for (int i = 0; i < p.n_mats; ++i) {
        w[i] = multi != nullptr ? multi->w[i] : d_w;
        p.y[i] = multi != nullptr ? multi->y[i] : d_y;
        p.rows[i] = multi != nullptr ? multi->rows[i] : N;
        bits |= (uintptr_t)w[i];
        for (int wr = 1; wr <= 4; ++wr) tiles[wr] += (p.rows[i] + 32 * wr - 1) / (32 * wr);
#ifdef JQ_BOUNDS_CHECK
        p.ext_y[i] = make_extent(p.y[i], (unsigned long long)M * (unsigned long long)p.rows[i] * sizeof(float));
#endif
    }
    if ((bits & 15u) != 0) return set_error(JQ_ERR_UNSUPPORTED, "small-batch kernel needs 16-byte aligned weights");
    const bool odd = n_super % 2 != 0;
    p.M = M;
    p.n_super = (int)n_super;
    p.order = order;
    p.fault = device_fault_ptr();
    p.poll_limit = copy_wait_poll_limit();
    p.early_stages = option_value(JQ_OPT_STATIC_WEIGHTS) != 0 ? 2 : 0;
    int64_t groups = 0;  // of columns
    const StreamShape shape = choose_shape(tiles, &groups, M, odd, (int)n_super, caps.sm_count);
    const int ct = shape.ct;
    StreamMaps maps{};
    for (int i = 0; i < p.n_mats; ++i)
        if (int rc = encode_weight_maps(&maps.w[i], &maps.w_odd[i], w[i], p.rows[i], row_bytes, 32 * shape.wr, odd)) return rc;
    const uint64_t x_row = (uint64_t)n_super * Q8_BYTES;
    if (int rc = order == JQ_ORDER_KSUPER_COL
                     ? encode_byte_map(&maps.x, d_xq, Q8_BYTES, (uint64_t)n_super * (uint64_t)M, Q8_BYTES, Q8_BYTES, 8u * (uint32_t)ct)
                     : encode_byte_map(&maps.x, d_xq, x_row, (uint64_t)M, x_row, Q8_BYTES, 8u * (uint32_t)ct))
        return rc;
    switch (ct) {
        case 1: return run_stream_columns<1>(st, p, maps, caps, shape, odd);
        case 2: return run_stream_columns<2>(st, p, maps, caps, shape, odd);
        case 3: return run_stream_columns<3>(st, p, maps, caps, shape, odd);
        case 4: return run_stream_columns<4>(st, p, maps, caps, shape, odd);
        case 5: return run_stream_columns<5>(st, p, maps, caps, shape, odd);
        case 6: return run_stream_columns<6>(st, p, maps, caps, shape, odd);
        case 7: return run_stream_columns<7>(st, p, maps, caps, shape, odd);
        default: return run_stream_columns<8>(st, p, maps, caps, shape, odd);
    }
}

}  // namespace jq
