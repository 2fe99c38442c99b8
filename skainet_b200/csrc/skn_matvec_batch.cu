// K2 for batches of some activation rows (up to 32 in one launch): Y[M, N] = X[M, K] . W_q[N, K]^T in the accuracy of the
// single-row kernels, on the 5th-generation tensor cores.
//
// The arithmetic is the one of skn_matvec_mma.cu -- 30-bit fixed-point activations per super-block, integer products,
// exact sums per scale block, outliers apart in fp32 -- in numbers that tcgen05 takes: a weight's integer is an exact fp16
// number (Q4_0, Q8_0: the signed quant; Q4_K: quant times 6-bit sub-block scale less about half its range, s q - 8 (s & 60), at
// most 480; Q6_K: quant times either part of its scale 16 h + l, at most 256), an activation is four signed byte digits
// (X = d0 2^24 + d1 2^16 + d2 2^8 + d3, each at most 128) for the K-quants, three of eleven bits (d0 2^22 + d1 2^11 + d2, at most 1024)
// for the others, and an fp32 accumulator holds the sum of such products exactly while it is at most 2^24: 256 columns of Q4_K stay
// below 128 x 480 x 256 = 15.8 M whatever the input is, those of Q6_K below 2^23, the 32 of a Q8_0 or Q4_0 block below 2^22.
// (Before, Q4_K took s q itself, Q6_K the scale as 2 h + b, both three digits: where activations of one sign met large scales the sums
// passed 2^24 and every further step chopped, products 1.6e-7 and 4.3e-7 too small on the mean.)  What the weights of Q4_K lack,
// 8 (s & 60) times the sum of x, joins the dmin term, which it nearly cancels: error against 64 bits 2.1e-7 -> 0.8e-7, time 28.2 ->
// 28.9 us for 14336 x 4096 at 16 rows.  The scale d of a block multiplies what is drained.
//
// What bounded the mma.sync form of this (skn_matvec_rows.cu) was the chain load, MMA, integer multiply-add per 16 rows x
// 32 columns of eight warps; here a thread that unpacks 64 weights needs about two instructions per weight, two threads
// issue the MMAs for 128 rows, and a drained number stands for 256 (32) products.
//
// A CTA owns 128 weight rows (DUAL: 16 gate rows, 16 up rows, ...) x a part of K; the c CTAs of a cluster share K and add their
// sums through distributed shared memory in rank order.
//   unpacking warps   raw super-block columns -> fp16 weight stages, in groups of four
//   four warps        the TMA of the digit planes, that of the raw blocks and block records, and two that issue MMAs
//   draining warps    lane = weight row; scales, offsets (fp32 sums of x), outliers, sums over K in registers; output
//
// Measured (B200, graph of distinct weights, us per call with the preparation of x; the kernels that took these rows before -> one issuing warp, weights
// in shared memory, eight draining warps -> now):
//   Q4_K 14336 x 4096: 16 rows 69 -> 28.1 -> 22.4, 32 rows 137 -> 35.6 -> 28.3; 28672 x 4096: 16 rows 110 -> 56 -> 44.4; 4096 x 4096: 22 -> 13.2 -> 10.1
//   Q4_0 4096 x 14336: 16 rows 75 -> 35.5 -> 31.9, 32 rows 149 -> 52.5 -> 46.0; Q8_0 14336 x 4096: 16 rows 73 -> 43.6 -> 34.1, 24 rows 143 -> 52.2 -> 48.8
//   Q6_K 32000 x 4096: 16 rows 116 -> 92; 4096 x 14336: 186 -> 53.6 -> 43.6
// No one part bounds it: for 14336 x 4096 Q4_K with any of unpacking, products and draining left out it took 24 of 26 us, with all of them left out (rings,
// barriers and loads of the blocks only) 15.4, of which 7.5 are preparation, start and end; two instead of one issuing warp gave 1.0, a second set of
// draining warps 0.8, a fourth unpacking group 0.8.  A deeper ring of blocks, and blocks copied as contiguous pieces, gave nothing.
#include "skn_mma_common.cuh"
#include "skn_tc.cuh"

#include <atomic>

constexpr int MB_ROWS = 128;                       // a stage: two weight tiles of 64 columns (one tile per
                                                  // stage cost the issuing thread its waits and commits every 64 columns)
constexpr int MB_A_TILE = 32, MB_A_COLS = 2 * MB_A_TILE;           // ... in columns of tensor memory
constexpr int MB_A_BYTES = 2 * MB_ROWS * 128;                      // ... in shared memory
constexpr int MB_CHUNK = 8, MB_COLS = 32;         // activation rows of a chunk; its columns (three or four digits of eight rows)
constexpr int MB_MAX_A = 4, MB_MAX_B = 6, MB_MAX_RAW = 4, MB_MAX_D = 8, MB_MAX_SPLIT = 8;
constexpr int MB_SMEM_MAX = 224 * 1024;

// record of one (super-block, activation row), the layout of mm_digitize's outputs
struct __align__(16) mb_meta {
    float scale;                                  // 2^(e-29) (NaN: the block is not finite)
    uint32_t ocnt, oidx, pad;                     // outliers: count, positions (one byte each)
    float oval[MM_MAX_OUT];                       // ... and values
    float xsum[8];                                // sums of 32 activations, outliers excluded
};
constexpr int MB_META = (int)sizeof(mb_meta);
static_assert(MB_META == 64, "block record layout");

// ---- activations -> digit planes and block records ------------------------------------------------------------------
// One CTA per activation row; f(x) = x, x / rms(x) * gain, or silu(x) * u.  Row a's digit p goes to row
// (a / 8) * 32 + p * 8 + a % 8 of `planes` ([32 * chunks][K] fp16); records to meta[super-block][8 * chunks].
// DIGITS: 3 (eleven bits) or 4 (bytes), the leading one first
template <int DIGITS>
__global__ void __launch_bounds__(1024)
skn_xsplit_kernel(const float *__restrict__ x, int K, const float *__restrict__ gain, float eps, const float *__restrict__ silu_u,
                  __half *__restrict__ planes, mb_meta *__restrict__ meta, int rows_pad) {
    skn_pdl_launch_dependents();                  // the product's CTAs may come in and unpack their first weights
    skn_pdl_wait();                               // x is the previous kernel's output; the planes may still be read by it
    const int a = blockIdx.x, nb = K / 256;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const float4 *xr = reinterpret_cast<const float4 *>(x + (size_t)a * K);
    const float4 *ur = silu_u ? reinterpret_cast<const float4 *>(silu_u + (size_t)a * K) : nullptr;
    __shared__ float s_ss[32];
    float rs = 1.f;
    if (gain) {
        float ss = 0.f;
        for (int i = threadIdx.x; i < K / 4; i += blockDim.x) {
            const float4 v = __ldg(xr + i);
            ss += (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) s_ss[warp] = ss;
        __syncthreads();
        float tot = 0.f;
        for (int w = 0; w < nw; ++w) tot += s_ss[w];
        rs = rsqrtf(tot / (float)K + eps);
    }
    auto load = [&](int f) {
        float4 v = __ldg(xr + f);
        if (ur) {
            const float4 u = __ldg(ur + f);
            v.x = v.x / (1.f + expf(-v.x)) * u.x; v.y = v.y / (1.f + expf(-v.y)) * u.y;
            v.z = v.z / (1.f + expf(-v.z)) * u.z; v.w = v.w / (1.f + expf(-v.w)) * u.w;
        }
        if (gain) {
            const float4 g = __ldg(reinterpret_cast<const float4 *>(gain) + f);
            v.x = v.x * rs * g.x; v.y = v.y * rs * g.y; v.z = v.z * rs * g.z; v.w = v.w * rs * g.w;
        }
        return v;
    };
    __half *row = planes + ((size_t)(a / MB_CHUNK) * MB_COLS + a % MB_CHUNK) * K;
    for (int sb = warp; sb < nb; sb += nw) {
        const float4 v0 = load(sb * 64 + lane), v1 = load(sb * 64 + 32 + lane);
        mb_meta *m = meta + (size_t)sb * rows_pad + a;
        int X[8];
        mm_fixed_point<false>(v0, v1, 0, lane, X, &m->scale, m->xsum, m->oval, &m->oidx, reinterpret_cast<uint8_t *>(&m->ocnt), nullptr);
        __half dig[DIGITS][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if constexpr (DIGITS == 4) {
                const uint32_t d = ((uint32_t)X[i] + 0x80808080u) ^ 0x80808080u;       // its bytes are the signed digits
#pragma unroll
                for (int p = 0; p < 4; ++p) dig[p][i] = __int2half_rn((int)(int8_t)(d >> (24 - 8 * p)));
            } else {
                const int d2 = ((X[i] + 1024) & 2047) - 1024, h = (X[i] - d2) >> 11;
                const int d1 = ((h + 1024) & 2047) - 1024;
                dig[0][i] = __int2half_rn((h - d1) >> 11);
                dig[1][i] = __int2half_rn(d1);
                dig[2][i] = __int2half_rn(d2);
            }
        }
#pragma unroll
        for (int p = 0; p < DIGITS; ++p) {
            uint2 *to = reinterpret_cast<uint2 *>(row + (size_t)p * MB_CHUNK * K + sb * 256) + lane;
            to[0] = *reinterpret_cast<const uint2 *>(&dig[p][0]);
            to[32] = *reinterpret_cast<const uint2 *>(&dig[p][4]);
        }
    }
}

// ---- raw blocks -> fp16 integers --------------------------------------------------------------------------------------
template <int TYPE> struct MbFmt;
template <> struct MbFmt<SKN_TYPE_Q4_K> { static constexpr int ROW = 144, MM = MM_FMT_Q4K, BLOCKS = 1, STAGES = 2, DIGITS = 4; };
template <> struct MbFmt<SKN_TYPE_Q4_0> { static constexpr int ROW = 144, MM = MM_FMT_Q40, BLOCKS = 8, STAGES = 2, DIGITS = 3; };
template <> struct MbFmt<SKN_TYPE_Q8_0> { static constexpr int ROW = 272, MM = MM_FMT_Q80, BLOCKS = 8, STAGES = 2, DIGITS = 3; };
// Q6_K: quant times 8-bit scale needs 12 bits.  The scale is taken as 16 h + l, -8 <= l < 8: a stage is 64 columns in two weight
// tiles, (q - 32) h and (q - 32) l, against one tile of digits, into two accumulators
template <> struct MbFmt<SKN_TYPE_Q6_K> { static constexpr int ROW = 240, MM = MM_FMT_Q6K, BLOCKS = 1, STAGES = 4, DIGITS = 4; };

// four bytes b of w -> fp16 (b + 1024) * mul + add: 1024 + b is the byte under the high byte 0x64; all values here are exact
__device__ __forceinline__ void mb_quad(uint32_t w, __half2 mul, __half2 add, uint32_t *out) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t h = __byte_perm(w, 0x64646464u, i ? 0x4342 : 0x4140);
        const __half2 v = __hfma2(*reinterpret_cast<const __half2 *>(&h), mul, add);
        out[i] = *reinterpret_cast<const uint32_t *>(&v);
    }
}
// bytes 0 and 1 of w as fp16
__device__ __forceinline__ void mb_pair(uint32_t w, uint32_t &out) {
    const uint32_t h = __byte_perm(w, 0x64646464u, 0x4140);
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&h), __float2half2_rn(1024.f));
    out = *reinterpret_cast<const uint32_t *>(&v);
}
// half g of stage u of the row at `row` (see the formats' notes in skn_matmul_tc.cu: same cut, same chunks)
template <int TYPE>
__device__ __forceinline__ void mb_half(uint32_t row, int u, int g, uint32_t sc2, uint32_t (&out)[16], int lead = 0, int v = 0) {
    if constexpr (TYPE == SKN_TYPE_Q4_K) {
        const uint4 q = tc_lds128(row + 16 + 32 * u + 16 * g);
        const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
        // (1024 + q) s + a = s q - 8 (s & 60): a is a multiple of 32 down to -64992, so an fp16 number
        uint32_t sp, tp;
        mb_pair(sc2, sp);
        mb_pair(sc2 & 0x3C3Cu, tp);
        const __half2 s = *reinterpret_cast<const __half2 *>(&sp);
        const __half2 a = __hfma2(*reinterpret_cast<const __half2 *>(&tp), __float2half2_rn(-8.f), __hmul2(s, __float2half2_rn(-1024.f)));
        const __half2 s0 = __low2half2(s), s1 = __high2half2(s), a0 = __low2half2(a), a1 = __high2half2(a);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            mb_quad(qw[i] & 0x0F0F0F0Fu, s0, a0, out + 2 * i);
            mb_quad((qw[i] >> 4) & 0x0F0F0F0Fu, s1, a1, out + 8 + 2 * i);
        }
    } else if constexpr (TYPE == SKN_TYPE_Q4_0) {
        uint32_t win[8], w[5];
        tc_window(row + 32 * u + 16 * g, win);
        tc_shift(win, u, 16u * g, w);
        const __half2 one = __float2half2_rn(1.f), add = __float2half2_rn(-1032.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t q = __funnelshift_r(w[i], w[i + 1], 16);
            mb_quad(q & 0x0F0F0F0Fu, one, add, out + 2 * i);
            mb_quad((q >> 4) & 0x0F0F0F0Fu, one, add, out + 8 + 2 * i);
        }
    } else if constexpr (TYPE == SKN_TYPE_Q6_K) {
        const uint32_t sh = (uint32_t)(lead & 2) * 8u;
        uint32_t wl[12], wh[12], ql[8], qh[8], s8;
        tc_window(row + 64 * (u >> 1) + 32 * g, wl);
        tc_window(row + 128 + 32 * (u >> 1), wh);
        tc_shift(wl, lead >> 2, sh, ql);
        tc_shift(wh, lead >> 2, sh, qh);
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(s8) : "r"(row + (uint32_t)lead + 192 + 8 * (u >> 1) + 4 * (u & 1) + 2 * g));   // two int8 scales
        const int i0 = (int)(int8_t)(s8 & 0xFFu), i1 = (int)(int8_t)(s8 >> 8);
        const int l0 = ((i0 + 8) & 15) - 8, l1 = ((i1 + 8) & 15) - 8;
        const __half2 s0 = __half2half2(__int2half_rn(v ? l0 : (i0 - l0) >> 4)), s1 = __half2half2(__int2half_rn(v ? l1 : (i1 - l1) >> 4));
        const int lsh = 4 * (u & 1), hsh = 4 * (u & 1) + 2 * g;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            mb_quad(((ql[i] >> lsh) & 0x0F0F0F0Fu) | (((qh[i] >> hsh) & 0x03030303u) << 4), __float2half2_rn(1.f), __float2half2_rn(-1056.f), out + 2 * i);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const __half2 w = __hmul2(*reinterpret_cast<const __half2 *>(&out[2 * i + e]), i < 4 ? s0 : s1);
                out[2 * i + e] = *reinterpret_cast<const uint32_t *>(&w);
            }
        }
    } else {
        uint32_t win[12], w[9];
        tc_window(row + 64 * u + 32 * g, win);
        tc_shift(win, u, 16u * g, w);
        const __half2 one = __float2half2_rn(1.f), add = __float2half2_rn(-1152.f);
#pragma unroll
        for (int i = 0; i < 8; ++i) mb_quad(__funnelshift_r(w[i], w[i + 1], 16) ^ 0x80808080u, one, add, out + 2 * i);
    }
}
// 6-bit scales (word 1) and minima (word 2) of a Q4_K header as bytes: sub-blocks 0-3, 4-7
__device__ __forceinline__ void mb_q4k_scales(const uint4 &h, uint32_t (&sc)[2], uint32_t (&mn)[2]) {
    sc[0] = h.y & 0x3F3F3F3Fu;
    sc[1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    mn[0] = h.z & 0x3F3F3F3Fu;
    mn[1] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
}
// bytes i and i + 1 as floats: 2^23 + byte, exactly, less 2^23
__device__ __forceinline__ uint64_t mb_bytes2(uint32_t w, int i) {
    return skn_add2(skn_pack2u(__byte_perm(w, 0x4B000000u, 0x7440 + i), __byte_perm(w, 0x4B000000u, 0x7441 + i)), skn_pack2(-8388608.f, -8388608.f));
}

// the sums that the digit sums of rows a and a + 1 stand for
template <int DIGITS> __device__ __forceinline__ uint64_t mb_join(const uint32_t (&D)[32], int a) {
    const uint64_t d0 = skn_pack2u(D[a], D[a + 1]), d1 = skn_pack2u(D[8 + a], D[9 + a]), d2 = skn_pack2u(D[16 + a], D[17 + a]);
    if constexpr (DIGITS == 3) return skn_fma2(d0, skn_pack2(4194304.f, 4194304.f), skn_fma2(d1, skn_pack2(2048.f, 2048.f), d2));
    const uint64_t b = skn_pack2(256.f, 256.f);
    return skn_fma2(skn_fma2(d0, b, d1), skn_pack2(65536.f, 65536.f), skn_fma2(d2, b, skn_pack2u(D[24 + a], D[25 + a])));
}

// The outliers of the record at m times their dequantised weights of the block at `blk`.  Rare and out of line: inlined for every
// row of x it made the kernels' code a tenth larger; times are the same.
template <int MM>
static __device__ __noinline__ float mb_outliers(uint32_t blk, uint32_t m, int n) {
    float sum = 0.f;
#pragma unroll 1
    for (int i = 0; i < n; ++i) sum = fmaf(mm_weight_at<MM>(blk, (int)mm_lds8(m + 8 + (uint32_t)i)), mm_lds32f(m + 16 + 4 * (uint32_t)i), sum);
    return sum;
}

struct mb_args {
    int count, n_act;
    int tcum[4];                                  // tiles before tensor t
    int64_t n_rows[3];
    float *y[3];
    const float *add[3];
    int64_t addstride[3];
};
// Where the weight stages live.  In tensor memory a thread stores its row with two or four instructions and neither its stores nor the MMAs' reads of
// them meet the digit tiles in shared memory (16 rows, one issuing warp: Q4_K 14336 x 4096 28.1 -> 26.2, Q8_0 43.6 -> 35.9, Q6_K 32000 x 4096 116 -> 100 us).  Q4_0 and Q8_0 from three chunks on keep shared memory: they drain two
// blocks of 32 columns at a time, an accumulator each, and beside weights tensor memory would hold one such set (4096 x 14336 Q4_0 at 24 and 32
// rows 49.8 and 52.5 us; with weights in tensor memory and a block at a time 58.7 and 61.7).
__host__ __device__ constexpr bool mb_ts(int type, int nch) { return type == SKN_TYPE_Q4_K || type == SKN_TYPE_Q6_K || nch <= 2; }
// columns of an accumulator set
__host__ __device__ constexpr int mb_set_cols(int type, int nch) { return nch * MB_COLS * (type == SKN_TYPE_Q4_K ? 1 : 2); }
// weight stages in tensor memory: one per unpacking group at least (a group tells its stage's turn by the parity of a phase), a fourth where that
// leaves two accumulator sets; and the sets
__host__ __device__ constexpr int mb_ts_stages(int type, int nch) { return (512 - 4 * MB_A_COLS) / mb_set_cols(type, nch) >= 2 ? 4 : 3; }
__host__ __device__ constexpr int mb_sets(int type, int nch) {
    const int n = (512 - (mb_ts(type, nch) ? mb_ts_stages(type, nch) * MB_A_COLS : 0)) / mb_set_cols(type, nch);
    return n > 8 ? 8 : n;
}
// The warps of a kernel: unpacking groups of four, four special ones (MMA, digits, blocks, MMA), draining ones.
//   GROUPS  a group per weight stage where there are four
//   SETS    draining: the super-blocks of Q4_K, the 64-column tiles of Q4_0 and Q8_0 in turn
//   PARTS   ... and the chunks of x
// The threads share 64 K registers, and a draining thread holds its sums for all its rows of x, so what pays depends on those (us): Q4_0 4096 x 14336 and
// Q8_0 14336 x 4096 at 16 rows, three groups and two sets 32.0 and 34.7, four groups and one set 35.2 and 37.9; Q4_K 14336 x 4096 at 16 rows, four groups
// and two sets 23.6, three 24.5 (1.2 more than now: see the launch's arguments below); at 24 and 32 rows three groups and one set 27.7 and 29.1, four groups 30.2 and 30.8.
template <int TYPE, int NCH> struct MbWarps {
    static constexpr bool FOUR = mb_ts(TYPE, NCH) && mb_ts_stages(TYPE, NCH) == 4, K4 = TYPE == SKN_TYPE_Q4_K, BLOCK = TYPE == SKN_TYPE_Q4_0 || TYPE == SKN_TYPE_Q8_0;
    static constexpr int GROUPS = FOUR && !(BLOCK && NCH > 1) && !(K4 && NCH > 2) ? 4 : 3;
    static constexpr int SETS = !(K4 || BLOCK) || NCH > 2 ? 1 : 2;
    static constexpr int PARTS = NCH == 1 || (K4 && NCH == 2) ? 1 : 2;
    static constexpr int MMA = 4 * GROUPS, TMA_X = MMA + 1, TMA_W = MMA + 2, MMA2 = MMA + 3, DRAIN = MMA + 4, DRAINS = 4 * SETS * PARTS, THREADS = 32 * (DRAIN + DRAINS);
};
struct mb_plan {
    int split, a, b, raw, d;                      // CTAs that share K; ring depths (weight tiles, digit tiles, raw columns, accumulators)
    size_t smem;
};

// (`ar` stays in the parameter space: it is indexed by the tensor of the CTA, and by value every thread would first copy its 120 bytes to local
// memory.  16 rows, Q4_0 8192 x 256 7.8 -> 5.7 us a call, Q4_K 14336 x 4096 23.6 -> 22.2)
template <int TYPE, int NCH, bool DUAL>
__global__ void __launch_bounds__((MbWarps<TYPE, NCH>::THREADS), 1)
skn_matvec_batch_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1,
                        const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ mb_args ar, int K, const mb_plan pl, const mb_meta *__restrict__ meta,
                        int32_t *__restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr bool TS = mb_ts(TYPE, NCH);
    typedef MbWarps<TYPE, NCH> WP;
    constexpr int SETS = WP::SETS, PARTS = WP::PARTS;
    constexpr int ROW = MbFmt<TYPE>::ROW, RAW_BYTES = MB_ROWS * ROW, BLOCKS = MbFmt<TYPE>::BLOCKS;
    constexpr int NCOL = NCH * MB_COLS, SET_COLS = mb_set_cols(TYPE, NCH), B_TILE = NCOL * 128, STAGES = MbFmt<TYPE>::STAGES, B_TILES = 4 / STAGES, B_BYTES = B_TILES * B_TILE, META_BYTES = NCH * MB_CHUNK * MB_META;
    __shared__ uint64_t a_full[MB_MAX_A], a_empty[MB_MAX_A], b_full[MB_MAX_B], b_empty[MB_MAX_B], raw_full[MB_MAX_RAW], meta_full[MB_MAX_RAW],
        raw_empty[MB_MAX_RAW], d_full[MB_MAX_D], d_empty[MB_MAX_D];
    __shared__ uint32_t tmem_slot;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int c = pl.split, kr = c > 1 ? (int)tc_cluster_rank() : 0, tile = (int)blockIdx.x / c;
    const int na = pl.a, nb = pl.b, nraw = pl.raw, nd = pl.d;
    uint8_t *b_ring = smem + (TS ? 0 : (size_t)na * MB_A_BYTES), *raw_ring = b_ring + (size_t)nb * B_BYTES, *meta_ring = raw_ring + (size_t)nraw * RAW_BYTES;
    float *slots = reinterpret_cast<float *>(smem);                // over the rings, once all CTAs of the cluster are done with them
    const int nsb = K / 256, sb0 = kr * nsb / c, sb1 = (kr + 1) * nsb / c, steps = STAGES * (sb1 - sb0);
    // the tile's tensor and first row
    int t = 0;
    if (!DUAL) t = (tile >= ar.tcum[1] ? 1 : 0) + (ar.count > 2 && tile >= ar.tcum[2] ? 1 : 0);
    const int n0 = DUAL ? tile * (MB_ROWS / 2) : (tile - ar.tcum[t]) * MB_ROWS;
    constexpr uint32_t TMEM_COLS = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < na; ++s) {
            skn_mbar_init(&a_full[s], 4);
            skn_mbar_init(&a_empty[s], TYPE == SKN_TYPE_Q4_K ? 1 : 2);       // a commit by every warp that reads the stage
        }
        for (int s = 0; s < nb; ++s) {
            skn_mbar_init(&b_full[s], 1);
            skn_mbar_init(&b_empty[s], TYPE == SKN_TYPE_Q4_K ? 1 : 2);
        }
        for (int s = 0; s < nd; ++s) {
            skn_mbar_init(&d_full[s], TYPE == SKN_TYPE_Q6_K ? 2 : 1);
            skn_mbar_init(&d_empty[s], 4 * PARTS);
        }
        skn_fence_mbar_init();
    }
    auto load_raw = [&](int sb, int rs) {
        uint8_t *dst = raw_ring + (size_t)rs * RAW_BYTES;
        skn_mbar_expect_tx(&raw_full[rs], RAW_BYTES);
        const int x = TYPE == SKN_TYPE_Q6_K ? ((sb * 210) >> 4) * 4 : sb * (ROW / 4);
        if (DUAL) {
            for (int i = 0; i < 4; ++i) {
                tc_tma_load_2d(dst + 32 * i * ROW, &tm_w0, x, n0 + 16 * i, &raw_full[rs]);
                tc_tma_load_2d(dst + (32 * i + 16) * ROW, &tm_w1, x, n0 + 16 * i, &raw_full[rs]);
            }
        } else {
            tc_tma_load_2d(dst, t == 0 ? &tm_w0 : (t == 1 ? &tm_w1 : &tm_w2), x, n0, &raw_full[rs]);
        }
    };
    auto load_meta = [&](int sb, int rs) {
        skn_mbar_expect_tx(&meta_full[rs], META_BYTES);
        skn_bulk_g2s(meta_ring + (size_t)rs * META_BYTES, meta + (size_t)sb * (NCH * MB_CHUNK), META_BYTES, &meta_full[rs]);
    };
    const int early = min(nraw, sb1 - sb0);
    if (warp == WP::TMA_W && lane == 0) {
        for (int s = 0; s < nraw; ++s) {
            skn_mbar_init(&raw_full[s], 1);
            skn_mbar_init(&meta_full[s], 1);
            skn_mbar_init(&raw_empty[s], 4 * WP::GROUPS + (BLOCKS == 1 ? 4 * PARTS : WP::DRAINS));
        }
        skn_fence_mbar_init();
        skn_fence_proxy_async();
        for (int i = 0; i < early; ++i) load_raw(sb0 + i, i);      // the weights depend on no launch before this one
    }
    if (warp == WP::MMA) tc_alloc(&tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot, tmem_a = tmem_base + TMEM_COLS - (uint32_t)(na * MB_A_COLS);      // accumulators, then weight stages

    bool failed = false;
    auto give_up = [&]() {
        failed = true;
        atomicExch(status, SKN_ERR_TIMEOUT);
    };
    if (warp < WP::MMA) {
        // ---------------- unpack: group `turn` takes the stages 3 i + turn ----------------
        const int turn = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t ta = tmem_a + ((uint32_t)(r & 96) << 16);
        const uint32_t raw0 = skn_smem_u32(raw_ring) + (uint32_t)(r * ROW);
        int s = turn % na, rs = 0, it = turn;
        uint32_t ph = (uint32_t)(turn / na), rph = 0;
#pragma unroll 1
        for (int sb = 0; sb < steps / STAGES; ++sb) {           // (every group sees every super-block, with a stage of its own in it or not)
            if (!failed && !tc_wait_warp(&raw_full[rs], rph, lane)) give_up();
            const uint32_t row = raw0 + (uint32_t)(rs * RAW_BYTES);
            const int lead = TYPE == SKN_TYPE_Q6_K ? ((sb0 + sb) * 210) & 15 : 0;
#pragma unroll 1
            for (; it / STAGES == sb; it += WP::GROUPS) {
                uint32_t sc[2] = {0, 0}, mn[2];
                if (TYPE == SKN_TYPE_Q4_K) mb_q4k_scales(tc_lds128(row), sc, mn);
                const uint32_t sc4 = sc[it & 1];           // scales of the stage's four sub-blocks
#pragma unroll 1
                for (int v = 0; v < 2; ++v) {              // the stage's two tiles
                    const uint32_t to = ta + (uint32_t)(s * MB_A_COLS + v * MB_A_TILE);
                    uint8_t *tile_a = smem + (size_t)s * MB_A_BYTES + v * (MB_A_BYTES / 2);
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        uint32_t p[16];
                        mb_half<TYPE>(row, STAGES == 4 ? it & 3 : 2 * (it & 1) + v, g, (sc4 >> (16 * v)) & 0xFFFFu, p, lead, v);
                        if (v == 0 && g == 0) {
                            if (!failed && !tc_wait_warp(&a_empty[s], ph ^ 1u, lane)) give_up();
                            if constexpr (TS) tc_fence_after();                     // the stores follow the MMAs that read the stage
                        }
                        if constexpr (!TS) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) tc_store_chunk(tile_a, r, 4 * g + i, make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]));
                        } else if constexpr (TYPE == SKN_TYPE_Q4_K) {  // 16 columns of either sub-block
                            tc_st8(to + (uint32_t)(8 * g), p);
                            tc_st8(to + (uint32_t)(16 + 8 * g), p + 8);
                        } else {
                            tc_st16(to + (uint32_t)(16 * g), p);
                        }
                    }
                }
                if constexpr (TS) {
                    tc_wait_st();
                    tc_fence_before();
                } else {
                    skn_fence_proxy_async();
                }
                __syncwarp();
                if (lane == 0) skn_mbar_arrive(&a_full[s]);
                for (s += WP::GROUPS; s >= na; s -= na) ph ^= 1u;
            }
            __syncwarp();
            if (lane == 0) skn_mbar_arrive(&raw_empty[rs]);
            if (++rs == nraw) { rs = 0; rph ^= 1u; }
        }
    } else if (warp == WP::TMA_W) {
        // ---------------- raw blocks, and the block records of the activations (previous launch's output) ----------------
        if (lane == 0) {
            skn_pdl_wait();
            for (int i = 0; i < early; ++i) load_meta(sb0 + i, i);
            int rs = 0;
            uint32_t rph = 0;
            for (int sb = sb0 + early; sb < sb1; ++sb) {
                if (!failed && !skn_mbar_wait(&raw_empty[rs], rph)) give_up();
                skn_fence_proxy_async();
                load_raw(sb, rs);
                load_meta(sb, rs);
                if (++rs == nraw) { rs = 0; rph ^= 1u; }
            }
        }
    } else if (warp == WP::TMA_X) {
        if (lane == 0) {
            skn_pdl_wait();
            int s = 0;
            uint32_t ph = 0;
            for (int it = 0; it < steps; ++it) {
                if (!failed && !skn_mbar_wait(TS ? &a_empty[s] : &b_empty[s], ph ^ 1u)) give_up();
                skn_mbar_expect_tx(&b_full[s], B_BYTES);
                for (int v = 0; v < B_TILES; ++v)
                    tc_tma_load_2d(b_ring + (size_t)s * B_BYTES + v * B_TILE, &tm_x, (sb0 * STAGES + it) * (64 * B_TILES) + 64 * v, 0, &b_full[s]);
                if (++s == nb) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == WP::MMA || warp == WP::MMA2) {
        // ---------------- MMAs: 128 rows x NCOL columns, fp16 operands, one accumulator per scale block ----------------
        // Two warps share them: Q4_K's super-blocks in turn, the two tiles of a stage of the others (of Q6_K the two parts of the scale).  A wait
        // by parity tells a phase from the one before it only, so a warp has to see every phase of a barrier that it waits for: the tiles'
        // warps see every stage, and Q4_K's super-blocks of two stages meet the same two of four stages, and the same half of the sets, each time.
        // (The unpacking groups and the digits' warp see a stage of one warp free while one of the other two stages before is not: they are never two
        // uses behind, because a raw column is loaded only when the super-block MB_MAX_RAW before it is drained.)
        static_assert(TYPE != SKN_TYPE_Q4_K || (mb_ts_stages(TYPE, NCH) == 2 * STAGES && MB_MAX_RAW * STAGES <= 2 * mb_ts_stages(TYPE, NCH)), "a warp's stages");
        static_assert(TYPE == SKN_TYPE_Q6_K || mb_sets(TYPE, NCH) % 2 == 0, "a warp's sets");
        // (a wait has one answer for the warp: its lanes elect, and fail, together)
        constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NCOL >> 3) << 17) | ((uint32_t)(MB_ROWS >> 4) << 24);
        const uint64_t a0 = tc_smem_desc(skn_smem_u32(smem)), b0 = tc_smem_desc(skn_smem_u32(b_ring));
        const int p = warp == WP::MMA ? 0 : 1;
        int s = 0, tb = 0, d = 0;
        uint32_t ph = 0, pb = 0, pd = 0;
        auto pass = [&](int stages, int sets) {            // on in the three rings
            for (s += stages; s >= na; s -= na) ph ^= 1u;
            for (tb += stages; tb >= nb; tb -= nb) pb ^= 1u;
            for (d += sets; d >= nd; d -= nd) pd ^= 1u;
        };
        if constexpr (TYPE == SKN_TYPE_Q4_K) {
            if (p) pass(STAGES, 1);
            for (int sb = p; sb < steps / STAGES; sb += 2) {
#pragma unroll 1
                for (int j = 0; j < STAGES; ++j) {
                    if (!failed && !tc_wait_warp(&b_full[tb], pb, &a_full[s], ph, lane)) failed = true;
                    if (j == 0 && !failed && !tc_wait_warp(&d_empty[d], pd ^ 1u, lane)) failed = true;
                    tc_fence_after();
                    const uint32_t ad = tmem_a + (uint32_t)(s * MB_A_COLS), to = tmem_base + (uint32_t)(d * SET_COLS);
                    const uint64_t bd = b0 + (uint64_t)(tb * (B_BYTES >> 4));
                    if (tc_elect()) {
                        // K step k (16 columns): 8 columns of weights; 32 bytes inside a digit tile's swizzle atom = +2 in the address field
#pragma unroll
                        for (int k = 0; k < 8; ++k) tc_mma_ts(to, ad + 8 * k, bd + (k >> 2) * (B_TILE >> 4) + 2 * (k & 3), idesc, (j || k) ? 1u : 0u);
                        tc_commit(&a_empty[s]);
                        if (j == STAGES - 1) tc_commit(&d_full[d]);
                    }
                    pass(1, 0);
                }
                pass(STAGES, 2);                           // the other warp's
            }
        } else {
            // Q6_K: a set of two accumulators, one per part, over four stages; Q4_0 and Q8_0: a set per tile, an accumulator for each of its two blocks
            constexpr bool Q6 = TYPE == SKN_TYPE_Q6_K;
            pass(0, Q6 ? 0 : p);
            for (int it = 0; it < steps; ++it) {
                const bool first = !Q6 || (it & 3) == 0, last = !Q6 || (it & 3) == 3;
                if (!failed && !tc_wait_warp(&b_full[tb], pb, &a_full[s], ph, lane)) failed = true;
                if (first && !failed && !tc_wait_warp(&d_empty[d], pd ^ 1u, lane)) failed = true;
                tc_fence_after();
                const uint32_t ad = tmem_a + (uint32_t)(s * MB_A_COLS + MB_A_TILE * p), to = tmem_base + (uint32_t)(d * SET_COLS + (Q6 ? p * NCOL : 0));
                const uint64_t am = a0 + (uint64_t)(s * (MB_A_BYTES >> 4) + p * (MB_A_BYTES >> 5)), bd = b0 + (uint64_t)(tb * (B_BYTES >> 4) + (Q6 ? 0 : p * (B_TILE >> 4)));
                if (tc_elect()) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t acc = Q6 ? ((it & 3) || k ? 1u : 0u) : (uint32_t)(k & 1), dst = to + (uint32_t)(Q6 ? 0 : (k >> 1) * NCOL);
                        if constexpr (TS) tc_mma_ts(dst, ad + 8 * k, bd + 2 * k, idesc, acc);
                        else tc_mma_bf16(dst, am + 2 * k, bd + 2 * k, idesc, acc);
                    }
                    if (last) tc_commit(&d_full[d]);
                    tc_commit(&a_empty[s]);
                    if constexpr (!TS) tc_commit(&b_empty[tb]);
                }
                pass(1, last ? (Q6 ? 1 : 2) : 0);
            }
        }
        if (failed && lane == 0) atomicExch(status, SKN_ERR_TIMEOUT);
    } else if (warp >= WP::DRAIN) {
        // ---------------- drain: lane = weight row ----------------
        const int wq = warp & 3, r = wq * 32 + lane, part = ((warp - WP::DRAIN) >> 2) % PARTS, set = ((warp - WP::DRAIN) >> 2) / PARTS;
        constexpr int MINE = (NCH + PARTS - 1) / PARTS;    // the chunks part, part + PARTS, ...
        const uint32_t raw0 = skn_smem_u32(raw_ring) + (uint32_t)(r * ROW), meta0 = skn_smem_u32(meta_ring);
        float y[MINE * MB_CHUNK];
#pragma unroll
        for (int a = 0; a < MINE * MB_CHUNK; ++a) y[a] = 0.f;
        // (Q4_K: a set's super-blocks meet the same half of the raw columns and of the accumulators each time; see the issuing warps)
        constexpr int TURN = BLOCKS == 1 ? SETS : 1;
        int rs = TURN > 1 ? set : 0, d = set;
        uint32_t rph = 0, pd = 0;
#pragma unroll 1
        for (int sb = sb0 + (TURN > 1 ? set : 0); sb < sb1; sb += TURN) {
            if (!failed && !tc_wait_warp(&raw_full[rs], rph, lane)) give_up();
            if (!failed && !tc_wait_warp(&meta_full[rs], rph, lane)) give_up();
            const uint32_t row = raw0 + (uint32_t)(rs * RAW_BYTES), mt = meta0 + (uint32_t)(rs * META_BYTES);
            const uint32_t blk = TYPE == SKN_TYPE_Q6_K ? row + (uint32_t)((sb * 210) & 15) : row;
            if constexpr (TYPE == SKN_TYPE_Q6_K) {
                const float db = mm_lds_half(blk + 208);
                if (!failed && !tc_wait_warp(&d_full[d], pd, lane)) give_up();
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < MINE; ++i) {
                    const int ch = PARTS * i + part;
                    if (ch >= NCH) break;
                    const uint32_t at = tmem_base + (uint32_t)(d * SET_COLS + ch * MB_COLS) + ((uint32_t)(wq * 32) << 16);
                    float v[MB_CHUNK];
#pragma unroll
                    for (int p = 0; p < 2; ++p) {                   // digits d3 and d2, then d1 and d0; the scale's parts join digit by digit
                        uint32_t H[16], L[16];
                        tc_ld16x2(at + (uint32_t)(16 * p), at + (uint32_t)(16 * p + NCOL), H, L);
#pragma unroll
                        for (int a = 0; a < MB_CHUNK; ++a) {
                            const float t1 = fmaf(__uint_as_float(H[a]), 16.f, __uint_as_float(L[a])),
                                        t0 = fmaf(__uint_as_float(H[8 + a]), 16.f, __uint_as_float(L[8 + a]));
                            const float t = fmaf(t1, 256.f, t0);
                            if (p == 0) v[a] = t;
                            else y[i * MB_CHUNK + a] = fmaf(fmaf(v[a], 65536.f, t), db * mm_lds32f(mt + (uint32_t)((ch * MB_CHUNK + a) * MB_META)), y[i * MB_CHUNK + a]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) skn_mbar_arrive(&d_empty[d]);
                if (++d == nd) { d = 0; pd ^= 1u; }
            } else if constexpr (TYPE == SKN_TYPE_Q4_K) {
                const uint4 hdr = tc_lds128(row);
                const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
                uint32_t sc[2], mn[2];
                mb_q4k_scales(hdr, sc, mn);
                // what a sub-block's sum of x counts, 8 (s & 60) d - m dmin (products exact, one rounding): sub-blocks 2 j and 2 j + 1
                uint64_t of[4];
                const uint64_t d8 = skn_pack2(8.f * dd.x, 8.f * dd.x), dm = skn_pack2(-dd.y, -dd.y);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    of[j] = skn_fma2(d8, mb_bytes2(sc[j >> 1] & 0x3C3C3C3Cu, 2 * (j & 1)), skn_fma2(dm, mb_bytes2(mn[j >> 1], 2 * (j & 1)), 0ull));
                if (!failed && !tc_wait_warp(&d_full[d], pd, lane)) give_up();
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < MINE; ++i) {
                    const int ch = PARTS * i + part;
                    if (ch >= NCH) break;
                    uint32_t D[32];
                    tc_ld32(tmem_base + (uint32_t)(d * SET_COLS + ch * MB_COLS) + ((uint32_t)(wq * 32) << 16), D);
#pragma unroll
                    for (int a = 0; a < MB_CHUNK; a += 2) {
                        float off[2], sx[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const uint32_t m = mt + (uint32_t)((ch * MB_CHUNK + a + e) * MB_META);
                            sx[e] = dd.x * mm_lds32f(m);
                            const uint4 s0 = tc_lds128(m + 32), s1 = tc_lds128(m + 48);
                            uint64_t o = skn_fma2(of[0], skn_pack2u(s0.x, s0.y), 0ull);
                            o = skn_fma2(of[1], skn_pack2u(s0.z, s0.w), o);
                            o = skn_fma2(of[2], skn_pack2u(s1.x, s1.y), o);
                            o = skn_fma2(of[3], skn_pack2u(s1.z, s1.w), o);
                            float even, uneven;
                            skn_unpack2(o, even, uneven);
                            off[e] = even + uneven;
                        }
                        float *to = y + i * MB_CHUNK + a;
                        skn_unpack2(skn_add2(skn_pack2(to[0], to[1]), skn_fma2(mb_join<4>(D, a), skn_pack2(sx[0], sx[1]), skn_pack2(off[0], off[1]))), to[0], to[1]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) skn_mbar_arrive(&d_empty[d]);
                for (d += SETS; d >= nd; d -= nd) pd ^= 1u;
            } else {
                uint64_t z[MINE * MB_CHUNK / 2];                    // sums over the super-block: short chains of roundings
#pragma unroll
                for (int a = 0; a < MINE * MB_CHUNK / 2; ++a) z[a] = 0ull;
#pragma unroll 1
                for (int u = set; u < 4; u += SETS) {
                    if (!failed && !tc_wait_warp(&d_full[d], pd, lane)) give_up();
                    tc_fence_after();
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float dj = mm_lds_half(row + (uint32_t)((2 * u + j) * (TYPE == SKN_TYPE_Q4_0 ? 18 : 34)));
#pragma unroll
                        for (int i = 0; i < MINE; ++i) {
                            const int ch = PARTS * i + part;
                            if (ch >= NCH) break;
                            uint32_t D[32];
                            tc_ld32(tmem_base + (uint32_t)(d * SET_COLS + j * NCOL + ch * MB_COLS) + ((uint32_t)(wq * 32) << 16), D);
#pragma unroll
                            for (int a = 0; a < MB_CHUNK; a += 2)
                                z[(i * MB_CHUNK + a) / 2] = skn_fma2(mb_join<3>(D, a), skn_pack2(dj, dj), z[(i * MB_CHUNK + a) / 2]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) skn_mbar_arrive(&d_empty[d]);
                    for (d += SETS; d >= nd; d -= nd) pd ^= 1u;
                }
#pragma unroll
                for (int a = 0; a < MINE * MB_CHUNK; ++a)
                    if (PARTS * (a / MB_CHUNK) + part < NCH) {
                        float z0, z1;
                        skn_unpack2(z[a / 2], z0, z1);
                        y[a] = fmaf(a & 1 ? z1 : z0, mm_lds32f(mt + (uint32_t)((MB_CHUNK * (PARTS * (a / MB_CHUNK) + part) + a % MB_CHUNK) * MB_META)), y[a]);
                    }
            }
            // outliers (rare): their products with the whole dequantised weight
            uint32_t any = 0;
            for (int a = BLOCKS == 1 || set == 0 ? lane : ar.n_act; a < ar.n_act; a += 32) any |= mm_lds32(mt + (uint32_t)(a * MB_META) + 4) & 0xFFu;
            if (__any_sync(0xffffffffu, any != 0)) {
#pragma unroll
                for (int a = 0; a < MINE * MB_CHUNK; ++a) {
                    const int act = MB_CHUNK * (PARTS * (a / MB_CHUNK) + part) + a % MB_CHUNK;
                    const uint32_t m = mt + (uint32_t)(act * MB_META);
                    const int n = act < ar.n_act ? (int)(mm_lds32(m + 4) & 0xFFu) : 0;
                    if (n > 0) y[a] += mb_outliers<MbFmt<TYPE>::MM>(blk, m, n);
                }
            }
            __syncwarp();
            if (lane == 0) skn_mbar_arrive(&raw_empty[rs]);
            for (rs += TURN; rs >= nraw; rs -= nraw) rph ^= 1u;
        }
        if constexpr (SETS == 2) {
            // the second set's sums join the first's, through the rings that both are done with
            float *meet = slots + (part * MINE * MB_CHUNK) * MB_ROWS + r;
            asm volatile("barrier.sync 1, %0;" ::"n"(32 * WP::DRAINS) : "memory");
            if (set)
#pragma unroll
                for (int a = 0; a < MINE * MB_CHUNK; ++a) meet[a * MB_ROWS] = y[a];
            asm volatile("barrier.sync 1, %0;" ::"n"(32 * WP::DRAINS) : "memory");
            if (!set)
#pragma unroll
                for (int a = 0; a < MINE * MB_CHUNK; ++a) y[a] += meet[a * MB_ROWS];
        }
        skn_pdl_launch_dependents();
        skn_pdl_wait();                                            // y and add belong to earlier launches
        // partial sums to the CTA that adds up a chunk: [owned chunk][source][row of x][weight row]
        if (c > 1) {
            tc_cluster_sync();
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
                const int ch = PARTS * i + part, owner = ch % c;
                if (set || ch >= NCH || owner == kr) continue;
                const uint32_t to = tc_mapa(skn_smem_u32(slots) + (uint32_t)(((ch / c) * (c - 1) + (kr < owner ? kr : kr - 1)) * (MB_CHUNK * MB_ROWS) + r) * 4u,
                                            (uint32_t)owner);
#pragma unroll
                for (int a = 0; a < MB_CHUNK; ++a)
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + (uint32_t)(a * MB_ROWS * 4)), "f"(y[i * MB_CHUNK + a]) : "memory");
            }
            tc_cluster_sync();
        }
        float *yo = ar.y[t];
        const float *ao = ar.add[t];
        const int64_t N = ar.n_rows[t];
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const int ch = PARTS * i + part;
            if (set || ch >= NCH || ch % c != kr) continue;
            float v[MB_CHUNK];
#pragma unroll
            for (int a = 0; a < MB_CHUNK; ++a) v[a] = y[i * MB_CHUNK + a];
            if (c > 1) {
#pragma unroll 1
                for (int j = 0; j < c; ++j) {                      // in the order of K, whoever adds
                    const float *from = slots + ((ch / c) * (c - 1) + (j < kr ? j : j - 1)) * (MB_CHUNK * MB_ROWS) + r;
#pragma unroll
                    for (int a = 0; a < MB_CHUNK; ++a) {
                        const float p = j == kr ? y[i * MB_CHUNK + a] : from[a * MB_ROWS];
                        v[a] = j == 0 ? p : v[a] + p;
                    }
                }
            }
            if (DUAL) {
                // lane l holds gate (l < 16) or up of column l & 15: the halves trade rows of x, each forms every other product
                const bool low = lane < 16;
                const int f = n0 + 16 * wq + (lane & 15);
#pragma unroll
                for (int a = 0; a < MB_CHUNK; a += 2) {
                    const float got = __shfl_xor_sync(0xffffffffu, low ? v[a + 1] : v[a], 16);
                    const float gate = low ? v[a] : got, up = low ? got : v[a + 1];
                    const int m = ch * MB_CHUNK + a + (low ? 0 : 1);
                    if (m < ar.n_act && f < N) yo[(int64_t)m * N + f] = gate / (1.f + expf(-gate)) * up;
                }
            } else if (n0 + r < N) {
#pragma unroll
                for (int a = 0; a < MB_CHUNK; ++a) {
                    const int m = ch * MB_CHUNK + a;
                    if (m < ar.n_act) yo[(int64_t)m * N + n0 + r] = v[a] + (ao ? ao[(int64_t)m * ar.addstride[t] + n0 + r] : 0.f);
                }
            }
        }
    }
    __syncwarp();
    if (c > 1 && warp < WP::DRAIN) {                                // the other warps' part of the two cluster barriers
        tc_cluster_sync();
        tc_cluster_sync();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == WP::MMA) {
        tc_fence_after();
        tc_dealloc(tmem_base, TMEM_COLS);
    }
}

// ---- launch --------------------------------------------------------------------------------------------------------
static int mb_row_bytes(int type) {
    return type == SKN_TYPE_Q8_0 ? MbFmt<SKN_TYPE_Q8_0>::ROW : (type == SKN_TYPE_Q6_K ? MbFmt<SKN_TYPE_Q6_K>::ROW : MbFmt<SKN_TYPE_Q4_K>::ROW);
}

// K over as many CTAs of a cluster as make the launch shortest: a start and end of 9000, MB_STAGE_CLOCKS per 64 columns of 128 rows and 500 for
// the exchange, in units of about 1.4 clocks (a launch of one super-block takes 7.3 us, 64 columns of Q4_K 680 clocks at 16 rows; Q4_0 and
// Q8_0 weigh more than they are given).  At 2000 for the exchange rows of two super-blocks stayed in one CTA: 512 x 512 at 16 rows
// 8.7 us, split 7.4, Q4_0 9.2 and 7.6, Q8_0 8192 x 768 13.3 and 11.0.  `fit[s]` = CTAs in flight in clusters of s.
constexpr int MB_STAGE_CLOCKS = 500;
static mb_plan mb_make_plan(int type, int nch, int64_t tiles, int K, const int *fit) {
    mb_plan pl = {};
    const int raw_bytes = MB_ROWS * mb_row_bytes(type) + nch * MB_CHUNK * MB_META, b_bytes = nch * MB_COLS * (type == SKN_TYPE_Q6_K ? 128 : 256), nsb = K / 256;
    int64_t best = 0;
    for (int c = 1; c <= MB_MAX_SPLIT && c <= nsb; ++c) {
        if (fit[c] < 1 && c > 1) continue;
        const int64_t f = fit[c] > 0 ? fit[c] : 1, waves = (tiles * c + f - 1) / f;
        const int64_t cost = waves * (9000 + (c > 1 ? 500 : 0) + (int64_t)((nsb + c - 1) / c) * 4 * MB_STAGE_CLOCKS * (type == SKN_TYPE_Q6_K ? 2 : 1));
        if (best == 0 || cost < best) { best = cost; pl.split = c; }
    }
    const bool ts = mb_ts(type, nch);
    pl.a = ts ? mb_ts_stages(type, nch) : 3;
    pl.d = mb_sets(type, nch);
    pl.b = ts ? pl.a : 2;                                          // (in tensor memory both tiles of a stage are freed by one commit)
    pl.raw = 2;                                                    // (an even number: Q4_K's draining sets take them in turn)
    auto bytes = [&](int a, int b, int raw) { return (ts ? 0 : a * MB_A_BYTES) + b * b_bytes + raw * raw_bytes; };
    auto fits = [&](int a, int b, int raw) { return bytes(a, b, raw) <= MB_SMEM_MAX - 1024; };
    for (bool grown = true; grown;) {
        grown = false;
        if (pl.raw < MB_MAX_RAW && fits(pl.a, pl.b, pl.raw + 2)) { pl.raw += 2; grown = true; }
        if (!ts && pl.b < MB_MAX_B && fits(pl.a, pl.b + 1, pl.raw)) { ++pl.b; grown = true; }
        if (!ts && pl.a < MB_MAX_A && fits(pl.a + 1, pl.b, pl.raw)) { ++pl.a; grown = true; }
    }
    pl.smem = (size_t)bytes(pl.a, pl.b, pl.raw) + 1024;      // (the partial sums, 28 KB at most, meet in it)
    return pl;
}

static cudaLaunchConfig_t mb_config(dim3 grid, dim3 block, int cluster, size_t smem, cudaStream_t stream, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cfg;
}

// CTAs in flight in clusters of 1 .. MB_MAX_SPLIT, asked of the driver once per device: the same for all kernels here (threads, shared memory,
// one CTA per SM); asked of each of them, its first call took 15 to 30 us longer on the host.
static cudaError_t mb_fits(const skn_ctx *ctx, const void *kern, int threads, cudaStream_t stream, int (&f)[MB_MAX_SPLIT + 1]) {
    static std::atomic<int> fits[64][MB_MAX_SPLIT + 1];            // 0: not asked yet, -1: none
    std::atomic<int> *fit = fits[ctx->device & 63];
    f[1] = ctx->sm_count;
    for (int s = MB_MAX_SPLIT; s > 1; --s) {
        f[s] = fit[s].load(std::memory_order_relaxed);
        if (f[s]) continue;
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t cfg = mb_config(dim3(s), dim3(threads), s, MB_SMEM_MAX, stream, attr);
        int k = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&k, kern, &cfg);
        if (e != cudaSuccess) return e;
        f[s] = k > 0 ? k * s : -1;
        fit[s].store(f[s], std::memory_order_relaxed);
    }
    return cudaSuccess;
}

template <int TYPE, int NCH, bool DUAL>
static cudaError_t mb_launch(skn_ctx *ctx, int n, const skn_tensor *const *w, const float *x, int M, const mb_args &ar, int64_t tiles, const float *gain,
                             float eps, const float *silu_u, cudaStream_t stream, bool &covered) {
    auto kern = skn_matvec_batch_kernel<TYPE, NCH, DUAL>;
    static std::atomic<bool> large[64];                            // per device: may use MB_SMEM_MAX
    cudaLaunchAttribute attr[2];
    cudaError_t e;
    if (!large[ctx->device & 63].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MB_SMEM_MAX);
        if (e != cudaSuccess) return e;
        large[ctx->device & 63].store(true, std::memory_order_release);
    }
    int f[MB_MAX_SPLIT + 1] = {0};
    if ((e = mb_fits(ctx, (const void *)kern, MbWarps<TYPE, NCH>::THREADS, stream, f)) != cudaSuccess) return e;
    const int K = (int)w[0]->n_cols, rows_pad = NCH * MB_CHUNK;
    const mb_plan pl = mb_make_plan(TYPE, NCH, tiles, K, f);
    const size_t planes = (size_t)NCH * MB_COLS * K * 2;           // a multiple of 1024
    // (while a graph is captured and the buffer is too small, the routes with smaller buffers or none take the call)
    const int32_t rc = skn_xq_reserve(ctx, planes + (size_t)(K / 256) * rows_pad * MB_META, stream);
    if (rc != SKN_OK) return rc == SKN_ERR_BUSY ? cudaErrorNotSupported : cudaErrorMemoryAllocation;
    __half *xp = (__half *)ctx->d_xq;
    mb_meta *meta = reinterpret_cast<mb_meta *>((uint8_t *)ctx->d_xq + planes);
    CUtensorMap tx, tw[3];
    if ((e = skn_tmap_bf16(xp, NCH * MB_COLS, K, (int64_t)K * 2, NCH * MB_COLS, &tx)) != cudaSuccess) return e;   // 16-bit elements, whatever they are
    for (int t = 0; t < 3; ++t)
        if ((e = skn_tmap_blocks(w[t < n ? t : 0], MbFmt<TYPE>::ROW, DUAL ? 16 : MB_ROWS, &tw[t])) != cudaSuccess) return e;
    covered = true;
    const int warps = K / 256 < 32 ? K / 256 : 32;
    const cudaLaunchConfig_t prep = mb_config(dim3((unsigned)M), dim3((unsigned)warps * 32), 1, 0, stream, attr);
    if ((e = cudaLaunchKernelEx(&prep, skn_xsplit_kernel<MbFmt<TYPE>::DIGITS>, x, K, gain, eps, silu_u, xp, meta, rows_pad)) != cudaSuccess) return e;
    const cudaLaunchConfig_t cfg = mb_config(dim3((unsigned)(tiles * pl.split)), dim3(MbWarps<TYPE, NCH>::THREADS), pl.split, pl.smem, stream, attr);
    return cudaLaunchKernelEx(&cfg, kern, tx, tw[0], tw[1], tw[2], ar, K, pl, (const mb_meta *)meta, ctx->d_status);
}

// most rows of a launch: what the shared memory holds beside two raw columns (Q8_0: 35 KB each) and three weight stages
int skn_batch_rows(int32_t type) { return type == SKN_TYPE_Q8_0 ? 24 : 32; }

// whether skn_batch_try_group takes these tensors
bool skn_batch_covers(int n, const skn_tensor *const *w) {
    const skn_tensor *w0 = w[0];
    if (w0->type != SKN_TYPE_Q4_K && w0->type != SKN_TYPE_Q4_0 && w0->type != SKN_TYPE_Q8_0 && w0->type != SKN_TYPE_Q6_K) return false;
    if (n < 1 || n > 3 || w0->n_cols % 256 || w0->n_cols < 256 || w0->n_cols > (1 << 18) || w0->pitch % 16) return false;
    for (int t = 0; t < n; ++t)
        if (w[t]->type != w0->type || w[t]->n_cols != w0->n_cols || w[t]->pitch != w0->pitch || w[t]->n_rows < 1 || w[t]->n_rows > (1 << 28)) return false;
    return true;
}

template <int TYPE, bool DUAL, class... A>
static cudaError_t mb_by_rows(int M, A &&...a) {
    switch ((M + MB_CHUNK - 1) / MB_CHUNK) {
    case 1: return mb_launch<TYPE, 1, DUAL>(a...);
    case 2: return mb_launch<TYPE, 2, DUAL>(a...);
    case 3: return mb_launch<TYPE, 3, DUAL>(a...);
    default:
        if constexpr (TYPE != SKN_TYPE_Q8_0) return mb_launch<TYPE, 4, DUAL>(a...);     // (skn_batch_rows)
        return cudaErrorNotSupported;
    }
}
template <bool DUAL, class... A>
static cudaError_t mb_by_type(int type, int M, A &&...a) {
    switch (type) {
    case SKN_TYPE_Q4_K: return mb_by_rows<SKN_TYPE_Q4_K, DUAL>(M, a...);
    case SKN_TYPE_Q4_0: return mb_by_rows<SKN_TYPE_Q4_0, DUAL>(M, a...);
    case SKN_TYPE_Q6_K: return mb_by_rows<SKN_TYPE_Q6_K, DUAL>(M, a...);
    default: return mb_by_rows<SKN_TYPE_Q8_0, DUAL>(M, a...);
    }
}

// Y[t][m] = W[t] . f(x[m]) (+ add[t]) for n <= 3 tensors of one type, K and pitch and 1 <= M <= skn_batch_rows() activation rows;
// arguments as of skn_rows_try_group.  Returns false when the tensors are not covered (nothing launched).
bool skn_batch_try_group(skn_ctx *ctx, int n, const skn_tensor *const *w, const float *x, int M, float *const *y, const float *const *add,
                         bool add_per_act, const float *norm_gain, float norm_eps, const float *silu_u, bool swiglu, cudaStream_t stream,
                         cudaError_t &err) {
    err = cudaSuccess;
    if (M < 1 || M > skn_batch_rows(w[0]->type) || !skn_batch_covers(n, w)) return false;
    if (swiglu && (n != 2 || w[0]->n_rows != w[1]->n_rows)) return false;
    mb_args ar = {};
    ar.count = n;
    ar.n_act = M;
    int64_t tiles = 0;
    for (int t = 0; t < n; ++t) {
        ar.tcum[t] = (int)tiles;
        if (!swiglu) tiles += (w[t]->n_rows + MB_ROWS - 1) / MB_ROWS;
        ar.n_rows[t] = w[t]->n_rows;
        ar.y[t] = y[t];
        ar.add[t] = add ? add[t] : nullptr;
        ar.addstride[t] = add_per_act ? w[t]->n_rows : 0;
    }
    for (int t = n; t < 4; ++t) ar.tcum[t] = (int)tiles + 1;
    if (swiglu) tiles = (w[0]->n_rows + MB_ROWS / 2 - 1) / (MB_ROWS / 2);
    bool covered = false;
    err = swiglu ? mb_by_type<true>(w[0]->type, M, ctx, n, w, x, M, ar, tiles, norm_gain, norm_eps, silu_u, stream, covered)
                 : mb_by_type<false>(w[0]->type, M, ctx, n, w, x, M, ar, tiles, norm_gain, norm_eps, silu_u, stream, covered);
    if (!covered && (err == cudaErrorInvalidValue || err == cudaErrorNotSupported)) {
        err = cudaSuccess;
        return false;
    }
    return true;
}
