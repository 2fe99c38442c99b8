// K3 / K4: prefill matmul on the 5th-generation tensor cores (tcgen05 + TMEM).
//
//   Y[M,N] = A[M,K] . W_q[N,K]^T      A = bf16 copy of the activations, W_q = raw GGUF blocks
//
// Weights are the MMA's first operand (TMEM lane = feature), tokens its columns.  A PAIR of CTAs (cta_group::2) owns
// 256 features x up to 512 tokens: each CTA dequantises its own 128 features, holds half of the tokens' operand tile
// and accumulates 128 features x all tokens in its TMEM (two accumulators of up to 256 columns).  What decides the
// shape: a weight has to be dequantised once per 512 tokens only (it was once per 256, and once per 128 for layers of
// few features, and the dequantising warps were the limit), and a pair reads 64 KB of activations from L2 for every
// 256 x 512 x 64 products, half of what two single CTAs read.
// Layers with few feature tiles are split along K over the c pairs of one cluster (c <= 4); the partial sums meet
// through distributed shared memory, every CTA adding up a slice of the tokens in rank order.
//
//   warps 4 i (the ones of scheduler 0) lead the asynchronous work: warp 0 issues the pair's MMAs (in the leading CTA) or
//               passes "my weights are in place" on to the leader (in the other), warp 4 is the TMA of the activations,
//               warp 8 that of the raw weights (no multicast)
//   the others  dequantise: raw super-block columns (128 rows x 256 weights, brought by TMA into a ring of their own)
//               -> bf16 rows of the K-major, 128B-swizzled operand tile, 64 weights of K per stage
//   all         epilogue
// The issuing thread shares its scheduler with no dequantising warp: beside four of them it took 1250 clocks for a
// stage's handful of instructions, whatever the number of tokens, and bounded every shape.
//
// Measured (B200, stream of distinct weights with the conversion of x, before -> now; before: one CTA per 128 features x 128 or 256
// tokens that read its weights with word loads from global memory), us:
//   512 tokens: 28672 x 4096 Q4_K 187 -> 106; 4096 x 14336 Q4_K 138 -> 64, Q8_0 311 -> 71, Q6_K 213 -> 71; 4096 x 4096 46 -> 29
//   96 tokens:  28672 x 4096 Q4_K 85 -> 66; 4096 x 14336 133 -> 42; 4096 x 4096 44 -> 22; 1024 x 4096 42 -> 18
// At 512 tokens the tensor cores bound a stage (1020 clocks for 8 MMAs of 256 x 256 x 16); below 350 the dequantisation does.
//
// All waits are bounded.
#include "skn_blocks.cuh"
#include "skn_ptx.cuh"
#include "skn_tc.cuh"

#include <atomic>

constexpr int TC_ROWS = 128, TC_BK = 64;
constexpr int TC_A_BYTES = TC_ROWS * TC_BK * 2;   // 16 KB: a CTA's weight tile of one stage
constexpr int TC_WARPS = 16, TC_THREADS = TC_WARPS * 32;
constexpr int TC_DQ_WARPS = 12, TC_DQ_GROUPS = 3; // groups of four warps (one row per thread) take the stages in turn
constexpr int TC_MMA = 0, TC_TMA_X = 4, TC_TMA_W = 8;
constexpr int TC_MAX_A = 6, TC_MAX_B = 8, TC_MAX_RAW = 4, TC_MAX_TOKENS = 512, TC_MAX_SPLIT = 4;
constexpr int TC_BLOCK = 32;                      // tokens per TMEM load; unit of the token slices
constexpr uint32_t TC_BLOCK_BYTES = TC_BLOCK * TC_ROWS * 4;
constexpr int TC_SMEM_MAX = 226 * 1024;

// ---- pair-of-CTAs forms of the tcgen05 wrappers, cluster barriers ----------------------------------------------
__device__ __forceinline__ void tc2_alloc(uint32_t *slot_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(skn_smem_u32(slot_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc2_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrives on the barrier at this offset in every CTA of `mask` once the MMAs issued so far are done
__device__ __forceinline__ void tc2_commit(uint64_t *bar, uint16_t mask) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(skn_smem_u32(bar)),
                 "h"(mask)
                 : "memory");
}
__device__ __forceinline__ void tc2_mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// tiled TMA load (no multicast) into this CTA's shared memory, counted on a barrier of the pair's leader
__device__ __forceinline__ void tc2_tma_load_2d(void *dst_smem, const CUtensorMap *tmap, int x, int y, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(skn_smem_u32(dst_smem)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(bar_cluster)
        : "memory");
}
// What the arrival announces is read by the tensor cores only and was handed to their proxy by a fence before, so the
// default scope does: `.release.cluster` waits for all of the warp's stores to be acknowledged.
__device__ __forceinline__ void tc_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// ---- raw blocks -> bf16 ----------------------------------------------------------------------------------------
// A raw stage holds 256 weights of 128 rows as a TMA box, ROW bytes per row.  ROW is a multiple of 16 whose word count
// is 4 mod 8, so the 16-byte loads of eight lanes on eight consecutive rows meet all 32 banks once.  A thread turns the
// 64 weights of its row and stage into eight 16-byte chunks, in two halves g.  Code is kept small (what differs between
// stages is an address, a shift, or one of four ways to cut words out of a window): it is fetched by every warp.
template <int TYPE> struct TcFmt;
template <> struct TcFmt<SKN_TYPE_Q4_K> { static constexpr int ROW = 144; };
template <> struct TcFmt<SKN_TYPE_Q4_0> { static constexpr int ROW = 144; };
template <> struct TcFmt<SKN_TYPE_Q8_0> { static constexpr int ROW = 272; };
template <> struct TcFmt<SKN_TYPE_Q6_K> { static constexpr int ROW = 240; };   // 210 from an address rounded down to 16, padded to 60 words
// x coordinate (in 4-byte units, a multiple of 4) of super-block sb's box
template <int TYPE> __device__ __forceinline__ int tc_box_x(int sb) {
    return TYPE == SKN_TYPE_Q6_K ? ((sb * 210) >> 4) * 4 : sb * (TcFmt<TYPE>::ROW / 4);
}

// Four bytes of w, each an unsigned integer weight -> two bf16 pairs of (byte - zero) * scale + off, rounded as in fp32.
// A byte under the high byte 0x64 is the fp16 number 1024 + byte: one permute makes two of them, one packed subtraction
// (exact; `base` = 1024 + zero) removes the 1024.  The path through fp16 keeps the logic pipe, which runs at half rate,
// to 1.4 instructions per weight; building the fp32 bit patterns directly took 1.9.
__device__ __forceinline__ void tc_quad(uint32_t w, __half2 base, uint64_t scale, uint64_t off, uint32_t *out) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t h = __byte_perm(w, 0x64646464u, i ? 0x4342 : 0x4140);
        const float2 f = __half22float2(__hsub2(*reinterpret_cast<const __half2 *>(&h), base));
        float lo, hi;
        skn_unpack2(skn_fma2(skn_pack2(f.x, f.y), scale, off), lo, hi);
        out[i] = tc_pack_bf16(lo, hi);
    }
}
constexpr uint64_t TC_NEG_ZERO2 = 0x8000000080000000ull;   // (-0, -0): v * s + (-0) is the rounded product

// Stage u (weights 64 u .. 64 u + 63 of the super-block) of the row at `row`: what both halves share, then half g as
// sixteen bf16 pairs.  `lead`: bytes between the box's start and the super-block's (even; 0 but for Q6_K).
template <int TYPE> struct TcStage;

// Q4_K: half g is bytes 16 g .. of the stage's 32-byte run; low nibbles belong to sub-block 2 u, high to 2 u + 1
template <> struct TcStage<SKN_TYPE_Q4_K> {
    uint64_t sc0, sc1, of0, of1;
    __device__ __forceinline__ TcStage(uint32_t row, int u, int) {
        const uint4 hdr = tc_lds128(row);
        const int sh = (u & 1) * 16;
        const uint32_t a2 = (hdr.y >> sh) & 0xFFFFu, b2 = (hdr.z >> sh) & 0xFFFFu, c2 = (hdr.w >> sh) & 0xFFFFu;
        const uint32_t sc2 = (u < 2) ? (a2 & 0x3F3Fu) : ((c2 & 0x0F0Fu) | ((a2 >> 2) & 0x3030u));
        const uint32_t mn2 = (u < 2) ? (b2 & 0x3F3Fu) : (((c2 >> 4) & 0x0F0Fu) | ((b2 >> 2) & 0x3030u));
        const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
        const float s0 = __fmul_rn(dd.x, (float)(sc2 & 0xFFu)), s1 = __fmul_rn(dd.x, (float)(sc2 >> 8));
        const float m0 = -__fmul_rn(dd.y, (float)(mn2 & 0xFFu)), m1 = -__fmul_rn(dd.y, (float)(mn2 >> 8));
        sc0 = skn_pack2(s0, s0); sc1 = skn_pack2(s1, s1); of0 = skn_pack2(m0, m0); of1 = skn_pack2(m1, m1);
    }
    __device__ __forceinline__ void half(uint32_t row, int u, int g, int, uint32_t (&out)[16]) const {
        const uint4 q = tc_lds128(row + 16 + 32 * u + 16 * g);
        const __half2 base = __float2half2_rn(1024.f);
        const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            tc_quad(qw[i] & 0x0F0F0F0Fu, base, sc0, of0, out + 2 * i);
            tc_quad((qw[i] >> 4) & 0x0F0F0F0Fu, base, sc1, of1, out + 8 + 2 * i);
        }
    }
};
// Q4_0, Q8_0: half g is block 2 u + g, which starts u words and g half-words into its 16-byte aligned window
template <> struct TcStage<SKN_TYPE_Q4_0> {
    __device__ __forceinline__ TcStage(uint32_t, int, int) {}
    __device__ __forceinline__ void half(uint32_t row, int u, int g, int, uint32_t (&out)[16]) const {
        uint32_t win[8], w[5];
        tc_window(row + 32 * u + 16 * g, win);           // (36 u + 18 g) & ~15
        tc_shift(win, u, 16u * g, w);                    // scale | first half-word of the quants, ...
        const float d = skn_half_bits_to_float(w[0] & 0xFFFFu);
        const __half2 base = __float2half2_rn(1024.f + 8.f);
        const uint64_t sc = skn_pack2(d, d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {                    // low nibbles: weights 0 .. 15, high: 16 .. 31
            const uint32_t q = __funnelshift_r(w[i], w[i + 1], 16);
            tc_quad(q & 0x0F0F0F0Fu, base, sc, TC_NEG_ZERO2, out + 2 * i);
            tc_quad((q >> 4) & 0x0F0F0F0Fu, base, sc, TC_NEG_ZERO2, out + 8 + 2 * i);
        }
    }
};
template <> struct TcStage<SKN_TYPE_Q8_0> {
    __device__ __forceinline__ TcStage(uint32_t, int, int) {}
    __device__ __forceinline__ void half(uint32_t row, int u, int g, int, uint32_t (&out)[16]) const {
        uint32_t win[12], w[9];
        tc_window(row + 64 * u + 32 * g, win);           // (68 u + 34 g) & ~15
        tc_shift(win, u, 16u * g, w);
        const float d = skn_half_bits_to_float(w[0] & 0xFFFFu);
        const __half2 base = __float2half2_rn(1024.f + 128.f);
        const uint64_t sc = skn_pack2(d, d);
#pragma unroll
        for (int i = 0; i < 8; ++i) tc_quad(__funnelshift_r(w[i], w[i + 1], 16) ^ 0x80808080u, base, sc, TC_NEG_ZERO2, out + 2 * i);
    }
};
// Q6_K: half g is run 2 (u & 1) + g of the block's half u / 2
template <> struct TcStage<SKN_TYPE_Q6_K> {
    float d;
    __device__ __forceinline__ TcStage(uint32_t row, int, int lead) {
        uint32_t dh;
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(dh) : "r"(row + (uint32_t)lead + 208));
        d = skn_half_bits_to_float(dh);
    }
    __device__ __forceinline__ void half(uint32_t row, int u, int g, int lead, uint32_t (&out)[16]) const {
        const uint32_t sh = (uint32_t)(lead & 2) * 8u;
        uint32_t wl[12], wh[12], ql[8], qh[8], s2;
        tc_window(row + 64 * (u >> 1) + 32 * g, wl);
        tc_window(row + 128 + 32 * (u >> 1), wh);
        tc_shift(wl, lead >> 2, sh, ql);
        tc_shift(wh, lead >> 2, sh, qh);
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(s2) : "r"(row + (uint32_t)lead + 192 + 8 * (u >> 1) + 4 * (u & 1) + 2 * g));   // two int8 scales
        const float s0 = __fmul_rn(d, (float)(int8_t)(s2 & 0xFFu)), s1 = __fmul_rn(d, (float)(int8_t)(s2 >> 8));
        const __half2 base = __float2half2_rn(1024.f + 32.f);
        const uint64_t sc0 = skn_pack2(s0, s0), sc1 = skn_pack2(s1, s1);
        const int lsh = 4 * (u & 1), hsh = 4 * (u & 1) + 2 * g;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            tc_quad(((ql[i] >> lsh) & 0x0F0F0F0Fu) | (((qh[i] >> hsh) & 0x03030303u) << 4), base, i < 4 ? sc0 : sc1, TC_NEG_ZERO2, out + 2 * i);
    }
};

__global__ void skn_f32_to_bf16_kernel(const float *__restrict__ in, __nv_bfloat16 *__restrict__ out, int64_t n4) {
    skn_pdl_launch_dependents();             // the product's CTAs may come in and dequantise their first weights meanwhile
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(in) + i);
        uint2 o;
        o.x = tc_pack_bf16(v.x, v.y);
        o.y = tc_pack_bf16(v.z, v.w);
        reinterpret_cast<uint2 *>(out)[i] = o;
    }
}

// How a launch is cut up (tc_make_plan below).
struct tc_plan {
    int nacc, nn;           // accumulators, tokens of each (a multiple of 32, at most 256)
    int blocks;             // token blocks of nacc * nn
    int split;              // pairs of a cluster = parts of K
    int a, b, raw;          // ring depths: weight tiles, token tiles, raw super-block columns
    size_t smem;
};

// what the kernel computes: (ONE) f32[0][m][n] = acc (+ resid[m][n]) (+ bias[n]), (GROUP) f32[t][m][n] = acc for two or three weights of one
// type that share the tokens, or (DUAL) bf16[m][n] = silu(gate) * up.  A kernel of its own for the group: with the choice of a weight in every
// launch each thread first copies these arguments to local memory and the epilogue spills (48 products 936 x 256 Q4_K of 82 tokens, each with
// its conversion: 543 us, without 422)
enum { TC_ONE, TC_DUAL, TC_GROUP };
struct tc_out {
    const float *bias;
    const float *resid;     // added to the product, laid out like f32 and possibly the same memory
    float *f32[3];
    __nv_bfloat16 *bf16;
    int n[3];               // features of each
    int64_t ld;             // those of the first once more: 64 bits that ONE need not keep in registers
    int t1, t2;             // first tile of the second and of the third
};

template <int TYPE, int KIND>
__global__ void __launch_bounds__(TC_THREADS, 1)
skn_matmul_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_w2,
                     const __grid_constant__ CUtensorMap tm_w3, int M, int K, const tc_plan pl, const tc_out out, int32_t *__restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    // operand tiles need 1024-byte alignment for the 128-byte swizzle; the offset is the same in every CTA
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int ROW = TcFmt<TYPE>::ROW, RAW_BYTES = TC_ROWS * ROW;
    constexpr bool DUAL = KIND == TC_DUAL, GROUP = KIND == TC_GROUP;
    __shared__ uint64_t a_full[TC_MAX_A], a_empty[TC_MAX_A], b_full[TC_MAX_B], b_empty[TC_MAX_B], raw_full[TC_MAX_RAW], raw_empty[TC_MAX_RAW], accum_bar;
    __shared__ uint32_t tmem_slot;

    // (through a shuffle: the compiler then knows that a warp's threads take one role together)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = (int)tc_cluster_rank(), half = rank & 1, kr = rank >> 1, c = pl.split;
    const int tile = (int)blockIdx.x / (2 * c), m0 = (int)blockIdx.y * (pl.nacc * pl.nn);
    const int na = pl.a, nb = pl.b, nraw = pl.raw;
    const int b_acc = (pl.nn >> 1) * (TC_BK * 2), b_bytes = pl.nacc * b_acc;
    uint8_t *b_ring = smem + (size_t)na * TC_A_BYTES, *raw_ring = b_ring + (size_t)nb * b_bytes;
    // this pair's part of K in super-blocks of 256 (the last one may be short), and in stages
    const int nsb = (K + 255) / 256, sb0 = kr * nsb / c, sb1 = (kr + 1) * nsb / c;
    const int steps = min(K / TC_BK, sb1 * 4) - sb0 * 4;
    // features of this CTA: DUAL interleaves 16 gate and 16 up rows (lanes 0-15 and 16-31 of a warp)
    const bool w1 = GROUP && tile >= out.t1, w2 = GROUP && tile >= out.t2;
    const int N = w2 ? out.n[2] : w1 ? out.n[1] : out.n[0];
    const int n0 = DUAL ? tile * TC_ROWS + half * (TC_ROWS / 2) : (tile - (w2 ? out.t2 : w1 ? out.t1 : 0)) * 2 * TC_ROWS + half * TC_ROWS;
    const uint32_t tmem_cols = pl.nacc == 2 ? 512u : 256u;
    const uint16_t pair_mask = (uint16_t)(3u << (rank & ~1));

    if (threadIdx.x == 0) {
        for (int s = 0; s < na; ++s) {
            skn_mbar_init(&a_full[s], half ? 4 : 4 + 1);  // a group of warps; leader: and the other CTA's pass-on
            skn_mbar_init(&a_empty[s], 1);                // one tcgen05.commit
        }
        for (int s = 0; s < nb; ++s) {
            skn_mbar_init(&b_full[s], 1);                 // leader only: both halves' bytes
            skn_mbar_init(&b_empty[s], 1);
        }
        skn_mbar_init(&accum_bar, 1);
        skn_fence_mbar_init();
    }
    // raw weights of super-block sb into ring place rs: rows past N and bytes past a row arrive as zeros
    auto load_raw = [&](int sb, int rs) {
        uint8_t *dst = raw_ring + (size_t)rs * RAW_BYTES;
        skn_mbar_expect_tx(&raw_full[rs], RAW_BYTES);
        const int x = tc_box_x<TYPE>(sb);
        if (DUAL) {
            for (int i = 0; i < 4; ++i) {
                tc_tma_load_2d(dst + 32 * i * ROW, &tm_w, x, n0 + 16 * i, &raw_full[rs]);
                tc_tma_load_2d(dst + (32 * i + 16) * ROW, &tm_w2, x, n0 + 16 * i, &raw_full[rs]);
            }
        } else {
            tc_tma_load_2d(dst, w2 ? &tm_w3 : w1 ? &tm_w2 : &tm_w, x, n0, &raw_full[rs]);
        }
    };
    const int early = min(nraw, sb1 - sb0);
    if (warp == TC_TMA_W && lane == 0) {
        // the weights depend on no launch before this one: the first ring-full is requested at once
        for (int s = 0; s < nraw; ++s) {
            skn_mbar_init(&raw_full[s], 1);
            skn_mbar_init(&raw_empty[s], TC_DQ_WARPS);
        }
        skn_fence_mbar_init();
        skn_fence_proxy_async();
        for (int i = 0; i < early; ++i) load_raw(sb0 + i, i);
    }
    if (warp == TC_MMA) tc2_alloc(&tmem_slot, tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;

    bool failed = false;
    auto give_up = [&]() {
        failed = true;
        atomicExch(status, SKN_ERR_TIMEOUT);
    };
    if (warp & 3) {
        // ---------------- weights: raw ring -> operand tile; group `turn` takes the stages 3 i + turn ----------------
        const int dq = (warp >> 2) * 3 + (warp & 3) - 1, turn = dq >> 2, r = (dq & 3) * 32 + lane;
        const uint32_t raw0 = skn_smem_u32(raw_ring) + (uint32_t)(r * ROW);
        int s = turn % na, rs = 0, have = -1;
        uint32_t ph = (uint32_t)(turn / na), rph = 0;
#pragma unroll 1
        for (int it = turn; it < steps; it += TC_DQ_GROUPS) {
            if (it >> 2 != have) {                         // the next super-block (it has more stages than lie between two turns)
                if (have >= 0) {
                    __syncwarp();
                    if (lane == 0) skn_mbar_arrive(&raw_empty[rs]);
                    if (++rs == nraw) { rs = 0; rph ^= 1u; }
                }
                have = it >> 2;
                if (!failed && !tc_wait_warp(&raw_full[rs], rph, lane)) give_up();
            }
            const uint32_t row = raw0 + (uint32_t)(rs * RAW_BYTES);
            const int u = it & 3, lead = TYPE == SKN_TYPE_Q6_K ? ((sb0 + have) * 210) & 15 : 0;
            uint8_t *tile_a = smem + (size_t)s * TC_A_BYTES;
            const TcStage<TYPE> st(row, u, lead);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                uint32_t p[16];
                st.half(row, u, g, lead, p);
                if (g == 0 && !failed && !tc_wait_warp(&a_empty[s], ph ^ 1u, lane)) give_up();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int chunk = TYPE == SKN_TYPE_Q4_K ? 4 * (i >> 1) + 2 * g + (i & 1) : 4 * g + i;
                    tc_store_chunk(tile_a, r, chunk, make_uint4(p[4 * i], p[4 * i + 1], p[4 * i + 2], p[4 * i + 3]));
                }
            }
            skn_fence_proxy_async();     // generic-proxy stores -> visible to the tensor core's async proxy
            __syncwarp();
            if (lane == 0) skn_mbar_arrive(&a_full[s]);
            for (s += TC_DQ_GROUPS; s >= na; s -= na) ph ^= 1u;
        }
    } else if (warp == TC_TMA_W) {
        // ---------------- raw weights: one thread, TMA ----------------
        if (lane == 0) {
            int rs = 0;
            uint32_t rph = 0;
            for (int sb = sb0 + early; sb < sb1; ++sb) {
                if (!failed && !skn_mbar_wait(&raw_empty[rs], rph)) give_up();
                skn_fence_proxy_async();
                load_raw(sb, rs);
                if (++rs == nraw) { rs = 0; rph ^= 1u; }
            }
        }
    } else if (warp == TC_TMA_X) {
        // ---------------- activations: one thread, TMA; this CTA's half of every accumulator's tokens ----------------
        if (lane == 0) {
            skn_pdl_wait();                                    // they are the previous launch's output
            int s = 0;
            uint32_t ph = 0;
            for (int it = 0; it < steps; ++it) {
                if (!failed && !skn_mbar_wait(&b_empty[s], ph ^ 1u)) give_up();
                uint8_t *dst = b_ring + (size_t)s * b_bytes;
                const uint32_t bar = tc_mapa(skn_smem_u32(&b_full[s]), (uint32_t)(rank & ~1));
                if (!half) skn_mbar_expect_tx(&b_full[s], 2u * (uint32_t)b_bytes);
                for (int a = 0; a < pl.nacc; ++a)              // tokens beyond M arrive as zeros
                    tc2_tma_load_2d(dst + a * b_acc, &tm_x, (sb0 * 4 + it) * TC_BK, m0 + a * pl.nn + half * (pl.nn >> 1), bar);
                if (++s == nb) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == TC_MMA && half) {
        // ---------------- pass on to the leader: this CTA's weights are in place ----------------
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            for (int it = 0; it < steps; ++it) {
                if (!failed && !skn_mbar_wait(&a_full[s], ph)) give_up();
                tc_arrive_remote(tc_mapa(skn_smem_u32(&a_full[s]), (uint32_t)(rank & ~1)));
                if (++s == na) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp == TC_MMA) {
        // ---------------- MMA issuer of the pair: 256 features x nn tokens per accumulator ----------------
        const uint32_t idesc = tc_idesc(2 * TC_ROWS, pl.nn);
        const uint64_t a0 = tc_smem_desc(skn_smem_u32(smem)), b0 = tc_smem_desc(skn_smem_u32(b_ring));
        const int b_step = b_bytes >> 4, acc_step = b_acc >> 4;    // address fields count 16 bytes
        int s = 0, t = 0;
        uint32_t ph = 0, pt = 0;
        for (int it = 0; it < steps; ++it) {
            if (!failed && !tc_wait_warp(&b_full[t], pt, &a_full[s], ph, lane)) failed = true;      // (one answer for the warp: its lanes elect, and fail, together)
            tc_fence_after();
            const uint64_t ad = a0 + (uint64_t)(s * (TC_A_BYTES >> 4)), bd = b0 + (uint64_t)(t * b_step);
            if (tc_elect()) {
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k) {
                    const uint32_t acc = (it > 0 || k > 0) ? 1u : 0u;
                    // advancing 16 bf16 (32 bytes) along K inside the swizzle atom = +2 in the address field
                    tc2_mma_bf16(tmem_base, ad + 2 * k, bd + 2 * k, idesc, acc);
                    if (pl.nacc == 2) tc2_mma_bf16(tmem_base + 256, ad + 2 * k, bd + acc_step + 2 * k, idesc, acc);
                }
                tc2_commit(&a_empty[s], pair_mask);            // frees the tiles in both CTAs once these MMAs have read them
                tc2_commit(&b_empty[t], pair_mask);
            }
            if (++s == na) { s = 0; ph ^= 1u; }
            if (++t == nb) { t = 0; pt ^= 1u; }
        }
        if (tc_elect()) {
            tc2_commit(&accum_bar, pair_mask);                 // all MMAs done: the accumulators are complete
            if (failed) atomicExch(status, SKN_ERR_TIMEOUT);
        }
    }
    __syncwarp();

    // ---------------- epilogue: TMEM lane = feature, blocks of 32 tokens ----------------
    const int nblk = pl.nacc * pl.nn / TC_BLOCK, wq = warp & 3, wb = warp >> 2;
    const int own0 = kr * nblk / c, own1 = (kr + 1) * nblk / c, slot_blk = (nblk + c - 1) / c;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(wq * 32) << 16);
    auto block_addr = [&](int b) { return lane_addr + (uint32_t)((b * TC_BLOCK / pl.nn) * 256 + b * TC_BLOCK % pl.nn); };
    skn_pdl_wait();                                            // the outputs may still be read by earlier launches
    const bool ok = tc_wait_warp(&accum_bar, 0u, lane);
    if (!ok) atomicExch(status, SKN_ERR_TIMEOUT);
    tc_fence_after();
    skn_pdl_launch_dependents();                               // the next launch may start and fetch its weights
    if (c > 1) {
        // all pairs of the cluster are done with their rings: the memory takes partial sums [slot][token][feature] now
        tc_cluster_sync();
        // [slot][token][feature]: a warp's store is 128 bytes in a row (16 bytes per lane of its own row ran at half the rate)
        const uint32_t mine = skn_smem_u32(smem) + (uint32_t)(wq * 32 + lane) * 4u;
        for (int j = 0; j < c; ++j) {
            if (j == kr) continue;
            const int f0 = j * nblk / c, f1 = (j + 1) * nblk / c, slot = kr < j ? kr : kr - 1;
            const uint32_t to = tc_mapa(mine + (uint32_t)(slot * slot_blk) * TC_BLOCK_BYTES, (uint32_t)(2 * j + half));
            for (int b = f0 + wb; b < f1; b += TC_WARPS / 4) {
                uint32_t acc[32];
                tc_ld32(block_addr(b), acc);
#pragma unroll
                for (int i = 0; i < TC_BLOCK; ++i)
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to + (uint32_t)(b - f0) * TC_BLOCK_BYTES + (uint32_t)(i * TC_ROWS * 4)), "r"(acc[i]) : "memory");
            }
        }
        tc_cluster_sync();
    }
    if (ok) {
        const float *slots = reinterpret_cast<const float *>(smem) + wq * 32 + lane;
        for (int b = own0 + wb; b < own1; b += TC_WARPS / 4) {
            uint32_t acc[32];
            tc_ld32(block_addr(b), acc);
            if (c > 1) {
                float sum[32];
#pragma unroll 1
                for (int j = 0; j < c; ++j) {                  // in the order of K, whoever adds
                    const float *from = slots + (size_t)((j < kr ? j : j - 1) * slot_blk + (b - own0)) * (TC_BLOCK * TC_ROWS);
#pragma unroll
                    for (int i = 0; i < TC_BLOCK; ++i) {
                        const float v = j == kr ? __uint_as_float(acc[i]) : from[i * TC_ROWS];
                        sum[i] = j == 0 ? v : sum[i] + v;
                    }
                }
#pragma unroll
                for (int i = 0; i < TC_BLOCK; ++i) acc[i] = __float_as_uint(sum[i]);
            }
            const int m = m0 + b * TC_BLOCK;
            if (DUAL) {
                // lane l holds gate (l < 16) or up of feature l & 15; the halves trade tokens so that each forms one
                // product per pair of tokens, then neighbours trade so that each stores two features at once
                const int f = n0 + 16 * wq + (lane & 14);
                const bool low = lane < 16, even = (lane & 1) == 0;
#pragma unroll
                for (int i = 0; i < TC_BLOCK; i += 4) {
                    float h[2];
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const uint32_t v0 = acc[i + 2 * p], v1 = acc[i + 2 * p + 1];
                        const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, low ? v1 : v0, 16));
                        const float gate = low ? __uint_as_float(v0) : got, up = low ? got : __uint_as_float(v1);
                        h[p] = gate / (1.f + __expf(-gate)) * up;
                    }
                    const float got = __shfl_xor_sync(0xffffffffu, even ? h[1] : h[0], 1);
                    const uint32_t two = even ? tc_pack_bf16(h[0], got) : tc_pack_bf16(got, h[1]);
                    const int tok = m + i + (even ? 0 : 2) + (low ? 0 : 1);
                    if (tok < M && f < N) *reinterpret_cast<uint32_t *>(out.bf16 + (int64_t)tok * N + f) = two;   // N is a multiple of 8
                }
            } else {
                const int f = n0 + wq * 32 + lane;
                const int64_t ld = GROUP ? N : out.ld;
                if (f < N) {
                    const float bias = !GROUP && out.bias ? __ldg(out.bias + f) : 0.f;
                    float *dst = (w2 ? out.f32[2] : w1 ? out.f32[1] : out.f32[0]) + m * ld + f;
                    if (!GROUP && out.resid) {                           // (all loads before the first store)
                        const float *res = out.resid + m * ld + f;
#pragma unroll
                        for (int i = 0; i < TC_BLOCK; ++i)
                            if (m + i < M) acc[i] = __float_as_uint(__uint_as_float(acc[i]) + res[i * ld]);
                    }
#pragma unroll
                    for (int i = 0; i < TC_BLOCK; ++i)
                        if (m + i < M) dst[i * ld] = __uint_as_float(acc[i]) + bias;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_cluster_sync();                   // no CTA leaves while another one reads its memory or arrives on its barriers
    if (warp == TC_MMA) {
        tc_fence_after();
        tc2_dealloc(tmem_base, tmem_cols);
    }
}

// ---- launch ------------------------------------------------------------------------------------------------
static int tc_row_bytes(int type) {
    return type == SKN_TYPE_Q8_0 ? TcFmt<SKN_TYPE_Q8_0>::ROW : (type == SKN_TYPE_Q6_K ? TcFmt<SKN_TYPE_Q6_K>::ROW : TcFmt<SKN_TYPE_Q4_K>::ROW);
}

// Tokens in equal blocks of at most 512 or 256, each over one or two accumulators of a multiple of 32 columns; K over
// as many pairs of a cluster as make the launch shortest.  The estimate is in SM clocks, from a timeline of the kernel: a
// stage costs the longer of its MMAs (two clocks per token) and its dequantisation (tc_stage_clocks), the start takes
// 6000, the epilogue stores 20 bytes per clock, the exchange of partial sums moves 17 and costs another 6000 of waiting
// for one another.  Measured: 4096 x 14336 at 512 tokens as 3 parts of K over 48 pairs 73 us (Q4_K) and 75 (Q6_K), as 2
// parts of K x 2 blocks of 256 tokens over 64 pairs 67 and 83 us.  `pairs[s]` = clusters of s pairs that fit on the GPU, times s.
static int tc_stage_clocks(int type) { return type == SKN_TYPE_Q6_K ? 970 : (type == SKN_TYPE_Q8_0 ? 800 : 710); }
static tc_plan tc_make_plan(int type, int M, int64_t tiles, int K, const int *pairs) {
    const int raw_bytes = TC_ROWS * tc_row_bytes(type), nsb = (K + 255) / 256;
    tc_plan best = {};
    int64_t best_cost = 0;
    for (int most = TC_MAX_TOKENS; most >= 256; most /= 2) {
        tc_plan pl = {};
        pl.blocks = (M + most - 1) / most;
        const int tok = (M + pl.blocks - 1) / pl.blocks;
        pl.nacc = tok > 256 ? 2 : 1;
        pl.nn = ((tok + pl.nacc - 1) / pl.nacc + 31) / 32 * 32;
        pl.blocks = (M + pl.nacc * pl.nn - 1) / (pl.nacc * pl.nn);
        const int cols = pl.nacc * pl.nn, nblk = cols / TC_BLOCK, b_bytes = (cols / 2) * TC_BK * 2;
        // ring depths: the tokens' tiles are what has to be on its way early (a round trip to L2 and through the pair's
        // barriers takes two to three stages), then the weights', then the raw blocks.  A weight tile per dequantising group
        // at least: a group that runs ahead could not tell by a phase's parity whether its tile is one or three uses behind.
        pl.a = TC_DQ_GROUPS;
        pl.b = pl.raw = 2;
        auto fits = [&](int a, int b, int raw) { return a * TC_A_BYTES + b * b_bytes + raw * raw_bytes <= TC_SMEM_MAX - 1024; };
        for (bool grown = true; grown;) {
            grown = false;
            if (pl.b < TC_MAX_B && pl.b <= pl.a && fits(pl.a, pl.b + 1, pl.raw)) { ++pl.b; grown = true; }
            if (pl.a < TC_MAX_A && fits(pl.a + 1, pl.b, pl.raw)) { ++pl.a; grown = true; }
            if (pl.raw < TC_MAX_RAW && pl.a >= 3 && fits(pl.a, pl.b, pl.raw + 1)) { ++pl.raw; grown = true; }
            if (pl.a == TC_MAX_A && pl.b < TC_MAX_B && fits(pl.a, pl.b + 1, pl.raw)) { ++pl.b; grown = true; }
        }
        const size_t rings = (size_t)pl.a * TC_A_BYTES + (size_t)pl.b * b_bytes + (size_t)pl.raw * raw_bytes;
        const int64_t step = 2 * cols > tc_stage_clocks(type) ? 2 * cols : tc_stage_clocks(type), bytes = (int64_t)cols * TC_ROWS * 4;
        for (int c = 1; c <= TC_MAX_SPLIT && c <= nsb; ++c) {
            if (pairs[c] < 1 && c > 1) continue;
            const int64_t units = tiles * pl.blocks * c, fit = pairs[c] > 0 ? pairs[c] : 1, waves = (units + fit - 1) / fit;
            int64_t cost = 6000 + (int64_t)((nsb + c - 1) / c * 4) * step + bytes / c / 20;
            if (c > 1) cost += 6000 + bytes * (c - 1) / c / 17;
            cost *= waves;
            if (best_cost && cost >= best_cost) continue;
            best_cost = cost;
            best = pl;
            best.split = c;
            const size_t exchange = (size_t)(c - 1) * ((nblk + c - 1) / c) * TC_BLOCK_BYTES;
            best.smem = (rings > exchange ? rings : exchange) + 1024;
        }
        if (M <= 256) break;
    }
    return best;
}

static cudaLaunchConfig_t tc_config(dim3 grid, int split, size_t smem, cudaStream_t stream, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

// Pairs in flight when clusters hold 1 .. TC_MAX_SPLIT of them.  Asked of the driver once per device, of whichever kernel comes first: threads,
// shared memory and one CTA per SM are the same for all of them (asked of each, the first call of each took 5 to 15 us longer on the host).
static cudaError_t tc_pairs(int dev, const void *kern, cudaStream_t stream, int (&pairs)[TC_MAX_SPLIT + 1]) {
    static std::atomic<int> fits[64][TC_MAX_SPLIT + 1];            // 0: not asked yet, -1: none
    std::atomic<int> *fit = fits[dev & 63];
    for (int s = TC_MAX_SPLIT; s >= 1; --s) {
        pairs[s] = fit[s].load(std::memory_order_relaxed);
        if (pairs[s]) continue;
        cudaLaunchAttribute attr[2];
        const cudaLaunchConfig_t cfg = tc_config(dim3(2 * s), s, TC_SMEM_MAX, stream, attr);
        int n = 0;
        const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
        if (e != cudaSuccess) return e;
        pairs[s] = n > 0 ? n * s : -1;
        fit[s].store(pairs[s], std::memory_order_relaxed);
    }
    return cudaSuccess;
}

template <int TYPE, int KIND>
static cudaError_t launch_tc(const __nv_bfloat16 *A, int M, int K, int n, const skn_tensor *const *w, tc_out out, int32_t *status, cudaStream_t stream) {
    constexpr bool DUAL = KIND == TC_DUAL;
    auto kern = skn_matmul_tc_kernel<TYPE, KIND>;
    static std::atomic<bool> large[64];                            // per device: may use TC_SMEM_MAX
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[2];
    if (!large[dev & 63].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_MAX);
        if (e != cudaSuccess) return e;
        large[dev & 63].store(true, std::memory_order_release);
    }
    int pairs[TC_MAX_SPLIT + 1] = {0};
    if ((e = tc_pairs(dev, (const void *)kern, stream, pairs)) != cudaSuccess) return e;
    int64_t tiles = 0;
    out.t1 = out.t2 = 0x7fffffff;
    out.ld = w[0]->n_rows;
    for (int t = 0; t < (DUAL ? 1 : n); ++t) {
        if (t == 1) out.t1 = (int)tiles;
        if (t == 2) out.t2 = (int)tiles;
        out.n[t] = (int)w[t]->n_rows;
        tiles += DUAL ? (w[t]->n_rows + TC_ROWS - 1) / TC_ROWS : (w[t]->n_rows + 2 * TC_ROWS - 1) / (2 * TC_ROWS);
    }
    const tc_plan pl = tc_make_plan(TYPE, M, tiles, K, pairs);
    CUtensorMap tx, tw[3];
    if ((e = skn_tmap_bf16(A, M, K, (int64_t)K * 2, pl.nn / 2, &tx)) != cudaSuccess) return e;
    for (int t = 0; t < n; ++t)
        if ((e = skn_tmap_blocks(w[t], TcFmt<TYPE>::ROW, DUAL ? 16 : TC_ROWS, &tw[t])) != cudaSuccess) return e;
    for (int t = n; t < 3; ++t) tw[t] = tw[0];
    const cudaLaunchConfig_t cfg = tc_config(dim3((unsigned)(tiles * 2 * pl.split), (unsigned)pl.blocks), pl.split, pl.smem, stream, attr);
    return cudaLaunchKernelEx(&cfg, kern, tx, tw[0], tw[1], tw[2], M, K, pl, out, status);
}

template <int KIND>
static cudaError_t dispatch_tc(const __nv_bfloat16 *A, int M, int n, const skn_tensor *const *w, const tc_out &out, int32_t *status, cudaStream_t stream) {
    const int K = (int)w[0]->n_cols;
    switch (w[0]->type) {
    case SKN_TYPE_Q4_0: return launch_tc<SKN_TYPE_Q4_0, KIND>(A, M, K, n, w, out, status, stream);
    case SKN_TYPE_Q8_0: return launch_tc<SKN_TYPE_Q8_0, KIND>(A, M, K, n, w, out, status, stream);
    case SKN_TYPE_Q4_K: return launch_tc<SKN_TYPE_Q4_K, KIND>(A, M, K, n, w, out, status, stream);
    case SKN_TYPE_Q6_K: return launch_tc<SKN_TYPE_Q6_K, KIND>(A, M, K, n, w, out, status, stream);
    default: return cudaErrorInvalidValue;
    }
}

// (the tensor map's base: 16 bytes)
bool skn_tc_supported(const skn_tensor *w, int32_t M) {
    const bool type_ok = w->type == SKN_TYPE_Q4_0 || w->type == SKN_TYPE_Q8_0 || w->type == SKN_TYPE_Q4_K || w->type == SKN_TYPE_Q6_K;
    return type_ok && M >= 1 && (w->n_cols % TC_BK) == 0 && w->n_cols >= TC_BK && (w->n_rows % 8) == 0 && (w->pitch % 16) == 0 &&
           (reinterpret_cast<uintptr_t>(w->d_blocks) & 15) == 0;
}

cudaError_t skn_launch_f32_to_bf16(const float *in, void *out_bf16, int64_t n, int sm_count, cudaStream_t stream) {
    const int64_t n4 = n / 4;
    if (n4 == 0) return cudaSuccess;
    int64_t blocks = (n4 + 255) / 256;
    if (blocks > (int64_t)sm_count * 8) blocks = (int64_t)sm_count * 8;
    skn_f32_to_bf16_kernel<<<(unsigned)blocks, 256, 0, stream>>>(in, (__nv_bfloat16 *)out_bf16, n4);
    return cudaGetLastError();
}

// Y = A_bf16 . W^T (+bias) (+resid), fp32 out
cudaError_t skn_launch_matmul_tc(skn_ctx *ctx, const skn_tensor *w, const void *a_bf16, int32_t M, const float *bias,
                                 float *y, cudaStream_t stream, const float *resid) {
    tc_out out = {};
    out.bias = bias; out.resid = resid; out.f32[0] = y;
    return dispatch_tc<TC_ONE>((const __nv_bfloat16 *)a_bf16, M, 1, &w, out, ctx->d_status, stream);
}

// Y[t] = A_bf16 . W[t]^T for two or three weights of one type and width in one launch: the key and value projections of a model with grouped
// heads have too few tiles for a launch of their own (512 tokens, 4096 x 4096 and twice 1024 x 4096 Q4_K: 74 us in three launches, 44 in one)
cudaError_t skn_launch_matmul_tc_group(skn_ctx *ctx, int n, const skn_tensor *const *w, const void *a_bf16, int32_t M, float *const *y, cudaStream_t stream) {
    if (n < 2 || n > 3) return cudaErrorInvalidValue;
    tc_out out = {};
    for (int t = 0; t < n; ++t) {
        if (w[t]->type != w[0]->type || w[t]->n_cols != w[0]->n_cols) return cudaErrorInvalidValue;
        out.f32[t] = y[t];
    }
    return dispatch_tc<TC_GROUP>((const __nv_bfloat16 *)a_bf16, M, n, w, out, ctx->d_status, stream);
}

// H_bf16 = silu(A . Wg^T) * (A . Wu^T)
cudaError_t skn_launch_gate_up_tc(skn_ctx *ctx, const skn_tensor *wg, const skn_tensor *wu, const void *a_bf16,
                                  int32_t M, void *h_bf16, cudaStream_t stream) {
    const skn_tensor *w[2] = {wg, wu};
    tc_out out = {};
    out.bf16 = (__nv_bfloat16 *)h_bf16;
    return dispatch_tc<TC_DUAL>((const __nv_bfloat16 *)a_bf16, M, 2, w, out, ctx->d_status, stream);
}
