// Causal attention of a prompt's queries over the ring cache (fp32, fp16 or Q8_0 rows), on the warp-level tensor cores in the
// accuracy of the fp32 kernels of skn_kv.cu.
//
// Every fp32 operand (queries, keys, probabilities, values) from 2^-110 up to the last 0.4 % of the range is the exact sum of three bf16 numbers
// a + b + c, and a product is the six of nine partial products that reach its 24 bits: ac + ca + bb, ab + ba, aa.  (Below, c loses its bits
// under 2^-133.  Above, and where an operand is not finite, a tile of keys is computed in plain fp32: one that holds such a key or value, and
// all of a CTA that holds such a query.)  A chain of the six runs from zero for each 16 elements of a
// reduction and its result is added in an fp32 register: the tensor cores chop what they add to an accumulator, a sum that stayed there
// would drift.  Probabilities, maxima, sums and outputs are fp32 as before; the error against 64 bits is not larger
// (tests/test_gpu_attn_prompt.py).
//
// A CTA takes 64 (query, head) rows of one kv head -- 64 / G queries, so the heads of a group share every key -- and walks the keys in
// tiles of 32: the even tiles by one group of four warps, the odd ones by another (a warp owns 16 rows), each with planes, maxima, sums and
// outputs of its own that meet at the end.  One group per CTA and two CTAs per SM left the longest rows, which have an SM to themselves
// for most of the time, twice as long.  A group's next tile is on its way into registers while this one is multiplied.
// CTAs with the most keys start first.
//
// 512 tokens, 32 heads of 128 over 8 kv heads, launches back to back: 194 to 219 us with the fp32 split kernels and their merge, 72 here;
// 16 sequences of 20 tokens 36 and 20, 128 tokens of 4 sequences after 384 others 262 and 118.  The products alone would take 23 (m16n8k16: 8 clocks of a scheduler, 96 of
// them for 16 rows x 8 keys); the tensor pipe is busy a third of the time, the rest is the latency of conversions, exponentials and
// fragment loads at two warps per scheduler.
#include "skn_internal.cuh"
#include "skn_mma.cuh"

#include <math.h>

constexpr int AP_ROWS = 64, AP_KEYS = 32, AP_RUN = 256, AP_GROUP = 128;

// four consecutive elements of a cached row
template <int DT> struct ApRow;
template <> struct ApRow<SKN_KV_F32> {
    typedef float elem;
    static __device__ __forceinline__ float4 ld(const float *p, const __half *) { return __ldg(reinterpret_cast<const float4 *>(p)); }
};
template <> struct ApRow<SKN_KV_F16> {
    typedef __half elem;
    static __device__ __forceinline__ float4 ld(const __half *p, const __half *) {
        const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
};
template <> struct ApRow<SKN_KV_Q8_0> {
    typedef int8_t elem;
    static __device__ __forceinline__ float4 ld(const int8_t *p, const __half *scale) {
        const uint32_t u = __ldg(reinterpret_cast<const uint32_t *>(p));
        const float s = __half2float(__ldg(scale));
        return make_float4((float)(int8_t)(u & 255u) * s, (float)(int8_t)((u >> 8) & 255u) * s, (float)(int8_t)((u >> 16) & 255u) * s,
                           (float)(int8_t)(u >> 24) * s);
    }
};

// one (sequence, kv head) of a cache plane; Q8_0: the scales follow the quants of all rows
template <int DT, int D> struct ApHead {
    typedef typename ApRow<DT>::elem E;
    const E *rows;
    const __half *scales;
    int s0, cap;
    __device__ __forceinline__ ApHead(const void *plane, size_t all_rows, size_t row0, int start, int cap_) : s0(start), cap(cap_) {
        rows = static_cast<const E *>(plane) + row0 * D;
        scales = DT == SKN_KV_Q8_0 ? reinterpret_cast<const __half *>(static_cast<const int8_t *>(plane) + all_rows * D) + row0 * (D / 32) : nullptr;
    }
    // elements d .. d + 3 of token j
    __device__ __forceinline__ float4 ld(int j, int d) const {
        int slot = s0 + j;
        if (slot >= cap) slot -= cap;
        return ApRow<DT>::ld(rows + (size_t)slot * D + d, DT == SKN_KV_Q8_0 ? scales + (size_t)slot * (D / 32) + (d >> 5) : nullptr);
    }
};

// v -> its bf16 terms, at the same place of NP planes; `last` adds up the last ones: a number that is not a sum of finite terms (infinities, NaN,
// the last 0.4 % of fp32) leaves NaN there
template <int NP>
__device__ __forceinline__ void ap_split_store(uint8_t *at, int plane_bytes, float4 v, __nv_bfloat162 &last) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const uint2 w = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
        *reinterpret_cast<uint2 *>(at + p * plane_bytes) = w;
        if (p < NP - 1) {
            less_bf16(v.x, v.y, w.x);
            less_bf16(v.z, v.w, w.y);
        } else {
            last = __hadd2(last, *reinterpret_cast<const __nv_bfloat162 *>(&w.x));
            last = __hadd2(last, *reinterpret_cast<const __nv_bfloat162 *>(&w.y));
        }
    }
}

__device__ __forceinline__ bool ap_finite(__nv_bfloat162 x) { return fabsf(__low2float(x)) < INFINITY && fabsf(__high2float(x)) < INFINITY; }

// barriers of one group
__device__ __forceinline__ void ap_sync(int group) { asm volatile("barrier.sync %0, %1;" ::"r"(group + 1), "n"(AP_GROUP) : "memory"); }
__device__ __forceinline__ bool ap_sync_or(int group, bool x) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"((uint32_t)x), "r"(group + 1), "n"(AP_GROUP) : "memory");
    return any != 0;
}

struct ap_args {
    const float *q;
    const void *k, *v;
    const int32_t *len, *start;
    float *out;
    __nv_bfloat16 *out16;                       // instead of out, or NULL
    int Hkv, G, cap, T, len_extra, B;
    float scale;
};

template <int D, int DT, int GROUPS>
__global__ void __launch_bounds__(GROUPS * AP_GROUP, 3 - GROUPS)
skn_attn_prompt_kernel(const ap_args a) {
    extern __shared__ __align__(16) uint8_t smb[];
    constexpr int LD = (D + 8) * 2;                                     // bytes of a row: eight rows meet all banks
    constexpr int QP = AP_ROWS * LD, KP = AP_KEYS * LD;                 // a plane
    constexpr int NP = DT == SKN_KV_F16 ? 2 : 3;                        // terms of a key or value
    constexpr int NLD = AP_KEYS * (D / 4) / AP_GROUP;                   // float4 per thread, tile and tensor
    const int group = threadIdx.x / AP_GROUP, tid = threadIdx.x % AP_GROUP, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    uint8_t *Q = smb, *K = Q + 3 * QP + group * 6 * KP, *V = K + 3 * KP;
    const int heads = a.Hkv * a.B, item = (int)blockIdx.x, kvh = item % a.Hkv, b = item % heads / a.Hkv;
    const int row0 = ((int)gridDim.x / heads - 1 - item / heads) * AP_ROWS;        // (the longest first)
    const int len = __ldg(a.len + b) + a.len_extra, s0 = __ldg(a.start + b);
    const int G = a.G, Hq = a.Hkv * G, nrows = min(AP_ROWS, a.T * G - row0);
    const ApHead<DT, D> kr(a.k, (size_t)a.B * a.Hkv * a.cap, ((size_t)b * a.Hkv + kvh) * a.cap, s0, a.cap),
        vr(a.v, (size_t)a.B * a.Hkv * a.cap, ((size_t)b * a.Hkv + kvh) * a.cap, s0, a.cap);
    // keys that the query of row r sees, and where its q and output are
    auto seen = [&](int r) { return min(a.cap, max(0, len - (a.T - 1 - (row0 + r) / G))); };
    auto at = [&](int r) { return (((size_t)b * a.T + (row0 + r) / G) * Hq + kvh * G + (row0 + r) % G) * D; };
    const int nk = seen(nrows - 1), tiles = (nk + AP_KEYS - 1) / AP_KEYS;

    auto query = [&](int r, int d) {
        float4 x = __ldg(reinterpret_cast<const float4 *>(a.q + at(r) + d));
        x.x *= a.scale; x.y *= a.scale; x.z *= a.scale; x.w *= a.scale;
        return x;
    };
    __nv_bfloat162 qlast = __floats2bfloat162_rn(0.f, 0.f);
    // (asked for in fours; not beside fp16 rows of 64, whose tile loop then comes out slower: 256 tokens over 2048, 124 us this way, 129 in fours)
    if constexpr (D == 64 && DT == SKN_KV_F16) {
        for (int i = threadIdx.x; i < AP_ROWS * (D / 4); i += GROUPS * AP_GROUP) {
            const int r = i / (D / 4), d = i % (D / 4) * 4;
            ap_split_store<3>(Q + r * LD + d * 2, QP, r < nrows ? query(r, d) : make_float4(0.f, 0.f, 0.f, 0.f), qlast);
        }
    } else {
#pragma unroll
        for (int i0 = 0; i0 < AP_ROWS * (D / 4) / (GROUPS * AP_GROUP); i0 += 4) {
            float4 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = (i0 + i) * GROUPS * AP_GROUP + threadIdx.x, r = at / (D / 4);
                x[i] = r < nrows ? query(r, at % (D / 4) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = (i0 + i) * GROUPS * AP_GROUP + threadIdx.x;
                ap_split_store<3>(Q + at / (D / 4) * LD + at % (D / 4) * 8, QP, x[i], qlast);
            }
        }
    }
    float4 rk[NLD], rv[NLD];
    auto fetch = [&](int t) {
#pragma unroll
        for (int i = 0; i < NLD; ++i) {
            const int j = t * AP_KEYS + (i * AP_GROUP + tid) / (D / 4), d = tid % (D / 4) * 4;
            rk[i] = rv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j < nk) {
                rk[i] = kr.ld(j, d);
                rv[i] = vr.ld(j, d);
            }
        }
    };
    if (group < tiles) fetch(group);
    // the queries are in place; where one of them has no three finite terms, all tiles are computed in plain fp32
    const bool qplain = __syncthreads_or(!ap_finite(qlast)) != 0;

    float o[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float mrow[2] = {-INFINITY, -INFINITY}, lrow[2] = {0.f, 0.f};
    const int ra = warp * 16 + (lane >> 2);                             // this lane's rows: ra, ra + 8
    const int vis[2] = {ra < nrows ? seen(ra) : 0, ra + 8 < nrows ? seen(ra + 8) : 0};
    const bool idle = warp * 16 >= nrows;
    const int wmin = idle ? 0 : seen(warp * 16), wmax = idle ? 0 : seen(min(warp * 16 + 15, nrows - 1));

    // Runs of AP_RUN keys have maxima, sums and outputs of their own, joined here (in local memory, once per run): a sum does not grow longer
    // than it was in the split kernels
    volatile float ot[D / 8][4];
    float mt[2], lt[2];
    bool joined = false;
    auto join = [&]() {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float mine = 1.f, old = 0.f;
            if (joined) {
                const float m = fmaxf(mt[i], mrow[i]), base = m == -INFINITY ? 0.f : m;
                old = expf(mt[i] - base);
                mine = expf(mrow[i] - base);
                mrow[i] = m;
                lrow[i] = lt[i] * old + lrow[i] * mine;
            }
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
#pragma unroll
                for (int e = 2 * i; e < 2 * i + 2; ++e) {
                    if (joined) o[n][e] = ot[n][e] * old + o[n][e] * mine;
                }
        }
    };

    for (int t = group, i = 0; t < tiles; t += GROUPS, ++i) {
        if (i > 0 && i % (AP_RUN / AP_KEYS) == 0) {
            join();
            joined = true;
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    ot[n][e] = o[n][e];
                    o[n][e] = 0.f;
                }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                mt[i] = mrow[i];
                lt[i] = lrow[i];
                mrow[i] = -INFINITY;
                lrow[i] = 0.f;
            }
        }
        const int j0 = t * AP_KEYS;
        ap_sync(group);                                                 // the last tile is read
        __nv_bfloat162 last = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < NLD; ++i) {
            const int off = ((i * AP_GROUP + tid) / (D / 4)) * LD + tid % (D / 4) * 8;
            ap_split_store<NP>(K + off, KP, rk[i], last);
            ap_split_store<NP>(V + off, KP, rv[i], last);
        }
        // a key or value without three finite bf16 terms must neither lose its meaning nor, times a masked weight of zero, reach
        // queries before it: such a tile is computed in plain fp32
        const bool plain = ap_sync_or(group, qplain || !ap_finite(last));
        const bool none = j0 >= wmax;                                   // no row of this warp sees the tile
        if (none && !plain) {
            if (t + GROUPS < tiles) fetch(t + GROUPS);
            continue;
        }
        float s[AP_KEYS / 8][4], rest[AP_KEYS / 8][4];
        float *buf = reinterpret_cast<float *>(K);                      // plain: [rows][keys + 1] scores, then probabilities
        if (plain) {
            for (int i = tid; i < AP_ROWS * AP_KEYS; i += AP_GROUP) {
                const int r = i / AP_KEYS, j = j0 + i % AP_KEYS;
                float dot = 0.f;
                if (r < nrows && j < seen(r))
                    for (int d = 0; d < D; d += 4) {
                        const float4 x = query(r, d), y = kr.ld(j, d);
                        dot = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, dot))));
                    }
                buf[r * (AP_KEYS + 1) + i % AP_KEYS] = dot;
            }
            ap_sync(group);
#pragma unroll
            for (int n = 0; n < AP_KEYS / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[n][e] = buf[(ra + (e >> 1) * 8) * (AP_KEYS + 1) + n * 8 + (lane & 3) * 2 + (e & 1)];
        } else {
#pragma unroll
            for (int n = 0; n < AP_KEYS / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = rest[n][0] = rest[n][1] = rest[n][2] = rest[n][3] = 0.f;
            // 32 elements at a time: two chained steps, then fp32 sums of their own for the two chains
            auto load = [&](int kk, uint32_t (&af)[3][4], uint32_t (&bf)[2][3][4]) {
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ldsm4(af[p], skn_smem_u32(Q + p * QP + (warp * 16 + (lane & 15)) * LD + (kk + (lane >> 4) * 8) * 2));
                    if (p >= NP) continue;
                    const uint32_t kb = skn_smem_u32(K + p * KP + ((lane & 7) + ((lane >> 4) << 3)) * LD + (kk + ((lane >> 3) & 1) * 8) * 2);
                    ldsm4(bf[0][p], kb);
                    ldsm4(bf[1][p], kb + 16 * LD);
                }
            };
            auto half = [&](int from, float (&sum)[AP_KEYS / 8][4]) {
#pragma unroll 1
                for (int kk = from; kk < from + D / 2; kk += 32) {
                    uint32_t af[3][4], bf[2][3][4];
                    float small[4][4], c[4][4];
                    load(kk, af, bf);
                    mma_terms<NP, true>(small, c, af, bf);
                    load(kk + 16, af, bf);
                    mma_terms<NP, false>(small, c, af, bf);
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            sum[n][e] += c[n][e];
                            rest[n][e] += small[n][e];
                        }
                }
            };
            // (two halves: fewer roundings at the size of the whole score)
            float other[AP_KEYS / 8][4] = {};
            half(0, s);
            half(D / 2, other);
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[n][e] += other[n][e] + rest[n][e];
        }
        if (t + GROUPS < tiles) fetch(t + GROUPS);                                // (here, not before the scores: their fragments need the registers)
        float mx[2] = {mrow[0], mrow[1]};
        const bool masked = j0 + AP_KEYS > wmin;
#pragma unroll
        for (int n = 0; n < AP_KEYS / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (masked && j0 + n * 8 + (lane & 3) * 2 + (e & 1) >= vis[e >> 1]) s[n][e] = -INFINITY;
                mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
            }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        }
        if (__any_sync(0xffffffffu, mx[0] > mrow[0] || mx[1] > mrow[1])) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float corr = expf(mrow[i] - (mx[i] == -INFINITY ? 0.f : mx[i]));
                mrow[i] = mx[i];
                lrow[i] *= corr;
#pragma unroll
                for (int n = 0; n < D / 8; ++n) {
                    o[n][2 * i] *= corr;
                    o[n][2 * i + 1] *= corr;
                }
            }
        }
        mx[0] = mx[0] == -INFINITY ? 0.f : mx[0];
        mx[1] = mx[1] == -INFINITY ? 0.f : mx[1];
#pragma unroll
        for (int n = 0; n < AP_KEYS / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = expf(s[n][e] - mx[e >> 1]);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            lrow[i] += ((s[0][2 * i] + s[0][2 * i + 1]) + (s[1][2 * i] + s[1][2 * i + 1])) + ((s[2][2 * i] + s[2][2 * i + 1]) + (s[3][2 * i] + s[3][2 * i + 1]));
        if (plain) {
            __syncwarp();                                               // (a warp's rows are its own from here on)
#pragma unroll
            for (int n = 0; n < AP_KEYS / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) buf[(ra + (e >> 1) * 8) * (AP_KEYS + 1) + n * 8 + (lane & 3) * 2 + (e & 1)] = s[n][e];
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < AP_KEYS && j0 + j < vis[i]; ++j) {
                    const float p = buf[(ra + i * 8) * (AP_KEYS + 1) + j];
#pragma unroll
                    for (int n = 0; n < D / 8; ++n) {
                        const float4 y = vr.ld(j0 + j, n * 8 + ((lane & 2) << 1));
                        o[n][2 * i] = fmaf(p, lane & 1 ? y.z : y.x, o[n][2 * i]);
                        o[n][2 * i + 1] = fmaf(p, lane & 1 ? y.w : y.y, o[n][2 * i + 1]);
                    }
                }
            continue;
        }
#pragma unroll
        for (int kk = 0; kk < AP_KEYS / 16; ++kk) {
            uint32_t pf[3][4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float *w = s[2 * kk + (x >> 1)] + (x & 1) * 2;
                uint32_t t[3];
                split_terms(w[0], w[1], t);
                pf[0][x] = t[0]; pf[1][x] = t[1]; pf[2][x] = t[2];
            }
#pragma unroll
            for (int n = 0; n < D / 32; ++n) {
                float small[4][4], c[4][4];
                uint32_t bf[2][3][4];
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const uint32_t vb = skn_smem_u32(V + p * KP + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + (n * 32 + (lane >> 4) * 8) * 2);
                    ldsm4t(bf[0][p], vb);
                    ldsm4t(bf[1][p], vb + 32);
                }
                mma_terms<NP, true>(small, c, pf, bf);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[4 * n + i][e] += c[i][e] + small[i][e];
            }
        }
    }
    if (joined) join();
    if constexpr (GROUPS == 2) {
        // the odd tiles' part meets the even tiles': the same thread of both groups holds the same elements
        float *meet = reinterpret_cast<float *>(smb + 3 * QP) + tid;        // (over the key planes: 32 KB of maxima, sums and outputs)
        __syncthreads();
        if (group) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                meet[i * AP_GROUP] = mrow[i];
                meet[(2 + i) * AP_GROUP] = lrow[i];
            }
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) meet[(4 + 4 * n + e) * AP_GROUP] = o[n][e];
        }
        __syncthreads();
        if (group) return;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float m1 = meet[i * AP_GROUP], m = fmaxf(mrow[i], m1), base = m == -INFINITY ? 0.f : m, f0 = expf(mrow[i] - base), f1 = expf(m1 - base);
            lrow[i] = lrow[i] * f0 + meet[(2 + i) * AP_GROUP] * f1;
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
#pragma unroll
                for (int e = 2 * i; e < 2 * i + 2; ++e) o[n][e] = o[n][e] * f0 + meet[(4 + 4 * n + e) * AP_GROUP] * f1;
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float l = lrow[i];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if (ra + i * 8 >= nrows) continue;
        const size_t to = at(ra + i * 8) + (lane & 3) * 2;
#pragma unroll
        for (int n = 0; n < D / 8; ++n) {                               // (no visible key: zeros)
            const float2 v = vis[i] ? make_float2(o[n][2 * i] / l, o[n][2 * i + 1] / l) : make_float2(0.f, 0.f);
            if (a.out16) *reinterpret_cast<uint32_t *>(a.out16 + to + n * 8) = pack_bf16(v.x, v.y);
            else *reinterpret_cast<float2 *>(a.out + to + n * 8) = v;
        }
    }
}

template <int D, int DT, int GROUPS>
static cudaError_t ap_launch(const ap_args &a, cudaStream_t st) {
    auto kern = skn_attn_prompt_kernel<D, DT, GROUPS>;
    constexpr int smem = 3 * (AP_ROWS + GROUPS * 2 * AP_KEYS) * (D + 8) * 2;
    static_assert(GROUPS * 6 * AP_KEYS * (D + 8) * 2 >= (GROUPS - 1) * (4 + D / 2) * AP_GROUP * 4, "the groups' parts meet over the planes");
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(a.Hkv * a.B * ((a.T * a.G + AP_ROWS - 1) / AP_ROWS)), GROUPS * AP_GROUP, smem, st>>>(a);
    return cudaGetLastError();
}
template <int D, int GROUPS>
static cudaError_t ap_by_type(int dtype, const ap_args &a, cudaStream_t st) {
    return dtype == SKN_KV_F32 ? ap_launch<D, SKN_KV_F32, GROUPS>(a, st) : dtype == SKN_KV_F16 ? ap_launch<D, SKN_KV_F16, GROUPS>(a, st) : ap_launch<D, SKN_KV_Q8_0, GROUPS>(a, st);
}

bool skn_attn_prompt_covers(const skn_kvcache *kv, int G, int T) {
    if (T < 2 || (kv->head_dim != 64 && kv->head_dim != 128)) return false;
    const int64_t heads = (int64_t)kv->n_kv_heads * kv->batch, rows = (int64_t)T * G, tiles = (rows + AP_ROWS - 1) / AP_ROWS;
    return tiles * heads < (1 << 30) && rows * heads >= SKN_ATTN_PROMPT_ROWS;
}

// Whether this kernel is expected to end before the split kernels.  Those share the keys out as well, so their time goes with rows x keys; here
// a CTA walks all keys of its 64 rows, and the time goes with the keys and the waves of CTAs, however few rows there are.  Microseconds
// on B200, fitted to 548 shapes (1 to 16 sequences, 1 to 8 heads a group, 2 to 1024 tokens, contexts to 16384): all but 9 of them take
// the faster kernel to within 3 %, the others lose 4 us at most.  Tokens over cached ones, 32 heads of 128 over 8 kv heads, fp32, split
// kernels / this one:
//          context 512     2048          8192
//   64     51 / 65         144 / 229     519 / 887
//   96     67 / 65         206 / 229     769 / 888
//   128    82 / 65         265 / 229     1014 / 887
//   256    155 / 66        500 / 229     1997 / 888
bool skn_attn_prompt_faster(const skn_kvcache *kv, int G, int T, int keys) {
    const bool q8 = kv->dtype == SKN_KV_Q8_0, wide = kv->head_dim == 128;
    const double heads = (double)kv->n_kv_heads * kv->batch, krows = heads * G * T / 1000.0, seen = keys - T / 2.0;
    // split kernels: a key for a thousand rows, by heads of a group
    static const double split[2][2][4] = {{{.061, .037, .025, .024}, {.075, .047, .031, .031}}, {{.081, .045, .028, .021}, {.093, .053, .034, .032}}};
    const double per = split[q8][wide][G == 1 ? 0 : G == 2 ? 1 : G == 4 ? 2 : 3];
    const double before = 14.0 + krows * (seen * per + 4.0 * (keys < 256 ? keys / 256.0 : 1.0));
    // here: a key for a wave; fp16 rows are converted as they arrive, which waits for them where the cache is not in L2
    static const double tile[3][2] = {{.057, .108}, {.055, .115}, {.071, .131}};
    double key = tile[q8 ? 2 : kv->dtype == SKN_KV_F16 ? 1 : 0][wide];
    if (kv->dtype == SKN_KV_F16 && heads * keys * kv->head_dim * 4.0 > 48e6) key *= 1.4;
    const double ctas = heads * ((T * G + AP_ROWS - 1) / AP_ROWS), waves = ceil(ctas / kv->ctx->sm_count);
    const double most = fmax(fmax((double)keys, (double)AP_KEYS), waves * seen);
    return 12.0 + key * most + 1.0 <= before;
}

cudaError_t skn_launch_attn_prompt(const skn_kvcache *kv, const float *q, int G, int T, float scale, int len_extra, int keys, float *out, void *out_bf16, cudaStream_t st) {
    const ap_args a = {q, kv->d_k, kv->d_v, kv->d_len, kv->d_start, out, (__nv_bfloat16 *)out_bf16, kv->n_kv_heads, G, kv->capacity, T, len_extra, kv->batch, scale};
    // (one tile of keys: a second group would have none, and takes the place of another CTA; 16 sequences of 20 tokens 19 us, with it 27)
    if (keys <= AP_KEYS) return kv->head_dim == 128 ? ap_by_type<128, 1>(kv->dtype, a, st) : ap_by_type<64, 1>(kv->dtype, a, st);
    return kv->head_dim == 128 ? ap_by_type<128, 2>(kv->dtype, a, st) : ap_by_type<64, 2>(kv->dtype, a, st);
}
