// Chunked attention and retention (see skn_mixers.cuh).
//
//  skn_mix_decode_kernel   one token per sequence.  Attention CTAs: (128-key split, group of up to four query heads of
//                          one kv head, row); the CTA that holds the newest key normalises, rotates and stores it.
//                          Splits meet in the CTA that draws the last ticket.  Retention CTAs of the same launch: one
//                          head of one row, the state read and written once.
//  skn_head_prep_kernel    many tokens: norm and rotation of every head, K and V into the cache
//  skn_attn_tc_kernel      64 queries of one head: scores and products on the tensor cores (bf16 operands, fp32 sums);
//                          the weights enter the second product as two bf16 terms, so they keep 16 bits
//  skn_attn_rows_kernel    the split kernel on prepared keys (fp32 cache, or head widths beyond the tensor-core form)
//  skn_ret_*_kernel        retention in chunks of 64 tokens: what each chunk adds to the state, the states at the chunk
//                          starts, and the outputs; on the CUDA cores (fp32 decoder) or the tensor cores (three bf16 terms)
#include "skn_mixers.cuh"
#include "skn_mma.cuh"

#include <math.h>
#include <stdlib.h>

constexpr int MIX_THREADS = 256;
constexpr int KS = SKN_ATTN_SPLIT_KEYS;

template <class CT> struct CacheVec;
template <> struct CacheVec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float *p, float *o) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
    static __device__ __forceinline__ float round(float v) { return v; }
    static __device__ __forceinline__ void store(float *p, float v) { *p = v; }
};
template <> struct CacheVec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16 *p, float *o) {
        const uint4 v = *reinterpret_cast<const uint4 *>(p);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            o[2 * i] = __uint_as_float(w[i] << 16);
            o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
        }
    }
    static __device__ __forceinline__ float round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
    static __device__ __forceinline__ void store(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// One warp: raw head (global) -> dst (shared, `pad` floats, zero-filled past dim): optional RMS norm with a gain, then
// rotation of the pairs (i, i + half), then a factor.
__device__ __forceinline__ void prep_head(const float *src, int dim, int pad, const float *gain, float eps, const skn_rot &rot, int64_t row,
                                          float mul, float *dst) {
    const int lane = threadIdx.x & 31;
    float ss = 0.f;
    for (int d = lane; d < pad; d += 32) {
        const float v = d < dim ? __ldcg(src + d) : 0.f;
        dst[d] = v;
        ss = fmaf(v, v, ss);
    }
    if (gain) {
        const float r = 1.f / sqrtf(warp_sum(ss) / (float)dim + eps);
        for (int d = lane; d < dim; d += 32) dst[d] = dst[d] * r * __ldg(gain + d);
    }
    __syncwarp();
    for (int i = lane; i < rot.half; i += 32) {
        const float2 cs = __ldcg(rot.table + row * rot.ld + i);
        const float u = dst[i], v = dst[i + rot.half];
        dst[i] = u * cs.x - v * cs.y;
        dst[i + rot.half] = v * cs.x + u * cs.y;
    }
    __syncwarp();
    if (mul != 1.f)
        for (int d = lane; d < dim; d += 32) dst[d] *= mul;
    __syncwarp();
}

// first key that the query at position p sees
__device__ __forceinline__ int first_visible(const skn_attn_args &a, int p) {
    return a.chunk > 0 ? p / a.chunk * a.chunk : a.window > 0 ? max(0, p - a.window + 1) : 0;
}

__device__ __forceinline__ void put_out(const skn_rows_out &o, int64_t m, int64_t c, float v) {
    if (o.y32) o.y32[m * o.ld32 + c] = v;
    if (o.y16) o.y16[m * o.ld16 + c] = __float2bfloat16_rn(v);
}

// ---- attention over a split of the keys ---------------------------------------------------------------------------
// smem (floats): q [RT][kp] | key [kp] | value [vp] | weights [RT][KS] | red [partial sums][RT][vp]
template <class CT, int RT>
static size_t attn_split_smem(int kp, int vp) {
    const int ng = vp / CacheVec<CT>::N, parts = ng <= 32 && 32 % ng == 0 ? MIX_THREADS / 32 : MIX_THREADS / ng;
    return ((size_t)RT * kp + kp + vp + RT * KS + (size_t)parts * RT * vp) * sizeof(float);
}

template <class CT, int RT, bool APPEND>
__device__ void attn_split(const skn_attn_args &a, const skn_step &st, const CT *__restrict__ kc_, const CT *__restrict__ vc_, int G, int cap, int dim,
                           int vdim, int kp, int vp, int vld, int split, int max_splits, int hg, int m, float *sm) {
    constexpr int VE = CacheVec<CT>::N;
    __shared__ float s_red[MIX_THREADS / 32][RT], s_max[RT], s_sum[RT];
    __shared__ bool s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = a.heads / G, ngr = (R + RT - 1) / RT, g = hg / ngr, sub = hg % ngr;
    const int h0 = g * R + sub * RT, nh = min(RT, R - sub * RT);
    const int seq = m / st.T, slot = st.slot0 + seq;
    const int p = min(st.pos[slot] + m % st.T, st.max_pos - 1);
    const int lo = first_visible(a, p);
    const int live = (p - lo) / KS + 1;
    if (split >= live) return;
    const int j0 = lo + split * KS, nk = min(KS, p + 1 - j0);
    const bool newest = APPEND && split == live - 1;       // this split ends with the step's own key
    float *qs = sm, *kn = qs + RT * kp, *vn = kn + kp, *ws = vn + vp, *red = ws + RT * KS;
    const size_t head_rows = ((size_t)slot * G + g) * cap;
    CT *kc = const_cast<CT *>(kc_) + head_rows * kp, *vc = const_cast<CT *>(vc_) + head_rows * vld;
    // keys and values on their way into L2 while the query is prepared: two threads per key
    const int key = tid >> 1, half = tid & 1;
    const int kslot = (j0 + key) % cap;
    if (key < nk) {
        const char *kr = reinterpret_cast<const char *>(kc + (size_t)kslot * kp), *vr = reinterpret_cast<const char *>(vc + (size_t)kslot * vld);
        for (int i = half * 128; i < (int)(kp * sizeof(CT)); i += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(kr + i));
        if (vc != kc)
            for (int i = half * 128; i < (int)(vp * sizeof(CT)); i += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(vr + i));
    }

    for (int i = warp; i < RT + 2; i += MIX_THREADS / 32) {
        if (i < RT) {
            if (i < nh) prep_head(a.q + (int64_t)m * a.ld + (int64_t)(h0 + i) * dim, dim, kp, a.q_gain, a.eps, a.rot, m, a.scale, qs + i * kp);
            else for (int d = lane; d < kp; d += 32) qs[i * kp + d] = 0.f;
        } else if (newest && i == RT) {
            prep_head(a.k + (int64_t)m * a.ld + (int64_t)g * dim, dim, kp, a.k_gain, a.eps, a.rot, m, 1.f, kn);
            for (int d = lane; d < dim; d += 32) {
                if (sub == 0) CacheVec<CT>::store(kc + (size_t)(p % cap) * kp + d, kn[d]);
                kn[d] = CacheVec<CT>::round(kn[d]);
            }
        } else if (newest) {
            for (int d = lane; d < vp; d += 32) {
                const float v = d < vdim ? __ldcg(a.v + (int64_t)m * a.ld + (int64_t)g * vdim + d) : 0.f;
                if (sub == 0 && d < vdim) CacheVec<CT>::store(vc + (size_t)(p % cap) * vld + d, v);
                vn[d] = CacheVec<CT>::round(v);
            }
        }
    }
    __syncthreads();

    // scores: two threads per key, each takes every other vector of the row
    const bool valid = key < nk, own = newest && key == nk - 1;
    float s[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) s[r] = 0.f;
    if (valid) {
        const CT *kr = kc + (size_t)kslot * kp;
#pragma unroll 4
        for (int u = half; u < kp / VE; u += 2) {
            float kv[VE];
            if (own) {
#pragma unroll
                for (int e = 0; e < VE; ++e) kv[e] = kn[u * VE + e];
            } else CacheVec<CT>::load(kr + u * VE, kv);
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int e = 0; e < VE; ++e) s[r] = fmaf(qs[r * kp + u * VE + e], kv[e], s[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        s[r] += __shfl_xor_sync(0xffffffffu, s[r], 1);
        if (a.softcap > 0.f) s[r] = a.softcap * tanhf(s[r] / a.softcap);
        if (!valid) s[r] = -INFINITY;
        const float wm = warp_max(s[r]);
        if (lane == 0) s_red[warp][r] = wm;
    }
    __syncthreads();
    float mx[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        mx[r] = s_red[0][r];
#pragma unroll
        for (int w = 1; w < MIX_THREADS / 32; ++w) mx[r] = fmaxf(mx[r], s_red[w][r]);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RT; ++r) {
        const float e = valid ? expf(s[r] - mx[r]) : 0.f;
        if (half == 0) ws[r * KS + key] = e;
        const float t = warp_sum(half == 0 ? e : 0.f);
        if (lane == 0) s_red[warp][r] = t;
    }
    __syncthreads();
    if (tid < RT) {
        float t = 0.f;
        for (int w = 0; w < MIX_THREADS / 32; ++w) t += s_red[w][tid];
        s_sum[tid] = t;
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
        if (tid == r) s_max[r] = mx[r];

    // values: a thread owns one vector of columns and every kl-th key
    const int ng = vp / VE, kl = MIX_THREADS / ng, cg_ = tid % ng, kk = tid / ng;
    float acc[RT][VE];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int e = 0; e < VE; ++e) acc[r][e] = 0.f;
    if (kk < kl) {
        const int first = j0 % cap;
#pragma unroll 4
        for (int j = kk; j < nk; j += kl) {
            float vv[VE];
            int sl = first + j;
            if (sl >= cap) sl -= cap;              // (a cache holds at least the keys that one query sees)
            if (newest && j == nk - 1) {
#pragma unroll
                for (int e = 0; e < VE; ++e) vv[e] = vn[cg_ * VE + e];
            } else CacheVec<CT>::load(vc + (size_t)sl * vld + cg_ * VE, vv);
#pragma unroll
            for (int r = 0; r < RT; ++r) {
                const float w = ws[r * KS + j];
#pragma unroll
                for (int e = 0; e < VE; ++e) acc[r][e] = fmaf(w, vv[e], acc[r][e]);
            }
        }
    }
    // a column vector's partial sums: first across the lanes of a warp that hold the same columns, then across the warps
    const bool fold = ng <= 32 && 32 % ng == 0;
    if (fold) {
        for (int o = ng; o < 32; o <<= 1)
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int e = 0; e < VE; ++e) acc[r][e] += __shfl_xor_sync(0xffffffffu, acc[r][e], o);
    }
    const int part = fold ? warp : kk;
    if (kk < kl && (!fold || lane < ng)) {
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
            for (int e = 0; e < VE; ++e) red[((size_t)part * RT + r) * vp + cg_ * VE + e] = acc[r][e];
    }
    __syncthreads();
    const int nk_l = fold ? MIX_THREADS / 32 : min(kl, nk);
    for (int i = tid; i < nh * vdim; i += MIX_THREADS) {
        const int r = i / vdim, c = i % vdim;
        float o = 0.f;
        for (int k2 = 0; k2 < nk_l; ++k2) o += red[((size_t)k2 * RT + r) * vp + c];
        if (live == 1) put_out(a.out, m, (int64_t)(h0 + r) * vdim + c, o / (a.sink ? s_sum[r] + expf(a.sink[h0 + r] - s_max[r]) : s_sum[r]) * a.out_scale);
        else __stcg(a.scratch + (((size_t)m * a.heads + h0 + r) * max_splits + split) * (vdim + 2) + 2 + c, o);
    }
    if (live == 1) return;
    if (tid < nh) {
        float *rec = a.scratch + (((size_t)m * a.heads + h0 + tid) * max_splits + split) * (vdim + 2);
        __stcg(rec, s_max[tid]);
        __stcg(rec + 1, s_sum[tid]);
    }
    __threadfence();
    __syncthreads();
    unsigned *ticket = a.tickets + (size_t)m * a.heads + h0;
    if (tid == 0) s_last = atomicAdd(ticket, 1u) == (unsigned)(live - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // weight of every split (in place of the scores): exp(max - top) / sum
    for (int r = warp; r < nh; r += MIX_THREADS / 32) {
        const float *rec = a.scratch + ((size_t)m * a.heads + h0 + r) * max_splits * (vdim + 2);
        float top = -INFINITY;
        for (int x = lane; x < live; x += 32) top = fmaxf(top, __ldcg(rec + (size_t)x * (vdim + 2)));
        top = warp_max(top);
        const float sink = a.sink ? a.sink[h0 + r] : -INFINITY;
        top = fmaxf(top, sink);
        float den = 0.f;
        for (int x = lane; x < live; x += 32) den += expf(__ldcg(rec + (size_t)x * (vdim + 2)) - top) * __ldcg(rec + (size_t)x * (vdim + 2) + 1);
        den = warp_sum(den) + (a.sink ? expf(sink - top) : 0.f);
        for (int x = lane; x < live; x += 32)
            if (x < KS) ws[r * KS + x] = expf(__ldcg(rec + (size_t)x * (vdim + 2)) - top) / den;
        if (lane == 0) { s_max[r] = top; s_sum[r] = den; }
    }
    __syncthreads();
    for (int i = tid; i < nh * vdim; i += MIX_THREADS) {
        const int r = i / vdim, c = i % vdim;
        const float *rec = a.scratch + ((size_t)m * a.heads + h0 + r) * max_splits * (vdim + 2);
        float num = 0.f;
#pragma unroll 8
        for (int x = 0; x < live; ++x) {
            const float f = x < KS ? ws[r * KS + x] : expf(__ldcg(rec + (size_t)x * (vdim + 2)) - s_max[r]) / s_sum[r];
            num = fmaf(f, __ldcg(rec + (size_t)x * (vdim + 2) + 2 + c), num);
        }
        put_out(a.out, m, (int64_t)(h0 + r) * vdim + c, num * a.out_scale);
    }
    if (tid == 0) *ticket = 0;
}

// ---- retention, one token ----------------------------------------------------------------------------------------
// smem (floats): q [dk] | k [dk] | v [vp] | o [vp] | red [MIX_THREADS * 4]
static size_t ret_step_smem(int dk, int vp) { return ((size_t)2 * ((dk + 3) / 4 * 4) + 2 * vp + MIX_THREADS * 4) * sizeof(float); }

__device__ void ret_step(const skn_ret_args &r, const skn_step &st, float *__restrict__ S, int H, int dk, int dv, int vp, int h, int m, float *sm) {
    __shared__ float s_w[MIX_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, dkp = (dk + 3) / 4 * 4;
    float *qs = sm, *ks = qs + dkp, *vs = ks + dkp, *os = vs + vp, *red = os + vp;
    const int slot = st.slot0 + m / st.T;
    const bool fresh = st.pos[slot] == 0;
    const float decay = __ldg(r.powers + (size_t)h * (SKN_RET_CHUNK + 1) + 1);
    if (warp == 0) prep_head(r.q + (int64_t)m * r.ld + (int64_t)h * dk, dk, dk, nullptr, 0.f, r.rot, m, 1.f, qs);
    else if (warp == 1) prep_head(r.k + (int64_t)m * r.ld + (int64_t)h * dk, dk, dk, nullptr, 0.f, r.rot, m, r.k_scale, ks);
    else if (warp == 2)
        for (int d = lane; d < vp; d += 32) vs[d] = d < dv ? __ldcg(r.v + (int64_t)m * r.ld + (int64_t)h * dv + d) : 0.f;
    __syncthreads();
    float *base = S + ((size_t)slot * H + h) * dk * vp;
    // the column groups that do not fill the block at once take further turns
    for (int c0 = 0; c0 < vp / 4; c0 += MIX_THREADS) {
        const int nc = min(MIX_THREADS, vp / 4 - c0), lanes = MIX_THREADS / nc, cg_ = tid % nc, rl = tid / nc;
        if (rl < lanes) {
            const int c = (c0 + cg_) * 4;
            const float4 v = *reinterpret_cast<const float4 *>(vs + c);
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int i = rl; i < dk; i += lanes) {
                float4 *p = reinterpret_cast<float4 *>(base + (size_t)i * vp + c);
                float4 s = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *p;
                const float k = ks[i], q = qs[i];
                s.x = fmaf(decay, s.x, k * v.x);
                s.y = fmaf(decay, s.y, k * v.y);
                s.z = fmaf(decay, s.z, k * v.z);
                s.w = fmaf(decay, s.w, k * v.w);
                *p = s;
                o.x = fmaf(q, s.x, o.x);
                o.y = fmaf(q, s.y, o.y);
                o.z = fmaf(q, s.z, o.z);
                o.w = fmaf(q, s.w, o.w);
            }
            *reinterpret_cast<float4 *>(red + ((size_t)rl * nc + cg_) * 4) = o;
        }
        __syncthreads();
        for (int i = tid; i < nc * 4; i += MIX_THREADS) {
            float t = 0.f;
            for (int x = 0; x < min(lanes, dk); ++x) t += red[(size_t)x * nc * 4 + i];
            os[c0 * 4 + i] = t;
        }
        __syncthreads();
    }
    float ss = 0.f;
    for (int d = tid; d < dv; d += MIX_THREADS) ss = fmaf(os[d], os[d], ss);
    ss = warp_sum(ss);
    if (lane == 0) s_w[warp] = ss;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < MIX_THREADS / 32; ++w) t += s_w[w];
    const float rs = 1.f / sqrtf(t / (float)dv + r.eps);
    for (int d = tid; d < dv; d += MIX_THREADS) {
        const float gt = __ldcg(r.g + (int64_t)m * r.ld + (int64_t)h * dv + d);
        put_out(r.out, m, (int64_t)h * dv + d, os[d] * rs * (gt / (1.f + expf(-gt))) * r.out_scale);
    }
}

template <class CT, int RT>
__global__ void __launch_bounds__(MIX_THREADS, 4)
skn_mix_decode_kernel(skn_attn_args a, skn_ret_args r, skn_step st, const CT *kc, const CT *vc, int G, int cap, int dim, int vdim, int kp,
                      int vp, int vld, int max_splits, int n_attn, float *S, int RH, int rdk, int rdv, int rvp) {
    extern __shared__ __align__(16) float sm[];
    // the next launch starts only when this one's CTAs end (no early trigger): the weights it would stream meanwhile make
    // every step of this chain of dependent loads wait longer
    skn_pdl_wait();
    const int m = blockIdx.y, b = blockIdx.x;
    if (b < n_attn) attn_split<CT, RT, true>(a, st, kc, vc, G, cap, dim, vdim, kp, vp, vld, b % max_splits, max_splits, b / max_splits, m, sm);
    else ret_step(r, st, S, RH, rdk, rdv, rvp, b - n_attn, m, sm);
}

template <class CT, int RT>
__global__ void __launch_bounds__(MIX_THREADS)
skn_attn_rows_kernel(skn_attn_args a, skn_step st, const CT *kc, const CT *vc, int G, int cap, int dim, int vdim, int kp, int vp, int vld,
                     int max_splits) {
    extern __shared__ __align__(16) float sm[];
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    attn_split<CT, RT, false>(a, st, kc, vc, G, cap, dim, vdim, kp, vp, vld, blockIdx.x % max_splits, max_splits, blockIdx.x / max_splits, blockIdx.y, sm);
}

template <class CT, int RT>
static cudaError_t launch_decode_t(const skn_step &s, const skn_attn_args *a, const skn_ret_args *r, bool rows_only, cudaStream_t st) {
    skn_attn_args aa = {};
    skn_ret_args rr = {};
    int G = 1, cap = 1, dim = 1, vdim = 1, kp = 16, vp = 16, vld = 16, ms = 1, n_attn = 0, RH = 0, dk = 1, dv = 1, rvp = 4;
    const CT *kc = nullptr, *vc = nullptr;
    float *S = nullptr;
    size_t smem = 0;
    if (a) {
        aa = *a;
        G = a->kv->n_kv_heads; cap = a->kv->capacity; dim = a->kv->head_dim; vdim = a->kv->v_dim; kp = a->kv->k_pitch; vp = a->kv->v_pitch;
        vld = a->kv->v_stride;
        kc = (const CT *)a->kv->d_k;
        vc = (const CT *)a->kv->d_v;
        ms = skn_attn_splits(a->chunk > 0 ? a->chunk : a->window, s.max_pos);
        n_attn = ms * G * ((a->heads / G + RT - 1) / RT);
        smem = attn_split_smem<CT, RT>(kp, vp);
    }
    if (r) {
        rr = *r;
        S = r->state->d;
        RH = r->state->heads; dk = r->state->k_dim; dv = r->state->v_dim; rvp = r->state->v_pitch;
        const size_t b = ret_step_smem(dk, rvp);
        if (b > smem) smem = b;
    }
    const dim3 grid(n_attn + (rows_only ? 0 : RH), s.n_seqs * s.T);
    if (rows_only) {
        auto kern = skn_attn_rows_kernel<CT, RT>;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        if (e != cudaSuccess) return e;
        return skn_launch_pdl(kern, grid, dim3(MIX_THREADS), smem, st, 1, aa, s, kc, vc, G, cap, dim, vdim, kp, vp, vld, ms);
    }
    auto kern = skn_mix_decode_kernel<CT, RT>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
    if (e != cudaSuccess) return e;
    return skn_launch_pdl(kern, grid, dim3(MIX_THREADS), smem, st, 1, aa, rr, s, kc, vc, G, cap, dim, vdim, kp, vp, vld, ms, n_attn, S, RH, dk, dv, rvp);
}

static cudaError_t launch_split(const skn_step &s, const skn_attn_args *a, const skn_ret_args *r, bool rows_only, cudaStream_t st) {
    const int R = a ? a->heads / a->kv->n_kv_heads : 1;
    if (a && a->kv->dtype == SKN_KV_BF16)
        return R > 2 ? launch_decode_t<__nv_bfloat16, 4>(s, a, r, rows_only, st) : R == 2 ? launch_decode_t<__nv_bfloat16, 2>(s, a, r, rows_only, st)
                                                                                : launch_decode_t<__nv_bfloat16, 1>(s, a, r, rows_only, st);
    return R > 2 ? launch_decode_t<float, 4>(s, a, r, rows_only, st) : R == 2 ? launch_decode_t<float, 2>(s, a, r, rows_only, st)
                                                                   : launch_decode_t<float, 1>(s, a, r, rows_only, st);
}

cudaError_t skn_launch_attn_rows(const skn_step &s, const skn_attn_args &a, cudaStream_t st) { return launch_split(s, &a, nullptr, true, st); }

cudaError_t skn_launch_mix_decode(skn_ctx *, const skn_step &s, const skn_attn_args *a, const skn_ret_args *r, cudaStream_t st) {
    if (s.T != 1) return cudaErrorInvalidValue;
    return launch_split(s, a, r, false, st);
}

// ---- many tokens: heads prepared, keys and values into the cache --------------------------------------------------
struct prep_args {
    int H, G, dim, vdim, kp, vp, cap;
    int RH, rdk;
};

template <class CT>
__global__ void __launch_bounds__(256)
skn_head_prep_kernel(skn_attn_args a, skn_ret_args r, skn_step st, prep_args p, CT *kc, CT *vc) {
    extern __shared__ __align__(16) float sm[];
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = blockIdx.x;
    const int width = max(p.kp, p.rdk);
    float *buf = sm + (size_t)warp * width;
    const int slot = st.slot0 + m / st.T, pos = min(st.pos[slot] + m % st.T, st.max_pos - 1);
    const int nq = a.q16 ? p.H : 0, units = nq + 2 * p.G + 2 * p.RH;
    for (int u = warp; u < units; u += 8) {
        if (u < nq) {
            prep_head(a.q + (int64_t)m * a.ld + (int64_t)u * p.dim, p.dim, p.kp, a.q_gain, a.eps, a.rot, m, 1.f, buf);
            for (int d = lane; d < p.kp; d += 32) a.q16[((int64_t)m * p.H + u) * p.kp + d] = __float2bfloat16_rn(buf[d]);
        } else if (u < nq + p.G) {
            const int g = u - nq;
            prep_head(a.k + (int64_t)m * a.ld + (int64_t)g * p.dim, p.dim, p.kp, a.k_gain, a.eps, a.rot, m, 1.f, buf);
            CT *dst = kc + (((size_t)slot * p.G + g) * p.cap + pos % p.cap) * p.kp;
            for (int d = lane; d < p.dim; d += 32) CacheVec<CT>::store(dst + d, buf[d]);
        } else if (u < nq + 2 * p.G) {
            const int g = u - nq - p.G;
            CT *dst = vc + (((size_t)slot * p.G + g) * p.cap + pos % p.cap) * p.vp;
            for (int d = lane; d < p.vdim; d += 32) CacheVec<CT>::store(dst + d, __ldcg(a.v + (int64_t)m * a.ld + (int64_t)g * p.vdim + d));
        } else {
            const int i = u - nq - 2 * p.G, h = i >> 1;
            float *src = ((i & 1) ? r.k : r.q) + (int64_t)m * r.ld + (int64_t)h * p.rdk;
            prep_head(src, p.rdk, p.rdk, nullptr, 0.f, r.rot, m, (i & 1) ? r.k_scale : 1.f, buf);
            for (int d = lane; d < p.rdk; d += 32) src[d] = buf[d];
        }
        __syncwarp();
    }
}

// four numbers into a cache row or prepared queries
__device__ __forceinline__ void put4(float *to, float4 v) { *reinterpret_cast<float4 *>(to) = v; }
__device__ __forceinline__ void put4(__nv_bfloat16 *to, float4 v) { *reinterpret_cast<uint2 *>(to) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)); }

// The same with a head in registers, four elements per lane and register of NV: for widths, halves of rotations and row strides that are multiples of four
// and rows on 16 bytes (head_prep_aligned).  The element-wise form above goes through shared memory three times and asks for 32 numbers at a time: 44 us
// for 2048 rows of 5120 head elements (70 MB), 26 us here; a warp's next head is on its way while it prepares one.
template <class CT, int NV>
__global__ void __launch_bounds__(256)
skn_head_prep_vec_kernel(skn_attn_args a, skn_ret_args r, skn_step st, prep_args p, CT *kc, CT *vc) {
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = blockIdx.x;
    const int slot = st.slot0 + m / st.T, pos = min(st.pos[slot] + m % st.T, st.max_pos - 1), at = p.cap ? pos % p.cap : 0;
    const int nq = a.q16 ? p.H : 0, units = nq + 2 * p.G + 2 * p.RH;
    // where the raw head of unit u is, and its width
    auto source = [&](int u, int &w) -> float * {
        if (u < nq) { w = p.dim; return const_cast<float *>(a.q) + (int64_t)m * a.ld + (int64_t)u * p.dim; }
        if (u < nq + p.G) { w = p.dim; return const_cast<float *>(a.k) + (int64_t)m * a.ld + (int64_t)(u - nq) * p.dim; }
        if (u < nq + 2 * p.G) { w = p.vdim; return const_cast<float *>(a.v) + (int64_t)m * a.ld + (int64_t)(u - nq - p.G) * p.vdim; }
        const int i = u - nq - 2 * p.G;
        w = p.rdk;
        return ((i & 1) ? r.k : r.q) + (int64_t)m * r.ld + (int64_t)(i >> 1) * p.rdk;
    };
    auto fetch = [&](int u, float4 (&x)[NV]) {
        int w = 0;
        const float *src = u < units ? source(u, w) : nullptr;
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            const int d = (c * 32 + lane) * 4;
            x[c] = d < w ? __ldcg(reinterpret_cast<const float4 *>(src + d)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    float4 x[NV], next[NV];
    fetch(warp, x);
    for (int u = warp; u < units; u += 8) {
        fetch(u + 8, next);
        int w;
        float *src = source(u, w);
        const bool value = u >= nq + p.G && u < nq + 2 * p.G, ret = u >= nq + 2 * p.G;
        const float *gain = ret || value ? nullptr : u < nq ? a.q_gain : a.k_gain;
        if (gain) {
            float ss = 0.f;
#pragma unroll
            for (int c = 0; c < NV; ++c) ss += (x[c].x * x[c].x + x[c].y * x[c].y) + (x[c].z * x[c].z + x[c].w * x[c].w);
            const float f = 1.f / sqrtf(warp_sum(ss) / (float)w + a.eps);
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                const int d = (c * 32 + lane) * 4;
                if (d >= w) continue;
                const float4 g = __ldg(reinterpret_cast<const float4 *>(gain + d));
                x[c] = make_float4(x[c].x * f * g.x, x[c].y * f * g.y, x[c].z * f * g.z, x[c].w * f * g.w);
            }
        }
        const skn_rot &rot = ret ? r.rot : a.rot;
        if (!value && rot.half > 0) {
            float4 y[NV];
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                // the other element of a pair is half a rotation away
                const int d = (c * 32 + lane) * 4, o = (d < rot.half ? d + rot.half : d - rot.half) >> 2, from = o & 31;
                y[c] = make_float4(__shfl_sync(0xffffffffu, x[0].x, from), __shfl_sync(0xffffffffu, x[0].y, from), __shfl_sync(0xffffffffu, x[0].z, from),
                                   __shfl_sync(0xffffffffu, x[0].w, from));
                if (NV > 1) {
                    const float4 z = make_float4(__shfl_sync(0xffffffffu, x[NV - 1].x, from), __shfl_sync(0xffffffffu, x[NV - 1].y, from),
                                                 __shfl_sync(0xffffffffu, x[NV - 1].z, from), __shfl_sync(0xffffffffu, x[NV - 1].w, from));
                    if (o >= 32) y[c] = z;
                }
            }
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                const int d = (c * 32 + lane) * 4;
                if (d >= 2 * rot.half) continue;
                const bool low = d < rot.half;
                const float4 *t = reinterpret_cast<const float4 *>(rot.table + (int64_t)m * rot.ld + (low ? d : d - rot.half));
                const float4 t0 = __ldcg(t), t1 = __ldcg(t + 1);
                const float sg = low ? -1.f : 1.f;                     // u c - v s, v c + u s
                x[c] = make_float4(x[c].x * t0.x + sg * (y[c].x * t0.y), x[c].y * t0.z + sg * (y[c].y * t0.w), x[c].z * t1.x + sg * (y[c].z * t1.y),
                                   x[c].w * t1.z + sg * (y[c].w * t1.w));
            }
        }
        if (ret && ((u - nq - 2 * p.G) & 1) && r.k_scale != 1.f)
#pragma unroll
            for (int c = 0; c < NV; ++c) x[c] = make_float4(x[c].x * r.k_scale, x[c].y * r.k_scale, x[c].z * r.k_scale, x[c].w * r.k_scale);
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            const int d = (c * 32 + lane) * 4;
            if (u < nq) {
                if (d < p.kp) put4(a.q16 + ((int64_t)m * p.H + u) * p.kp + d, x[c]);
            } else if (d < w) {
                if (ret) put4(src + d, x[c]);
                else if (value) put4(vc + (((size_t)slot * p.G + u - nq - p.G) * p.cap + at) * p.vp + d, x[c]);
                else put4(kc + (((size_t)slot * p.G + u - nq) * p.cap + at) * p.kp + d, x[c]);
            }
            x[c] = next[c];
        }
    }
}
static bool head_prep_aligned(const skn_attn_args *a, const skn_ret_args *r, const prep_args &p) {
    uintptr_t at = 0;
    int64_t n = 0;
    if (a) {
        at |= (uintptr_t)a->q | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->q_gain | (uintptr_t)a->k_gain | (uintptr_t)a->rot.table | (uintptr_t)a->q16;
        n |= a->ld | p.dim | p.vdim | p.kp | p.vp | a->rot.half | (a->rot.half ? a->rot.ld : 0);
    }
    if (r) {
        at |= (uintptr_t)r->q | (uintptr_t)r->k | (uintptr_t)r->rot.table;
        n |= r->ld | p.rdk | r->rot.half | (r->rot.half ? r->rot.ld : 0);
    }
    return !(at & 15) && !(n & 3);
}

// ---- attention on the tensor cores ---------------------------------------------------------------------------------
constexpr int ATQ = 64, ATK = 32;      // queries and keys of a tile
constexpr int AT_THREADS = ATQ * 2;    // a warp owns 16 queries

// (results below 2^-126 are zero: such a weight beside a largest one of 1)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// What bounds it: the instructions beside the products.  It issued 66 per score and was busy with 8 x 8 products for a quarter of
// its time (2048 tokens, 16 heads of 128, chunk 1024, soft cap: 135 us).  Now the soft cap is five instructions a score (c - 2 c / (e^(2 s / cap) + 1)
// needs no clamp: the exponential may overflow), masks are looked at in tiles that have one, outputs are rescaled in tiles that raise a
// maximum of the warp, fragments are fetched a step ahead of the products that take them, and CTAs with the most keys start first (86 us; 23 would be the products').
template <int DV>
__global__ void __launch_bounds__(AT_THREADS, DV <= 128 ? 3 : 1)
skn_attn_tc_kernel(skn_attn_args a, skn_step st, skn_attn_keys src) {
    extern __shared__ __align__(16) uint8_t smb[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kp = src.kp, vp = src.vp, cap = src.cap, vdim = src.vdim;
    const int ks = kp + 8, vs = DV + 8;                                  // row strides in elements
    __nv_bfloat16 *Q = reinterpret_cast<__nv_bfloat16 *>(smb), *K = Q + ATQ * ks, *V = K + 2 * ATK * ks;
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    // query tiles by the keys they see, most first: in chunks, by their place in the chunk
    const int nt = (st.T + ATQ - 1) / ATQ, pc = a.chunk > 0 ? min(nt, (a.chunk + ATQ - 1) / ATQ) : nt, nc = (nt + pc - 1) / pc;
    const int qt = ((int)blockIdx.y % nc) * pc + pc - 1 - (int)blockIdx.y / nc;
    if (qt >= nt) return;
    const int t0 = qt * ATQ, h = blockIdx.x, seq = blockIdx.z, slot = st.slot0 + seq, g = h / src.group;
    const int p0 = st.pos[slot], nq = min(ATQ, st.T - t0);
    const int pf = p0 + t0, pl = pf + nq - 1;                            // first and last query position
    const int lo = first_visible(a, pf);
    const int tiles = (pl - lo) / ATK + 1;
    const __nv_bfloat16 *kc = src.k + slot * src.k_slot + g * src.k_head, *vc = src.v + slot * src.v_slot + g * src.v_head;
    const __nv_bfloat16 *kc2 = src.k2 ? src.k2 + slot * src.k2_slot : nullptr;

    const int slot0 = lo % cap;
    const bool idle = warp * 16 >= nq;                                   // none of this warp's queries exist
    // four threads per key row (two per query row), every fourth 16-byte piece each
    const int cr = tid >> 2, cc = tid & 3;
    auto load_tile = [&](int t, int buf) {
        const int j = lo + t * ATK + cr;
        const bool in = j <= pl;
        int sl = slot0 + t * ATK + cr;
        if (sl >= cap) sl %= cap;
        const __nv_bfloat16 *kr = kc + sl * src.k_row, *vr = vc + sl * src.v_row, *kr2 = kc2 + sl * src.k2_row - src.k1;
        const uint32_t kd = skn_smem_u32(K + ((size_t)buf * ATK + cr) * ks), vd = skn_smem_u32(V + ((size_t)buf * ATK + cr) * vs);
        for (int c = cc * 8; c < kp; c += 32) cp_async16(kd + c * 2, (c < src.k1 ? kr : kr2) + c, in);
#pragma unroll
        for (int c = cc * 8; c < DV; c += 32) cp_async16(vd + c * 2, vr + (c < vp ? c : 0), in && c < vp);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    {
        const int r = tid >> 1;
        const __nv_bfloat16 *q = a.q16 + (((int64_t)seq * st.T + t0 + (r < nq ? r : 0)) * a.heads + h) * kp;
        for (int c = (tid & 1) * 8; c < kp; c += 16) cp_async16(skn_smem_u32(Q + (size_t)r * ks + c), q + c, r < nq);
    }
    load_tile(0, 0);

    float o[DV / 8][4];
#pragma unroll
    for (int i = 0; i < DV / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    // a sink is one more key without a value: it opens the running maximum and, once per row, the sum
    const float L2E = 1.4426950408889634f, sink = a.sink ? a.sink[h] * L2E : -INFINITY, l0 = a.sink && (lane & 3) == 0 ? 1.f : 0.f;
    float mrow[2] = {sink, sink}, lrow[2] = {l0, l0};
    const int r0 = warp * 16 + (lane >> 2);
    const int qi[2] = {pf + r0, pf + r0 + 8};
    int qlo[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) qlo[i] = first_visible(a, qi[i]);
    const int w0 = pf + warp * 16, wlo = first_visible(a, w0), whi = first_visible(a, w0 + 15);
    const bool capped = a.softcap > 0.f;
    const float mul = capped ? 2.f * (a.scale / a.softcap) * L2E : a.scale * L2E, top = a.softcap * L2E;

    for (int t = 0; t < tiles; ++t) {
        const int buf = t & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (t + 1 < tiles) load_tile(t + 1, buf ^ 1);
        const int j0 = lo + t * ATK;
        // tiles that none of the warp's queries sees: past its last query, or in an earlier chunk than its first
        if (idle || j0 > w0 + 15 || j0 + ATK <= wlo) {
            __syncthreads();
            continue;
        }
        const bool masked = j0 + ATK - 1 > w0 || j0 < whi;               // some pair of this tile is invisible
        float s[ATK / 8][4];
#pragma unroll
        for (int i = 0; i < ATK / 8; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
        const __nv_bfloat16 *Kb = K + (size_t)buf * ATK * ks, *Vb = V + (size_t)buf * ATK * vs;
        {
            const uint32_t qa = skn_smem_u32(Q + (size_t)(warp * 16 + (lane & 15)) * ks + (lane >> 4) * 8),
                           ka = skn_smem_u32(Kb + (size_t)((lane & 7) + ((lane >> 4) << 3)) * ks + ((lane >> 3) & 1) * 8);
            uint32_t af[2][4], bf[2][ATK / 16][4];
            auto load = [&](int kk, int x) {
                ldsm4(af[x], qa + (uint32_t)kk * 2);
#pragma unroll
                for (int n = 0; n < ATK / 16; ++n) ldsm4(bf[x][n], ka + (uint32_t)(n * 16 * ks + kk) * 2);
            };
            load(0, 0);
            for (int kk = 0; kk < kp; kk += 32)
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    if (kk + 16 * x >= kp) break;
                    if (kk + 16 * x + 16 < kp) load(kk + 16 * x + 16, x ^ 1);
#pragma unroll
                    for (int n = 0; n < ATK / 16; ++n) {
                        mma_bf16(s[2 * n], af[x], bf[x][n][0], bf[x][n][1]);
                        mma_bf16(s[2 * n + 1], af[x], bf[x][n][2], bf[x][n][3]);
                    }
                }
        }
        if (capped) {
#pragma unroll
            for (int n = 0; n < ATK / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[n][e] = fmaf(-2.f * top, rcp(ex2(s[n][e] * mul) + 1.f), top);
        } else {
#pragma unroll
            for (int n = 0; n < ATK / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[n][e] *= mul;
        }
        if (masked) {
#pragma unroll
            for (int n = 0; n < ATK / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = e >> 1, j = j0 + n * 8 + (lane & 3) * 2 + (e & 1);
                    if (j > qi[i] || j < qlo[i]) s[n][e] = -INFINITY;
                }
        }
        float base[2];
        bool grown = false;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float mx = mrow[i];
#pragma unroll
            for (int n = 0; n < ATK / 8; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * i], s[n][2 * i + 1]));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            base[i] = mx;
            grown = grown || mx > mrow[i];
        }
        if (__any_sync(0xffffffffu, grown)) {
            float corr[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                corr[i] = ex2(mrow[i] - (base[i] == -INFINITY ? 0.f : base[i]));
                mrow[i] = base[i];
                lrow[i] *= corr[i];
            }
#pragma unroll
            for (int i = 0; i < DV / 8; ++i) {
                o[i][0] *= corr[0]; o[i][1] *= corr[0];
                o[i][2] *= corr[1]; o[i][3] *= corr[1];
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float b = base[i] == -INFINITY ? 0.f : base[i];
#pragma unroll
            for (int n = 0; n < ATK / 8; ++n) {
                s[n][2 * i] = ex2(s[n][2 * i] - b);
                s[n][2 * i + 1] = ex2(s[n][2 * i + 1] - b);
                lrow[i] += s[n][2 * i] + s[n][2 * i + 1];
            }
        }
#pragma unroll
        for (int kk = 0; kk < ATK / 16; ++kk) {
            uint32_t hi[4], lw[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float *w = s[2 * kk + (x >> 1)];
                const float w0 = w[(x & 1) * 2], w1 = w[(x & 1) * 2 + 1];
                hi[x] = pack_bf16(w0, w1);
                lw[x] = pack_bf16(w0 - __uint_as_float(hi[x] << 16), w1 - __uint_as_float(hi[x] & 0xFFFF0000u));
            }
            const uint32_t va = skn_smem_u32(Vb + (size_t)(kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * vs + (lane >> 4) * 8);
            uint32_t bf[2][4];
            ldsm4t(bf[0], va);
#pragma unroll
            for (int n = 0; n < DV / 16; ++n) {
                if (n + 1 < DV / 16) ldsm4t(bf[(n + 1) & 1], va + (uint32_t)(n + 1) * 32);
                const uint32_t(&b)[4] = bf[n & 1];
                mma_bf16(o[2 * n], lw, b[0], b[1]);
                mma_bf16(o[2 * n + 1], lw, b[2], b[3]);
                mma_bf16(o[2 * n], hi, b[0], b[1]);
                mma_bf16(o[2 * n + 1], hi, b[2], b[3]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        lrow[i] += __shfl_xor_sync(0xffffffffu, lrow[i], 1);
        lrow[i] += __shfl_xor_sync(0xffffffffu, lrow[i], 2);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = r0 + i * 8;
        if (r >= nq) continue;
        const float f = a.out_scale / lrow[i];
        const int64_t m = (int64_t)seq * st.T + t0 + r;
#pragma unroll
        for (int n = 0; n < DV / 8; ++n) {
            const int c = n * 8 + (lane & 3) * 2;
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (c + e < vdim) {
                    float v = o[n][i * 2 + e] * f;
                    if (a.gate) v *= __fdividef(1.f, 1.f + __expf(fminf(-__ldcg(a.gate + m * a.ld_gate + (int64_t)h * vdim + c + e), 80.f)));
                    put_out(a.out, m, (int64_t)h * vdim + c + e, v);
                }
        }
    }
}

template <int DV>
static cudaError_t launch_attn_tc(const skn_step &s, const skn_attn_args &a, const skn_attn_keys &k, cudaStream_t st) {
    auto kern = skn_attn_tc_kernel<DV>;
    const size_t smem = ((size_t)(ATQ + 2 * ATK) * (k.kp + 8) + (size_t)2 * ATK * (DV + 8)) * 2;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    // (whole chunks of query tiles: the kernel orders them)
    const int nt = (s.T + ATQ - 1) / ATQ, per = (a.chunk + ATQ - 1) / ATQ, pc = a.chunk > 0 && per < nt ? per : nt;
    return skn_launch_pdl(kern, dim3(a.heads, (nt + pc - 1) / pc * pc, s.n_seqs), dim3(AT_THREADS), smem, st, 1, a, s, k);
}

cudaError_t skn_launch_attn_tiles(const skn_step &s, const skn_attn_args &a, const skn_attn_keys &k, cudaStream_t st) {
    const int vp = k.vp;
    return vp <= 32 ? launch_attn_tc<32>(s, a, k, st) : vp <= 64 ? launch_attn_tc<64>(s, a, k, st) : vp <= 96 ? launch_attn_tc<96>(s, a, k, st)
           : vp <= 128 ? launch_attn_tc<128>(s, a, k, st) : vp <= 192 ? launch_attn_tc<192>(s, a, k, st) : launch_attn_tc<256>(s, a, k, st);
}

static skn_attn_keys cache_keys(const skn_kvcache *kv, int heads) {
    skn_attn_keys k = {};
    k.kp = k.k1 = kv->k_pitch; k.vp = kv->v_pitch; k.vdim = kv->v_dim; k.cap = kv->capacity; k.group = heads / kv->n_kv_heads;
    k.k = (const __nv_bfloat16 *)kv->d_k; k.k_row = kv->k_pitch; k.k_head = (int64_t)kv->capacity * kv->k_pitch; k.k_slot = k.k_head * kv->n_kv_heads;
    k.v = (const __nv_bfloat16 *)kv->d_v; k.v_row = kv->v_stride; k.v_head = (int64_t)kv->capacity * kv->v_stride; k.v_slot = k.v_head * kv->n_kv_heads;
    return k;
}

bool skn_attn_tiles_fit(int kp, int vp) { return kp <= 256 && vp <= 256; }
bool skn_chunk_attn_tc(const skn_kvcache *kv) { return kv->dtype == SKN_KV_BF16 && skn_attn_tiles_fit(kv->k_pitch, kv->v_pitch); }

// ---- retention in chunks --------------------------------------------------------------------------------------------
constexpr int RC = SKN_RET_CHUNK;

// what chunk c adds to the state by its end: sum over its tokens j of decay^(L - 1 - j) k_j v_j^T.  CTA: a 64 x 64 tile.
__global__ void __launch_bounds__(256)
skn_ret_chunk_kernel(skn_ret_args r, int T, int H, int dk, int dv, int vp, int nchunks, int vtiles) {
    __shared__ __align__(16) float kt[RC][64], vt[RC][64];
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int c = blockIdx.x, h = blockIdx.y % H, seq = blockIdx.y / H, i0 = (blockIdx.z / vtiles) * 64, j0 = (blockIdx.z % vtiles) * 64;
    const int t0 = c * RC, L = min(RC, T - t0);
    const float *pw = r.powers + (size_t)h * (RC + 1);
    const int64_t row0 = (int64_t)seq * T + t0;
    for (int i = threadIdx.x; i < RC * 64; i += 256) {
        const int t = i >> 6, d = i & 63;
        kt[t][d] = t < L && i0 + d < dk ? __ldcg(r.k + (row0 + t) * r.ld + (int64_t)h * dk + i0 + d) * pw[L - 1 - t] : 0.f;
        vt[t][d] = t < L && j0 + d < dv ? __ldcg(r.v + (row0 + t) * r.ld + (int64_t)h * dv + j0 + d) : 0.f;
    }
    __syncthreads();
    const int ti = (threadIdx.x >> 4) * 4, tj = (threadIdx.x & 15) * 4;
    float acc[4][4] = {};
    for (int t = 0; t < L; ++t) {
        const float4 a = *reinterpret_cast<const float4 *>(&kt[t][ti]), b = *reinterpret_cast<const float4 *>(&vt[t][tj]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    float *out = r.chunks + ((((size_t)seq * nchunks + c) * H + h) * dk) * vp;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (i0 + ti + i < dk && j0 + tj < vp)
            *reinterpret_cast<float4 *>(out + (size_t)(i0 + ti + i) * vp + j0 + tj) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// chunk sums -> states at the chunk starts (in place), and the state after the step
__global__ void __launch_bounds__(128)
skn_ret_scan_kernel(skn_ret_args r, skn_step st, float *S, int H, int dk, int vp, int nchunks) {
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int seq = blockIdx.y, slot = st.slot0 + seq, T = st.T;
    const int64_t per = (int64_t)H * dk * (vp / 4), i = (int64_t)blockIdx.x * 128 + threadIdx.x;
    if (i >= per) return;
    const int h = (int)(i / ((int64_t)dk * (vp / 4)));
    const float *pw = r.powers + (size_t)h * (RC + 1);
    float4 *p = reinterpret_cast<float4 *>(r.chunks) + (size_t)seq * nchunks * per + i;
    float4 *sp = reinterpret_cast<float4 *>(S) + (size_t)slot * per + i;
    float4 s = st.pos[slot] == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *sp;
    const float full = pw[RC], tail = pw[T - (nchunks - 1) * RC];
    for (int c0 = 0; c0 < nchunks; c0 += 8) {
        float4 a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c0 + u < nchunks) a[u] = __ldcg(p + (size_t)(c0 + u) * per);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (c0 + u < nchunks) {
                __stcg(p + (size_t)(c0 + u) * per, s);
                const float d = c0 + u == nchunks - 1 ? tail : full;
                s = make_float4(fmaf(d, s.x, a[u].x), fmaf(d, s.y, a[u].y), fmaf(d, s.z, a[u].z), fmaf(d, s.w, a[u].w));
            }
    }
    *sp = s;
}

// rows of outputs (at(row, column), in shared memory): divided by their root mean square, gated, scaled, stored
template <class AT>
__device__ __forceinline__ void ret_finish(const skn_ret_args &r, AT at, int64_t row0, int L, int h, int dv) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int R = 4, C = 4;                    // rows of a warp at a time, and columns per lane: their gates are asked for together
    for (int t0 = warp * R; t0 < L; t0 += 8 * R) {
        float ss[R] = {}, g[R][C];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int d = lane + 32 * c;
                g[i][c] = t0 + i < L && d < dv ? __ldcg(r.g + (row0 + t0 + i) * r.ld + (int64_t)h * dv + d) : 0.f;
            }
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (t0 + i < L)
                for (int d = lane; d < dv; d += 32) ss[i] = fmaf(at(t0 + i, d), at(t0 + i, d), ss[i]);
#pragma unroll
        for (int i = 0; i < R; ++i) ss[i] = r.out_scale / sqrtf(warp_sum(ss[i]) / (float)dv + r.eps);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int t = t0 + i;
            if (t >= L) break;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int d = lane + 32 * c;
                if (d < dv) put_out(r.out, row0 + t, (int64_t)h * dv + d, at(t, d) * ss[i] * (g[i][c] / (1.f + expf(-g[i][c]))));
            }
            for (int d = lane + 32 * C; d < dv; d += 32) {
                const float x = __ldcg(r.g + (row0 + t) * r.ld + (int64_t)h * dv + d);
                put_out(r.out, row0 + t, (int64_t)h * dv + d, at(t, d) * ss[i] * (x / (1.f + expf(-x))));
            }
        }
    }
}

// outputs of one chunk: o_i = sum_{j <= i} decay^(i - j) (q_i . k_j) v_j + decay^(i + 1) S^T q_i, then normalised and gated.
// smem (floats): A [RC][RC + 4] | x [32][RC + 4] | y [32][68] | o [RC][vw + 4], vw = dv rounded up to 64
static size_t ret_out_smem(int dv) { return ((size_t)RC * (RC + 4) + 32 * (RC + 4) + 32 * 68 + (size_t)RC * ((dv + 63) / 64 * 64 + 4)) * sizeof(float); }

__global__ void __launch_bounds__(256)
skn_ret_out_kernel(skn_ret_args r, int T, int H, int dk, int dv, int vp, int nchunks) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float pw[RC + 1];
    constexpr int AS = RC + 4;
    const int vw = (dv + 63) / 64 * 64, os = vw + 4;
    float *A = sm, *X = A + RC * AS, *Y = X + 32 * AS, *O = Y + 32 * 68;
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int tid = threadIdx.x, c = blockIdx.x, h = blockIdx.y, seq = blockIdx.z, t0 = c * RC, L = min(RC, T - t0);
    const int64_t row0 = (int64_t)seq * T + t0;
    const float *q = r.q + row0 * r.ld + (int64_t)h * dk, *k = r.k + row0 * r.ld + (int64_t)h * dk, *v = r.v + row0 * r.ld + (int64_t)h * dv;
    if (tid <= RC) pw[tid] = r.powers[(size_t)h * (RC + 1) + tid];
    const int ti = (tid >> 4) * 4, tj = (tid & 15) * 4;
    float acc[4][4] = {};
    for (int d0 = 0; d0 < dk; d0 += 32) {
        __syncthreads();
        for (int i = tid; i < RC * 32; i += 256) {
            const int t = i >> 5, d = i & 31;
            const bool in = t < L && d0 + d < dk;
            X[d * AS + t] = in ? __ldcg(q + (int64_t)t * r.ld + d0 + d) : 0.f;
            Y[d * 68 + t] = in ? __ldcg(k + (int64_t)t * r.ld + d0 + d) : 0.f;
        }
        __syncthreads();
#pragma unroll 8
        for (int d = 0; d < 32; ++d) {
            const float4 a = *reinterpret_cast<const float4 *>(X + d * AS + ti), b = *reinterpret_cast<const float4 *>(Y + d * 68 + tj);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
    }
    // stored transposed: A[j][i]
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) A[(tj + j) * AS + ti + i] = tj + j <= ti + i ? acc[i][j] * pw[ti + i - tj - j] : 0.f;
    const float *S = r.chunks + ((((size_t)seq * nchunks + c) * H + h) * dk) * vp;
    for (int v0 = 0; v0 < vw; v0 += 64) {
        float o[4][4] = {};
        for (int j0 = 0; j0 < RC; j0 += 32) {
            __syncthreads();
            for (int i = tid; i < 32 * 64; i += 256) {
                const int j = i >> 6, d = i & 63;
                Y[j * 68 + d] = j0 + j < L && v0 + d < dv ? __ldcg(v + (int64_t)(j0 + j) * r.ld + v0 + d) : 0.f;
            }
            __syncthreads();
#pragma unroll 8
            for (int j = 0; j < 32; ++j) {
                const float4 a = *reinterpret_cast<const float4 *>(A + (j0 + j) * AS + ti), b = *reinterpret_cast<const float4 *>(Y + j * 68 + tj);
                const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) o[x][y] = fmaf(av[x], bv[y], o[x][y]);
            }
        }
        float p[4][4] = {};
        for (int d0 = 0; d0 < dk; d0 += 32) {
            __syncthreads();
            for (int i = tid; i < RC * 32; i += 256) {
                const int t = i >> 5, d = i & 31;
                X[d * AS + t] = t < L && d0 + d < dk ? __ldcg(q + (int64_t)t * r.ld + d0 + d) : 0.f;
            }
            for (int i = tid; i < 32 * 64; i += 256) {
                const int d = i >> 6, x = i & 63;
                Y[d * 68 + x] = d0 + d < dk && v0 + x < vp ? __ldcg(S + (size_t)(d0 + d) * vp + v0 + x) : 0.f;
            }
            __syncthreads();
#pragma unroll 8
            for (int d = 0; d < 32; ++d) {
                const float4 a = *reinterpret_cast<const float4 *>(X + d * AS + ti), b = *reinterpret_cast<const float4 *>(Y + d * 68 + tj);
                const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) p[x][y] = fmaf(av[x], bv[y], p[x][y]);
            }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) O[(ti + x) * os + v0 + tj + y] = fmaf(pw[ti + x + 1], p[x][y], o[x][y]);
    }
    __syncthreads();
    ret_finish(r, [&](int t, int d) { return O[t * os + d]; }, row0, L, h, dv);
}

// ---- retention chunks on the tensor cores -----------------------------------------------------------------------------
// Every fp32 operand enters as three bf16 terms (skn_mma.cuh), split once where it is stored to shared memory, and sums over 32 elements are
// added in fp32.  (Two tf32 terms split where fragments were read, a dozen instructions and six scalar loads per product, were bound by
// those: 2048 tokens, 8 heads of 128 x 128: outputs 61 us, chunk sums 22; now 43 and 18.)  The 32 columns of a block of a
// warp's tiles share the fragments of its 16 rows; row strides are 16 bytes off a multiple of 128.
constexpr int RT2 = 128;              // columns of a tile
constexpr int RTS = (RT2 + 8) * 2;    // bytes of a row of its planes

// planes of [rows][32 cols' words...]: pair (x, y) at `at` of the first
__device__ __forceinline__ void put_terms(uint8_t *at, int plane, float x, float y) {
    uint32_t w[3];
    split_terms(x, y, w);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t *>(at + p * plane) = w[p];
}
// elements c, c + 1 of a row of n; even: rows start on 8 bytes and n is even
__device__ __forceinline__ float2 pair_at(const float *row, int c, int n, bool even) {
    if (even) return c < n ? __ldcg(reinterpret_cast<const float2 *>(row + c)) : make_float2(0.f, 0.f);
    return make_float2(c < n ? __ldcg(row + c) : 0.f, c + 1 < n ? __ldcg(row + c + 1) : 0.f);
}
__device__ __forceinline__ bool pairs_even(const float *p, int64_t ld, int n) { return !((reinterpret_cast<uintptr_t>(p) & 7) | (ld & 1) | (n & 1)); }

// what chunk c adds to the state by its end (see skn_ret_chunk_kernel).  CTA: a 128 x 128 tile, a warp 16 of its rows.
__global__ void __launch_bounds__(256, 2)
skn_ret_chunk_tc_kernel(skn_ret_args r, int T, int H, int dk, int dv, int vp, int nchunks, int vtiles) {
    extern __shared__ __align__(16) uint8_t smb[];
    __shared__ float pw[RC + 1];
    constexpr int PL = RC * RTS;
    uint8_t *Ks = smb, *Vs = smb + 3 * PL;
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int c = blockIdx.x, h = blockIdx.y % H, seq = blockIdx.y / H, i0 = (blockIdx.z / vtiles) * RT2, j0 = (blockIdx.z % vtiles) * RT2;
    const int t0 = c * RC, L = min(RC, T - t0), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t row0 = (int64_t)seq * T + t0;
    const float *k = r.k + row0 * r.ld + (int64_t)h * dk + i0, *v = r.v + row0 * r.ld + (int64_t)h * dv + j0;
    const bool ke = pairs_even(k, r.ld, dk), ve = pairs_even(v, r.ld, dv);
    if (tid <= RC) pw[tid] = r.powers[(size_t)h * (RC + 1) + tid];
    __syncthreads();
    for (int t1 = tid >> 6; t1 < RC; t1 += 32) {
        float2 a[8], b[8];
        const int d = (tid & 63) * 2;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = t1 + 4 * i;
            a[i] = t < L ? pair_at(k + (int64_t)t * r.ld, d, dk - i0, ke) : make_float2(0.f, 0.f);
            b[i] = t < L ? pair_at(v + (int64_t)t * r.ld, d, dv - j0, ve) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = t1 + 4 * i;
            const float f = t < L ? pw[L - 1 - t] : 0.f;
            put_terms(Ks + t * RTS + d * 2, PL, a[i].x * f, a[i].y * f);
            put_terms(Vs + t * RTS + d * 2, PL, b[i].x, b[i].y);
        }
    }
    __syncthreads();
    if (i0 + warp * 16 >= dk) return;
    float *out = r.chunks + ((((size_t)seq * nchunks + c) * H + h) * dk) * vp;
#pragma unroll 1
    for (int nb = 0; nb < RT2 / 32 && j0 + nb * 32 < vp; ++nb) {
        float acc[4][4] = {};
#pragma unroll
        for (int kk = 0; kk < RC; kk += 32) {
            float s[4][4], m[4][4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                uint32_t af[3][4], bf[2][3][4];
                const int t = kk + 16 * x;
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ldsm4t(af[p], skn_smem_u32(Ks + p * PL + (t + (lane & 7) + ((lane >> 4) << 3)) * RTS + (warp * 16 + ((lane >> 3) & 1) * 8) * 2));
                    const uint32_t vb = skn_smem_u32(Vs + p * PL + (t + (lane & 7) + ((lane >> 3) & 1) * 8) * RTS + (nb * 32 + (lane >> 4) * 8) * 2);
                    ldsm4t(bf[0][p], vb);
                    ldsm4t(bf[1][p], vb + 32);
                }
                if (x == 0) mma_terms<3, true>(s, m, af, bf);
                else mma_terms<3, false>(s, m, af, bf);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[n][e] += m[n][e] + s[n][e];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int row = i0 + warp * 16 + (lane >> 2) + e * 8;
            if (row >= dk) continue;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int col = j0 + nb * 32 + n * 8 + (lane & 3) * 2;
                if (col < vp) *reinterpret_cast<float2 *>(out + (size_t)row * vp + col) = make_float2(acc[n][2 * e], acc[n][2 * e + 1]);
            }
        }
    }
}

// Outputs of one chunk (see skn_ret_out_kernel).  Bytes of shared memory: planes of q [RC][dkp + 8] | of the scores [RC][RC + 8] | of a tile
// [32][RT2 + 8] (keys, then rows of the state and values) | the fp32 outputs of all blocks of RT2 columns but the last [RC][vw - RT2 + 4].  Those of
// the last block [RC][RT2 + 4] lie over the planes, which nothing reads any more: with all of them behind, 128 x 512, 256 x 384 and 352 x 256
// (keys x values) would not fit.  A warp owns 16 rows and half of a tile's columns.
struct ret_out_layout {
    int dkp, vw, lq, la, scores, tile, out, bytes;                      // row strides and offsets in bytes
    __host__ __device__ ret_out_layout(int dk, int dv) {
        dkp = (dk + 31) / 32 * 32;
        vw = (dv + RT2 - 1) / RT2 * RT2;
        lq = (dkp + 8) * 2;
        la = (RC + 8) * 2;
        scores = 3 * RC * lq;
        tile = scores + 3 * RC * la;
        const int end = tile + 3 * 32 * RTS, last = RC * (RT2 + 4) * 4;
        out = end > last ? end : last;
        bytes = out + (vw > RT2 ? RC * (vw - RT2 + 4) * 4 : 0);
    }
};
constexpr size_t RET_SMEM_MAX = 226 * 1024;
static size_t ret_out_tc_smem(int dk, int dv) { return (size_t)ret_out_layout(dk, dv).bytes; }

__global__ void __launch_bounds__(256, 2)
skn_ret_out_tc_kernel(skn_ret_args r, int T, int H, int dk, int dv, int vp, int nchunks) {
    extern __shared__ __align__(16) uint8_t smb[];
    __shared__ float pw[RC + 1];
    const ret_out_layout l(dk, dv);
    uint8_t *Q = smb, *A = smb + l.scores, *B = smb + l.tile;
    float *O = reinterpret_cast<float *>(smb + l.out), *P = reinterpret_cast<float *>(smb);     // outputs up to column `first`, those of the last block
    const int QP = RC * l.lq, AP = RC * l.la, BP = 32 * RTS, first = l.vw - RT2, os = first + 4;
    constexpr int ps = RT2 + 4;
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = blockIdx.x, h = blockIdx.y, seq = blockIdx.z, t0 = c * RC, L = min(RC, T - t0);
    const int64_t row0 = (int64_t)seq * T + t0;
    const float *q = r.q + row0 * r.ld + (int64_t)h * dk, *k = r.k + row0 * r.ld + (int64_t)h * dk, *v = r.v + row0 * r.ld + (int64_t)h * dv;
    const float *S = r.chunks + ((((size_t)seq * nchunks + c) * H + h) * dk) * vp;
    const bool qe = pairs_even(q, r.ld, dk), ke = pairs_even(k, r.ld, dk), ve = pairs_even(v, r.ld, dv), se = pairs_even(S, vp, vp);
    if (tid <= RC) pw[tid] = r.powers[(size_t)h * (RC + 1) + tid];
    const int m0 = (warp & 3) * 16, half = warp >> 2, g = lane >> 2, t = lane & 3;
    // columns [from, end) of `rows` rows; a warp's 32 lanes take the words of 64 columns of a row
    auto rows_in = [&](uint8_t *to, int stride, int plane, const float *src, bool even, int first, int rows, int from, int end) {
        for (int d0 = from; d0 < end; d0 += 64) {
            const int d = d0 + 2 * lane;
            if (d >= end) continue;
            for (int i = warp; i < rows; i += 64) {
                float2 x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int y = first + i + 8 * j;
                    x[j] = i + 8 * j < rows && y < L ? pair_at(src + (int64_t)y * r.ld, d, dk, even) : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (i + 8 * j < rows) put_terms(to + (i + 8 * j) * stride + (d - from) * 2, plane, x[j].x, x[j].y);
            }
        }
    };
    rows_in(Q, l.lq, QP, q, qe, 0, RC, 0, l.dkp);
#pragma unroll 1
    for (int kt = 0; kt < RC; kt += 32) {
        const int n0 = kt + half * 16;
        float s[2][4] = {}, rest[2][4] = {};
#pragma unroll 1
        for (int d0 = 0; d0 < l.dkp; d0 += RT2) {
            const int d1 = min(d0 + RT2, l.dkp);
            if (kt | d0) __syncthreads();          // the keys before are done with
            rows_in(B, RTS, BP, k, ke, kt, 32, d0, d1);
            __syncthreads();
            if (n0 > m0 + 15) continue;            // every pair of this tile lies in the future
#pragma unroll 1
            for (int kk = d0; kk < d1; kk += 32) {
                float sm[2][4], mn[2][4];
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    uint32_t af[3][4], bf[1][3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        ldsm4(af[p], skn_smem_u32(Q + p * QP + (m0 + (lane & 15)) * l.lq + (kk + 16 * x + (lane >> 4) * 8) * 2));
                        ldsm4(bf[0][p], skn_smem_u32(B + p * BP + (half * 16 + (lane & 7) + ((lane >> 4) << 3)) * RTS + (kk - d0 + 16 * x + ((lane >> 3) & 1) * 8) * 2));
                    }
                    if (x == 0) mma_terms<3, true>(sm, mn, af, bf);
                    else mma_terms<3, false>(sm, mn, af, bf);
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        s[n][e] += mn[n][e];
                        rest[n][e] += sm[n][e];
                    }
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = m0 + g + e * 8, j = n0 + n * 8 + t * 2;
                const float x = j <= i ? (s[n][2 * e] + rest[n][2 * e]) * pw[i - j] : 0.f, y = j + 1 <= i ? (s[n][2 * e + 1] + rest[n][2 * e + 1]) * pw[i - j - 1] : 0.f;
                put_terms(A + i * l.la + j * 2, AP, x, y);
            }
    }
    for (int v0 = 0; v0 < l.vw; v0 += RT2) {
        float o[8][4] = {};
        const int c0 = half * (RT2 / 2);
        // tiles of 32 rows: the state's first, then the chunk's values
        const int stiles = l.dkp / 32, tiles = stiles + (L + 31) / 32;
        float2 pre[8];
        auto fetch = [&](int x) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int row = (x < stiles ? x : x - stiles) * 32 + (tid >> 6) + i * 4, col = v0 + (tid & 63) * 2;
                if (x < stiles) pre[i] = row < dk ? pair_at(S + (size_t)row * vp, col, vp, se) : make_float2(0.f, 0.f);
                else pre[i] = row < L ? pair_at(v + (int64_t)row * r.ld, col, dv, ve) : make_float2(0.f, 0.f);
            }
        };
        fetch(0);
#pragma unroll 1
        for (int x = 0; x < tiles; ++x) {
            __syncthreads();                       // the tile before (or the keys) is done with
#pragma unroll
            for (int i = 0; i < 8; ++i) put_terms(B + ((tid >> 6) + i * 4) * RTS + (tid & 63) * 4, BP, pre[i].x, pre[i].y);
            __syncthreads();
            if (x + 1 < tiles) fetch(x + 1);
            if (x == stiles)
#pragma unroll
                for (int n = 0; n < 8; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[n][e] *= pw[m0 + g + (e >> 1) * 8 + 1];
            const bool state = x < stiles;
            if (!state && (x - stiles) * 32 > m0 + 15) continue;
            const uint8_t *a = state ? Q + x * 64 : A + (x - stiles) * 64;
            const int lda = state ? l.lq : l.la, pla = state ? QP : AP;
#pragma unroll
            for (int nb = 0; nb < 2; ++nb) {
                float sm[4][4], mn[4][4];
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    uint32_t af[3][4], bf[2][3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        ldsm4(af[p], skn_smem_u32(a + p * pla + (m0 + (lane & 15)) * lda + (y * 16 + (lane >> 4) * 8) * 2));
                        const uint32_t bb = skn_smem_u32(B + p * BP + (y * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * RTS + (c0 + nb * 32 + (lane >> 4) * 8) * 2);
                        ldsm4t(bf[0][p], bb);
                        ldsm4t(bf[1][p], bb + 32);
                    }
                    if (y == 0) mma_terms<3, true>(sm, mn, af, bf);
                    else mma_terms<3, false>(sm, mn, af, bf);
                }
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[4 * nb + n][e] += mn[n][e] + sm[n][e];
            }
        }
        __syncthreads();                           // the last block's outputs lie over q, the scores and the tile
        float *to = v0 < first ? O + v0 : P;
        const int ts = v0 < first ? os : ps;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                *reinterpret_cast<float2 *>(to + (m0 + g + e * 8) * ts + c0 + n * 8 + t * 2) = make_float2(o[n][2 * e], o[n][2 * e + 1]);
    }
    __syncthreads();
    ret_finish(r, [&](int t, int d) { return d < first ? O[t * os + d] : P[t * ps + d - first]; }, row0, L, h, dv);
}

template <class CT>
static cudaError_t launch_prep(const skn_step &s, const skn_attn_args *a, const skn_ret_args *r, cudaStream_t st) {
    prep_args p = {};
    skn_attn_args aa = {};
    skn_ret_args rr = {};
    CT *kc = nullptr, *vc = nullptr;
    p.kp = p.vp = 16; p.cap = 1; p.dim = p.vdim = p.rdk = 1;
    if (a) {
        aa = *a;
        p.H = a->heads; p.G = a->kv->n_kv_heads; p.dim = a->kv->head_dim; p.vdim = a->kv->v_dim; p.kp = a->kv->k_pitch; p.vp = a->kv->v_pitch;
        p.cap = a->kv->capacity;
        kc = (CT *)a->kv->d_k;
        vc = (CT *)a->kv->d_v;
        if (!skn_chunk_attn_tc(a->kv)) aa.q16 = nullptr;
    }
    if (r) {
        rr = *r;
        p.RH = r->state->heads; p.rdk = r->state->k_dim;
    }
    const int keys = p.kp > p.vdim ? p.kp : p.vdim, widest = keys > p.rdk ? keys : p.rdk;
    if (widest <= 256 && head_prep_aligned(a ? &aa : nullptr, r, p)) {
        auto kern = widest <= 128 ? skn_head_prep_vec_kernel<CT, 1> : skn_head_prep_vec_kernel<CT, 2>;
        return skn_launch_pdl(kern, dim3(s.n_seqs * s.T), dim3(256), 0, st, 1, aa, rr, s, p, kc, vc);
    }
    const size_t smem = (size_t)8 * (p.kp > p.rdk ? p.kp : p.rdk) * sizeof(float);
    return skn_launch_pdl(skn_head_prep_kernel<CT>, dim3(s.n_seqs * s.T), dim3(256), smem, st, 1, aa, rr, s, p, kc, vc);
}

cudaError_t skn_launch_mix_prefill(skn_ctx *, const skn_step &s, const skn_attn_args *a, const skn_ret_args *r, cudaStream_t st) {
    cudaError_t e = a && a->kv->dtype == SKN_KV_BF16 ? launch_prep<__nv_bfloat16>(s, a, r, st) : launch_prep<float>(s, a, r, st);
    if (e != cudaSuccess) return e;
    if (a) {
        if (skn_chunk_attn_tc(a->kv)) {
            e = skn_launch_attn_tiles(s, *a, cache_keys(a->kv, a->heads), st);
        } else {
            e = launch_split(s, a, nullptr, true, st);
        }
        if (e != cudaSuccess) return e;
    }
    if (r) {
        const int H = r->state->heads, dk = r->state->k_dim, dv = r->state->v_dim, vp = r->state->v_pitch;
        const int nchunks = (s.T + RC - 1) / RC;
        const bool tc = !r->exact && ret_out_tc_smem(dk, dv) <= RET_SMEM_MAX;
        const int tile = tc ? RT2 : 64, kt = (dk + tile - 1) / tile, vt = (dv + tile - 1) / tile;
        const dim3 cgrid(nchunks, H * s.n_seqs, kt * vt), ogrid(nchunks, H, s.n_seqs);
        if (tc) {
            e = cudaFuncSetAttribute(skn_ret_chunk_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * RC * RTS);
            if (e != cudaSuccess) return e;
            e = skn_launch_pdl(skn_ret_chunk_tc_kernel, cgrid, dim3(256), (size_t)6 * RC * RTS, st, 1, *r, s.T, H, dk, dv, vp, nchunks, vt);
        } else {
            e = skn_launch_pdl(skn_ret_chunk_kernel, cgrid, dim3(256), 0, st, 1, *r, s.T, H, dk, dv, vp, nchunks, vt);
        }
        if (e != cudaSuccess) return e;
        const int64_t per = (int64_t)H * dk * (vp / 4);
        e = skn_launch_pdl(skn_ret_scan_kernel, dim3((unsigned)((per + 127) / 128), s.n_seqs), dim3(128), 0, st, 1, *r, s, r->state->d, H, dk, vp, nchunks);
        if (e != cudaSuccess) return e;
        if (tc) {
            e = cudaFuncSetAttribute(skn_ret_out_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RET_SMEM_MAX);
            if (e != cudaSuccess) return e;
            e = skn_launch_pdl(skn_ret_out_tc_kernel, ogrid, dim3(256), ret_out_tc_smem(dk, dv), st, 1, *r, s.T, H, dk, dv, vp, nchunks);
        } else {
            e = cudaFuncSetAttribute(skn_ret_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            if (e != cudaSuccess) return e;
            e = skn_launch_pdl(skn_ret_out_kernel, ogrid, dim3(256), ret_out_smem(dv), st, 1, *r, s.T, H, dk, dv, vp, nchunks);
        }
    }
    return e;
}

// ---- angles and positions --------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
skn_rot_table_kernel(skn_step st, const double *__restrict__ freq, int half, float2 *out, int ld) {
    skn_pdl_launch_dependents();
    skn_pdl_wait();
    const int m = blockIdx.x, pos = st.pos[st.slot0 + m / st.T] + m % st.T;
    for (int i = threadIdx.x; i < half; i += 128) {
        // an fp32 product would be off by pos * 2^-24: the angle is formed and reduced in double
        const double a = (double)pos * freq[i], turns = rint(a * 0.15915494309189535);
        float s, c;
        sincosf((float)(a - turns * 6.283185307179586), &s, &c);
        out[(int64_t)m * ld + i] = make_float2(c, s);
    }
}

cudaError_t skn_launch_rot_table(const skn_step &s, const double *freq, int half, float2 *out, int ld, cudaStream_t st) {
    return skn_launch_pdl(skn_rot_table_kernel, dim3(s.n_seqs * s.T), dim3(128), 0, st, 1, s, freq, half, out, ld);
}

// Triggers no launch early: what follows it in the stream (the next step) starts when every launch before it is done, so a
// step's kernels may read what earlier steps left (states, caches) ahead of their own dependency wait.
__global__ void skn_advance_kernel(skn_step st, int32_t *pos, int32_t *status) {
    skn_pdl_wait();
    for (int s = threadIdx.x; s < st.n_seqs; s += blockDim.x) {
        const int p = pos[st.slot0 + s] + st.T;
        if (p > st.max_pos) atomicExch(status, SKN_ERR_SHAPE);
        pos[st.slot0 + s] = min(p, st.max_pos);
    }
}

cudaError_t skn_launch_advance(const skn_step &s, int32_t *pos, int32_t *status, cudaStream_t st) {
    return skn_launch_pdl(skn_advance_kernel, dim3(1), dim3(128), 0, st, 1, s, pos, status);
}

// ---- host-pointer forms ------------------------------------------------------------------------------------------------
namespace {
// carves 256-byte aligned pieces out of one allocation; first run with base NULL to measure
struct Arena {
    uint8_t *base;
    size_t used;
    template <class T> T *take(size_t n) {
        T *p = reinterpret_cast<T *>(base + used);
        used += (n * sizeof(T) + 255) / 256 * 256;
        return p;
    }
};
}

static int32_t upload(skn_ctx *ctx, void *dst, const void *src, size_t bytes) {
    SKN_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return SKN_OK;
}

static int32_t check_step(skn_ctx *ctx, int32_t slots, int32_t seq0, int32_t n_seqs, int32_t T, const int32_t *pos, int32_t max_ctx) {
    if (seq0 < 0 || n_seqs < 1 || T < 1 || seq0 + n_seqs > slots || !pos) return skn_fail(ctx, SKN_ERR_ARG, "sequences outside the cache, or no positions");
    for (int s = 0; s < n_seqs; ++s)
        if (pos[s] < 0 || pos[s] + T > max_ctx) return skn_fail(ctx, SKN_ERR_SHAPE, "context of %d tokens exceeded", max_ctx);
    return SKN_OK;
}

void skn_rot_freqs(double base, int dims, double *out) {
    for (int i = 0; i < dims / 2; ++i) out[i] = pow(base, -2.0 * i / dims);
}

void skn_decay_powers(const double *decay, int heads, float *out) {
    for (int h = 0; h < heads; ++h)
        for (int n = 0; n <= SKN_RET_CHUNK; ++n) out[h * (SKN_RET_CHUNK + 1) + n] = (float)pow(decay[h], n);
}

int32_t skn_check_attn_spec(skn_ctx *ctx, const skn_attn_spec *a) {
    if (a->heads < 1 || a->kv_heads < 1 || a->dim < 1 || a->vdim < 1 || a->chunk < 0 || a->window < 0 || (a->chunk && a->window)) return skn_fail(ctx, SKN_ERR_ARG, "invalid attention geometry");
    if (a->heads % a->kv_heads || a->rot_dims < 0 || a->rot_dims % 2 || a->rot_dims > a->dim || a->dim > SKN_ATTN_MAX_DIM || a->vdim > SKN_ATTN_MAX_DIM)
        return skn_fail(ctx, SKN_ERR_SHAPE, "Shapes do not align.");
    return SKN_OK;
}

int32_t skn_check_retention_spec(skn_ctx *ctx, const skn_retention_spec *r) {
    if (r->heads < 1 || r->dim < 1 || r->vdim < 1 || !r->decay) return skn_fail(ctx, SKN_ERR_ARG, "invalid retention geometry");
    if (r->rot_dims < 0 || r->rot_dims % 2 || r->rot_dims > r->dim || r->dim > SKN_ATTN_MAX_DIM || r->vdim > SKN_ATTN_MAX_DIM)
        return skn_fail(ctx, SKN_ERR_SHAPE, "Shapes do not align.");
    return SKN_OK;
}

extern "C" {

int32_t skn_chunk_attn(skn_kvcache *kv, const skn_attn_spec *spec, int32_t seq0, int32_t n_seqs, int32_t T, const int32_t *pos_host,
                       int32_t max_ctx, const float *q_gain_host, const float *k_gain_host, const float *q_host, const float *k_host,
                       const float *v_host, const float *sink_host, float *out_host) {
    if (!skn_kv_ok(kv) || !kv->by_position) return skn_fail(nullptr, SKN_ERR_BAD_HANDLE, "not a position-addressed cache");
    skn_ctx *ctx = kv->ctx;
    SKN_ENTER(ctx);
    if (!spec || !q_host || !k_host || !v_host || !out_host || !q_gain_host != !k_gain_host) return skn_fail(ctx, SKN_ERR_ARG, "NULL argument");
    int32_t rc = skn_check_attn_spec(ctx, spec);
    if (rc) return rc;
    if (spec->kv_heads != kv->n_kv_heads || spec->dim != kv->head_dim || spec->vdim != kv->v_dim) return skn_fail(ctx, SKN_ERR_SHAPE, "Shapes do not align.");
    if ((rc = check_step(ctx, kv->batch, seq0, n_seqs, T, pos_host, max_ctx))) return rc;
    const int span = spec->chunk > 0 ? spec->chunk : spec->window;
    const int need = span > 0 && span + T < max_ctx ? span + T : max_ctx;
    if (kv->capacity < need) return skn_fail(ctx, SKN_ERR_SHAPE, "this step needs a cache of %d tokens", need);
    SKN_CUDA(ctx, cudaSetDevice(ctx->device));
    const int H = spec->heads, G = spec->kv_heads, D = spec->dim, V = spec->vdim, M = n_seqs * T, half = spec->rot_dims / 2;
    float *q, *out, *scratch, *qg, *kg, *sink;
    int32_t *pos;
    unsigned *tickets;
    float2 *rot;
    double *freq;
    __nv_bfloat16 *q16;
    const size_t nscr = skn_attn_scratch(M, H, V, span, max_ctx);
    Arena a = {nullptr, 0};
    for (int pass = 0; pass < 2; ++pass) {
        q = a.take<float>((size_t)M * ((size_t)H * D + (size_t)G * (D + V)));
        out = a.take<float>((size_t)M * H * V); scratch = a.take<float>(nscr); qg = a.take<float>(D); kg = a.take<float>(D); sink = a.take<float>(H);
        pos = a.take<int32_t>(kv->batch); tickets = a.take<unsigned>((size_t)M * H); rot = a.take<float2>((size_t)M * (half + 1));
        freq = a.take<double>(half + 1); q16 = a.take<__nv_bfloat16>((size_t)M * H * kv->k_pitch);
        if (pass == 0) {
            if ((rc = skn_stage_reserve(ctx, &ctx->d_scratch, &ctx->d_scratch_bytes, a.used))) return rc;
            a.base = (uint8_t *)ctx->d_scratch;
            a.used = 0;
        }
    }
    double hf[SKN_ATTN_MAX_DIM / 2 + 1];
    skn_rot_freqs(spec->rot_base, spec->rot_dims, hf);
    if ((rc = upload(ctx, pos + seq0, pos_host, sizeof(int32_t) * n_seqs)) || (rc = upload(ctx, freq, hf, sizeof(double) * half))) return rc;
    if (q_gain_host && ((rc = upload(ctx, qg, q_gain_host, sizeof(float) * D)) || (rc = upload(ctx, kg, k_gain_host, sizeof(float) * D)))) return rc;
    if (sink_host && (rc = upload(ctx, sink, sink_host, sizeof(float) * H))) return rc;
    SKN_CUDA(ctx, cudaMemsetAsync(tickets, 0, (size_t)M * H * sizeof(unsigned), ctx->stream));
    // joint rows [q | k | v], as the projection of a decoder leaves them
    const int64_t ld = (int64_t)H * D + (int64_t)G * (D + V);
    SKN_CUDA(ctx, cudaMemcpy2DAsync(q, ld * 4, q_host, (size_t)H * D * 4, (size_t)H * D * 4, M, cudaMemcpyHostToDevice, ctx->stream));
    SKN_CUDA(ctx, cudaMemcpy2DAsync(q + H * D, ld * 4, k_host, (size_t)G * D * 4, (size_t)G * D * 4, M, cudaMemcpyHostToDevice, ctx->stream));
    SKN_CUDA(ctx, cudaMemcpy2DAsync(q + H * D + G * D, ld * 4, v_host, (size_t)G * V * 4, (size_t)G * V * 4, M, cudaMemcpyHostToDevice, ctx->stream));
    const skn_step st = {seq0, n_seqs, T, pos, max_ctx};
    if (half) SKN_CUDA(ctx, skn_launch_rot_table(st, freq, half, rot, half, ctx->stream));
    skn_attn_args x = {};
    x.kv = kv; x.heads = H; x.chunk = spec->chunk; x.window = spec->window; x.sink = sink_host ? sink : nullptr; x.scale = spec->scale; x.softcap = spec->softcap; x.eps = spec->eps;
    x.q_gain = q_gain_host ? qg : nullptr; x.k_gain = q_gain_host ? kg : nullptr;
    x.rot = skn_rot{rot, half, half};
    x.q = q; x.k = q + H * D; x.v = q + H * D + G * D; x.ld = ld;
    x.out_scale = 1.f; x.out = skn_rows_out{out, (int64_t)H * V, nullptr, 0};
    x.scratch = scratch; x.tickets = tickets; x.q16 = q16;
    SKN_CUDA(ctx, T == 1 ? skn_launch_mix_decode(ctx, st, &x, nullptr, ctx->stream) : skn_launch_mix_prefill(ctx, st, &x, nullptr, ctx->stream));
    SKN_CUDA(ctx, cudaMemcpyAsync(out_host, out, (size_t)M * H * V * 4, cudaMemcpyDeviceToHost, ctx->stream));
    return skn_sync(ctx);
}

int32_t skn_retention(skn_state *s, const skn_retention_spec *spec, int32_t seq0, int32_t n_seqs, int32_t T, const int32_t *pos_host,
                      int32_t max_ctx, const float *q_host, const float *k_host, const float *v_host, const float *g_host, float *out_host) {
    if (!s || s->magic != SKN_MAGIC_STATE || !skn_ctx_ok(s->ctx)) return skn_fail(nullptr, SKN_ERR_BAD_HANDLE, "bad state handle");
    skn_ctx *ctx = s->ctx;
    SKN_ENTER(ctx);
    if (!spec || !q_host || !k_host || !v_host || !g_host || !out_host) return skn_fail(ctx, SKN_ERR_ARG, "NULL argument");
    int32_t rc = skn_check_retention_spec(ctx, spec);
    if (rc) return rc;
    if (spec->heads != s->heads || spec->dim != s->k_dim || spec->vdim != s->v_dim) return skn_fail(ctx, SKN_ERR_SHAPE, "Shapes do not align.");
    if ((rc = check_step(ctx, s->slots, seq0, n_seqs, T, pos_host, max_ctx))) return rc;
    SKN_CUDA(ctx, cudaSetDevice(ctx->device));
    const int H = spec->heads, D = spec->dim, V = spec->vdim, M = n_seqs * T, half = spec->rot_dims / 2, nch = (T + SKN_RET_CHUNK - 1) / SKN_RET_CHUNK;
    const int64_t ld = (int64_t)H * (2 * D + 2 * V);
    float *rows, *out, *pw, *chunks;
    int32_t *pos;
    float2 *rot;
    double *freq;
    Arena a = {nullptr, 0};
    for (int pass = 0; pass < 2; ++pass) {
        rows = a.take<float>((size_t)M * ld); out = a.take<float>((size_t)M * H * V); pw = a.take<float>((size_t)H * (SKN_RET_CHUNK + 1));
        chunks = a.take<float>((size_t)n_seqs * nch * H * D * s->v_pitch); pos = a.take<int32_t>(s->slots);
        rot = a.take<float2>((size_t)M * (half + 1)); freq = a.take<double>(half + 1);
        if (pass == 0) {
            if ((rc = skn_stage_reserve(ctx, &ctx->d_scratch, &ctx->d_scratch_bytes, a.used))) return rc;
            a.base = (uint8_t *)ctx->d_scratch;
            a.used = 0;
        }
    }
    double hf[SKN_ATTN_MAX_DIM / 2 + 1];
    skn_rot_freqs(spec->rot_base, spec->rot_dims, hf);
    float *hp = (float *)malloc((size_t)H * (SKN_RET_CHUNK + 1) * sizeof(float));
    if (!hp) return skn_fail(ctx, SKN_ERR_OOM, "host allocation failed");
    skn_decay_powers(spec->decay, H, hp);
    rc = upload(ctx, pw, hp, (size_t)H * (SKN_RET_CHUNK + 1) * sizeof(float));
    cudaStreamSynchronize(ctx->stream);
    free(hp);
    if (rc || (rc = upload(ctx, pos + seq0, pos_host, sizeof(int32_t) * n_seqs)) || (rc = upload(ctx, freq, hf, sizeof(double) * half))) return rc;
    const float *src[4] = {q_host, k_host, v_host, g_host};
    const size_t w[4] = {(size_t)H * D, (size_t)H * D, (size_t)H * V, (size_t)H * V};
    float *dst = rows;
    for (int i = 0; i < 4; ++i) {
        SKN_CUDA(ctx, cudaMemcpy2DAsync(dst, ld * 4, src[i], w[i] * 4, w[i] * 4, M, cudaMemcpyHostToDevice, ctx->stream));
        dst += w[i];
    }
    const skn_step st = {seq0, n_seqs, T, pos, max_ctx};
    if (half) SKN_CUDA(ctx, skn_launch_rot_table(st, freq, half, rot, half, ctx->stream));
    skn_ret_args x = {};
    x.state = s; x.eps = spec->eps; x.rot = skn_rot{rot, half, half}; x.k_scale = (float)(1.0 / sqrt((double)D)); x.powers = pw;
    x.q = rows; x.k = rows + w[0]; x.v = rows + 2 * w[0]; x.g = rows + 2 * w[0] + w[2]; x.ld = ld;
    x.out_scale = 1.f; x.out = skn_rows_out{out, (int64_t)H * V, nullptr, 0}; x.exact = spec->exact != 0; x.chunks = chunks;
    SKN_CUDA(ctx, T == 1 ? skn_launch_mix_decode(ctx, st, nullptr, &x, ctx->stream) : skn_launch_mix_prefill(ctx, st, nullptr, &x, ctx->stream));
    SKN_CUDA(ctx, cudaMemcpyAsync(out_host, out, (size_t)M * H * V * 4, cudaMemcpyDeviceToHost, ctx->stream));
    return skn_sync(ctx);
}

}  // extern "C"
