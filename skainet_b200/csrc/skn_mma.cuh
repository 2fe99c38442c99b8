// Warp-level bf16 products (mma.sync) and their fragment loads, for the mixers' small tiles.
#pragma once
#include "skn_ptx.cuh"

#include <cuda_bf16.h>

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c = a b, from zero
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool in) {
    const int n = in ? 16 : 0;         // 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
// (a, b) minus what their packed bf16 form holds
__device__ __forceinline__ void less_bf16(float &a, float &b, uint32_t packed) {
    a -= __uint_as_float(packed << 16);
    b -= __uint_as_float(packed & 0xFFFF0000u);
}

// ---- fp32 operands as sums of three bf16 terms a + b + c (exact) ----------------------------------------------------
// (x, y) -> packed terms
__device__ __forceinline__ void split_terms(float x, float y, uint32_t (&w)[3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        w[p] = pack_bf16(x, y);
        if (p < 2) less_bf16(x, y, w[p]);
    }
}
// Sums over 16 elements of 2 NB tiles of 16 x 8: the small products of the six that reach the 24 bits (ac, ca, bb, ba, ab) in one chain, aa in a chain of
// its own (exact in nearly every case: products of 16 bits), so that what the tensor cores chop off when they add is far below the last
// bit of the two together.  NP: terms of the second operand; FIRST: from zero
template <int NP, bool FIRST, int NB>
__device__ __forceinline__ void mma_terms(float (&s)[2 * NB][4], float (&c)[2 * NB][4], const uint32_t (&a)[3][4], const uint32_t (&b)[NB][3][4]) {
    constexpr int P0 = NP == 3 ? 0 : 1, PA[5] = {0, 2, 1, 1, 0}, PB[5] = {2, 0, 1, 0, 1};       // smallest first
#pragma unroll
    for (int p = P0; p < 5; ++p)
#pragma unroll
        for (int i = 0; i < 2 * NB; ++i) {
            const uint32_t b0 = b[i >> 1][PB[p]][(i & 1) * 2], b1 = b[i >> 1][PB[p]][(i & 1) * 2 + 1];
            if (FIRST && p == P0) mma_bf16_first(s[i], a[PA[p]], b0, b1);
            else mma_bf16(s[i], a[PA[p]], b0, b1);
        }
#pragma unroll
    for (int i = 0; i < 2 * NB; ++i) {
        const uint32_t b0 = b[i >> 1][0][(i & 1) * 2], b1 = b[i >> 1][0][(i & 1) * 2 + 1];
        if (FIRST) mma_bf16_first(c[i], a[0], b0, b1);
        else mma_bf16(c[i], a[0], b0, b1);
    }
}
