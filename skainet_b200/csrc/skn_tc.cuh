// tcgen05 / TMEM / tiled-TMA wrappers shared by the tensor-core kernels (K-major bf16 operand tiles of 64 columns
// with 128-byte swizzle, fp32 accumulators).
#pragma once
#include "skn_internal.cuh"
#include "skn_ptx.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

// One lane of a converged warp, chosen by the instruction made for it: under a plain `lane == 0` the operands of every
// tcgen05 instruction take a detour through vector registers (measured for the four MMAs of a 64-column stage: 445 clocks
// instead of 100, more than the 256 to 512 that the tensor cores need for them).
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// ---- tcgen05 wrappers ---------------------------------------------------------------------
__device__ __forceinline__ void tc_alloc(uint32_t *slot_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(skn_smem_u32(slot_smem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(skn_smem_u32(bar))
                 : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, 128 x N x 16, bf16 in, fp32 out
__device__ __forceinline__ void tc_mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the same with A in tensor memory: lane = row of A, a 32-bit column holds two of its elements (a step of 16 takes eight columns)
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// a warp's quarter of the lanes (32 (warp % 4) ...): 8 or 16 registers per thread -> as many columns
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                 "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 32 lanes x 32 columns of 32-bit accumulators -> 32 registers per thread
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 16 columns at each of two addresses
__device__ __forceinline__ void tc_ld16x2(uint32_t at0, uint32_t at1, uint32_t (&r)[16], uint32_t (&q)[16]) {
#define TC_LD16(at, r)                                                                                                          \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"        \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),   \
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])                      \
                 : "r"(at))
    TC_LD16(at0, r);
    TC_LD16(at1, q);
#undef TC_LD16
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- clusters, warp-wide waits, shared-memory windows ------------------------------------------------------------
__device__ __forceinline__ uint32_t tc_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t tc_mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void tc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// A bounded wait of a whole warp with one answer for all its lanes.  All of them look once; where that does not settle it, one
// lane polls by its clock and shares the result.  (One lane from the start: a broadcast on every wait, 333 -> 341 us for eight
// 4096 x 14336 Q4_0 products of 16 rows and 4.49 -> 4.60 ms for a 2048-token Lugasun prompt; this form 288 us and 4.52 ms.)
__device__ __forceinline__ bool tc_wait_warp(uint64_t *bar, uint32_t parity, int lane) {
    if (__all_sync(0xffffffffu, skn_mbar_try_wait(bar, parity))) return true;
    bool ok = true;
    if (lane == 0) ok = skn_mbar_wait(bar, parity);
    return __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
}
// ... for two barriers: one vote where both are complete (two cost 14336 x 4096 Q4_K at 16 rows 29.8 us instead of 29.0)
__device__ __forceinline__ bool tc_wait_warp(uint64_t *bar, uint32_t parity, uint64_t *bar2, uint32_t parity2, int lane) {
    if (__all_sync(0xffffffffu, skn_mbar_try_wait(bar, parity) && skn_mbar_try_wait(bar2, parity2))) return true;
    return tc_wait_warp(bar, parity, lane) && tc_wait_warp(bar2, parity2, lane);
}
__device__ __forceinline__ uint4 tc_lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// words of a byte run that starts `sel` words and sh bits (0 or 16) into an aligned window (sel: the same for the warp)
template <int SEL, int N, int W>
__device__ __forceinline__ void tc_cut(const uint32_t (&win)[W], uint32_t sh, uint32_t (&out)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = __funnelshift_rc(win[i + SEL], (i + SEL + 1 < W) ? win[i + SEL + 1 < W ? i + SEL + 1 : 0] : 0u, sh);
}
template <int N, int W>
__device__ __forceinline__ void tc_shift(const uint32_t (&win)[W], int sel, uint32_t sh, uint32_t (&out)[N]) {
    switch (sel) {
    case 0: tc_cut<0>(win, sh, out); break;
    case 1: tc_cut<1>(win, sh, out); break;
    case 2: tc_cut<2>(win, sh, out); break;
    default: tc_cut<3>(win, sh, out); break;
    }
}
template <int N> __device__ __forceinline__ void tc_window(uint32_t addr, uint32_t (&w)[N]) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
        const uint4 v = tc_lds128(addr + 16 * i);
        w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
}


// 2-D tiled TMA load (no multicast) of a box at element coordinates (x = column, y = row); the
// tensor map's 128-byte swizzle lays the box out exactly as tc_store_chunk does
__device__ __forceinline__ void tc_tma_load_2d(void *dst_smem, const CUtensorMap *tmap, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(skn_smem_u32(dst_smem)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(skn_smem_u32(bar))
        : "memory");
}

// Shared-memory matrix descriptor: K-major operand, rows of 64 bf16 (128 bytes) in 8-row
// groups of 1024 bytes, 128-byte swizzle (16-byte chunk c of row r sits at chunk c ^ (r & 7)).
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);   // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset: 8 rows * 128 bytes
    d |= (uint64_t)1 << 46;                          // descriptor version of this architecture
    d |= (uint64_t)2 << 61;                          // swizzle mode: 128 bytes
    return d;
}
// Instruction descriptor: fp32 accumulator, bf16 A and B, both K-major, M x N tile
__device__ __forceinline__ uint32_t tc_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// store 8 consecutive bf16 (one 16-byte chunk `c` of row `r`) into a swizzled tile
__device__ __forceinline__ void tc_store_chunk(uint8_t *tile, int r, int c, uint4 v) {
    *reinterpret_cast<uint4 *>(tile + (r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4)) = v;
}

__device__ __forceinline__ uint32_t tc_pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

typedef CUresult (*skn_encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                        const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                        CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's tensor-map encoder (looked up once)
static inline cudaError_t skn_tmap_encoder(skn_encode_tiled_fn *out) {
    static skn_encode_tiled_fn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess) return e;
        if (!fn || q != cudaDriverEntryPointSuccess) return cudaErrorNotSupported;
        encode = (skn_encode_tiled_fn)fn;
    }
    *out = encode;
    return cudaSuccess;
}

// Tensor map of a row-major bf16 matrix [rows][cols] with a row pitch in bytes (a multiple of 16): boxes of 64 columns
// x box_rows rows, 128-byte swizzle, elements outside the matrix read as zeros.
static inline cudaError_t skn_tmap_bf16(const void *base, int64_t rows, int64_t cols, int64_t pitch_bytes, int box_rows, CUtensorMap *out) {
    skn_encode_tiled_fn encode = nullptr;
    const cudaError_t e = skn_tmap_encoder(&encode);
    if (e != cudaSuccess) return e;
    const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)pitch_bytes};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), gdim, gstride, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Tensor map of a tensor's raw blocks: boxes of `rows` rows x box_bytes bytes, coordinates in 4-byte units
static inline cudaError_t skn_tmap_blocks(const skn_tensor *w, int box_bytes, int rows, CUtensorMap *out) {
    skn_encode_tiled_fn encode = nullptr;
    const cudaError_t e = skn_tmap_encoder(&encode);
    if (e != cudaSuccess) return e;
    const cuuint64_t gdim[2] = {(cuuint64_t)((w->row_bytes + 3) / 4), (cuuint64_t)w->n_rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)w->pitch};
    const cuuint32_t box[2] = {(cuuint32_t)(box_bytes / 4), (cuuint32_t)rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, w->d_blocks, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
