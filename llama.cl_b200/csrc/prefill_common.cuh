// What the two prefill kernels share: the tile's parameters, bounded waits, and the PTX of TMA, tensor memory and packed fp32.
#pragma once
#include <cuda.h>  // CUtensorMap

#include "common.cuh"
#include "ring_ptx.cuh"

namespace q4fc {

constexpr int kTileN = 128;     // weight columns per tile = TMEM lanes
constexpr int kStageRow = 128;  // bytes of an activation row in a stage: one row of the 128-byte swizzle

enum Format { kQ4_0 = 0, kQ4_1 = 1, kQ4_0Signed = 2, kQ8C = 3 };
enum { kWhole, kFirst, kRemainder };
struct PrefillParams {
    const uint8_t* wq;
    const float* sc;       // [row tile][Kg][scale | sum][TM]
    const float* wscales;  // Q8C
    float* y;
    int* status;
    int64_t rows, N, ldy;
    int Ng, Kg, split;
    int n_tiles;         // column tiles; tiles are counted along them
    int n_off, m_off;    // this launch's first tile
    int n_end, m_end;    // and the one behind its last
    int fold;            // Q4: stages of 128 k of a running sum, 0: one sum over all of a CTA's stages
    int part;            // kWhole, or of two launches kFirst (whole rounds) and kRemainder (the tiles that are left)
};

// 128-row tiles of Q4 weights (fc_prefill_wide.cu)
int launch_prefill_wide(int fmt, int G, const PrefillParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t s);

#ifdef __CUDACC__
// one lane of a converged warp.  (The compiler knows that exactly one lane runs the branch and keeps descriptors in
// uniform registers; behind `lane == 0` it cannot, and issuing an MMA takes about a third longer.)
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}
// 2-D tiled TMA load (no multicast): box at (x, y) of the tensor map -> shared memory, completion on `bar`
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y)
                 : "memory");
}
// packed fp32 pairs (sm_100): one issue slot for two fused multiply-adds
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ void fence_gpu_and_copies() { asm volatile("fence.acq_rel.gpu;\n\tfence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void tc_st(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// K-major operand tile with 128-byte rows and 128-byte swizzle: rows 128 B apart, 8-row groups
// 1024 B apart (stride byte offset), descriptor version 1, layout type 2 (SWIZZLE_128B)
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}
// the eight nibbles of a word as bytes: k = 0..3 (low nibbles) and 4..7 (high nibbles)
template <bool SIGNED>
__device__ __forceinline__ void unpack_nibbles(uint32_t word, uint32_t& lo, uint32_t& hi) {
    lo = word & 0x0F0F0F0Fu, hi = (word >> 4) & 0x0F0F0F0Fu;
    if (SIGNED) {  // sign-extend each nibble into its byte
        lo |= (lo & 0x08080808u) * 0x1Eu;
        hi |= (hi & 0x08080808u) * 0x1Eu;
    }
}

#endif

}  // namespace q4fc
