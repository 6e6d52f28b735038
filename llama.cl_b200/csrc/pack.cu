// Weight packer and dequantizer for the Q4_0 / Q4_1 block format.
//
// pack_kernel replaces offline_FC_quant_Q4A (ops/op_fc.hpp:151-219): fp32
// W[N][K] -> int8 [Ng][Kg][BS].  HBM-bound streaming kernel: 4 bytes read and
// 0.52-0.63 bytes written per weight.
//
// Work split: one thread owns two 32-bit output words = one column n x 16
// consecutive k (two 256-bit loads where the rows start on 32 bytes).  The G/16 threads that share a (column,
// K group) sit in adjacent lanes, so the group minimum / maximum is a
// segmented warp-shuffle reduction.  A CTA stages a tile of 32 columns x 256 k of packed output in
// shared memory and writes it out with 128-bit stores.
//
// What bounds it: issue slots, then HBM.  One word per thread and one path for all values took 22 warp instructions per 32
// weights; the instructions a group costs (shuffles, scale and its reciprocal, addresses) are now shared by 16 weights of a
// thread, and full groups of ordinary finite values take a path without clamps and float-to-int conversions.
// 11008 x 4096, Q4_1 group 128: 45.2 -> 36.5 us (5.6 TB/s).
//
// General path: the reduction keeps the reference's
// "first value wins a tie" rule of get_min_max (ops/op_fc.hpp:112-122) by
// always combining an earlier k range (left) with a later one (right) under
// the same strict compares, which matters only for the sign of a zero
// minimum.
//
// Arithmetic is the reference's, in fp32 with IEEE division: Q4_1
// d=(max-min)/15, m=min, q=clamp(roundf((w-m)/d'),0,15) with d'=1/d computed
// first; Q4_0 d=max(|min|,|max|)/7, q=clamp(roundf(w*d'),-7,7), roundf as
// round_half_away of common.cuh.
#include "common.cuh"

namespace q4fc {
namespace {

constexpr int kPackThreads = 256;
constexpr int kTileK = 256;  // k covered by one CTA tile

struct MinMax {
    float vmin, vmax;
    int has;
};

__device__ __forceinline__ void mm_take(MinMax& a, float v) {  // sequential step of get_min_max
    if (a.vmax < v) a.vmax = v;
    if (a.vmin > v) a.vmin = v;
}

// 256-bit load (sm_100), 32-byte aligned
__device__ __forceinline__ void ldg_v8(const float* p, float* v) {
    asm volatile("ld.global.nc.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
// Sixteen values from any 4-byte place: the 16-byte pieces around them, shifted by what they start too early.  (As sixteen
// 4-byte loads, each of them 32 sectors wide for a warp, 8747 x 2816, Q4_0 group 128 took 41 us, so 28.)
__device__ __forceinline__ void ldg_any16(const float* src, float* v) {
    const int a = (int)(reinterpret_cast<uintptr_t>(src) >> 2) & 3;
    float t[20];
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(src - a) + i);
        t[4 * i] = q.x, t[4 * i + 1] = q.y, t[4 * i + 2] = q.z, t[4 * i + 3] = q.w;
    }
#pragma unroll
    for (int i = 0; i < 19; i++) t[i] = a & 1 ? t[i + 1] : t[i];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = a & 2 ? t[i + 2] : t[i];
}
// of three values (sm_100); NaN if one of them is
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float scale_of(int qtype, float vmin, float vmax) {
    return qtype == 1 ? div_const_rn(__fsub_rn(vmax, vmin), 15.0f, 1.0f / 15.0f)
                      : div_const_rn(fmaxf(fabsf(vmin), fabsf(vmax)), 7.0f, 1.0f / 7.0f);
}
// where code j of a word goes: byte (j&3), low nibble for j<4, high nibble for j>=4 (ops/op_fc.hpp:39-48)
__host__ __device__ constexpr uint32_t place(int j) { return 1u << (8 * (j & 3) + 4 * (j >> 2)); }

// Eight codes of values whose group has a scale between 2^-100 and 2^100: no clamp is needed, |w - m| / d and |w| / d exceed 15
// and 7 by a few roundings at most.  The words are sums: nibbles do not overlap, a multiply-add places a code.
template <int QTYPE>
__device__ __forceinline__ uint32_t codes_of(const float* v, float m, float id) {
    uint32_t word;
    if (QTYPE == 1) {
        // t >= 0: roundf is trunc(t + 0.5) with the add rounded toward zero; adding 2^23, rounded the same way, leaves the
        // integer in the low bits (0x4B000000 above it, whose multiples the start value takes off again)
        word = 0u - (0x4B000000u * place(0) + 0x4B000000u * place(4));
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float t = __fmul_rn(__fsub_rn(v[j], m), id);
            word += __float_as_uint(__fadd_rz(__fadd_rz(t, 0.5f), 8388608.0f)) * place(j);
        }
    } else {
        word = 0x88888888u;  // code + 8 in every nibble, so that no borrow crosses
#pragma unroll
        for (int j = 0; j < 8; j++) word += (uint32_t)round_half_away(__fmul_rn(v[j], id)) * place(j);
        word ^= 0x88888888u;
    }
    return word;
}

constexpr int kPerThread = 16;                    // consecutive k of a thread
constexpr int kRowWords = 36;                     // staged block rows: 32 words and a gap, against bank conflicts

template <int G, int QTYPE>
__global__ void __launch_bounds__(kPackThreads) pack_kernel(const float* __restrict__ w, int64_t N, int64_t K,
                                                            int64_t Kg, int tiles_k, int vec_ok,
                                                            uint8_t* __restrict__ out) {
    constexpr int BS = block_bytes(QTYPE, G);
    constexpr int SEG = G / kPerThread;     // lanes sharing one (column, group)
    constexpr int NPW = 32 / SEG;           // columns per warp step
    constexpr int GB = kTileK / G;          // groups per CTA tile
    constexpr int STEPS = 32 / NPW;         // warp steps per group: the columns
    constexpr int WARPS = kPackThreads / 32;
    constexpr int ITERS = GB * STEPS / WARPS;
    constexpr int STAGE = (G / 8 + 1) * kRowWords;  // words of a staged block: its rows, then scales (and minima)
    static_assert(ITERS == 2 && WARPS % STEPS == 0, "a warp keeps its columns and moves on by half a tile");

    __shared__ __align__(16) uint32_t stage[GB * STAGE];

    const int64_t nb = blockIdx.x / tiles_k;
    const int tile = blockIdx.x % tiles_k;
    const int64_t kb0 = (int64_t)tile * GB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int seg_lane = lane % SEG;
    const int n_l = (warp % STEPS) * NPW + lane / SEG;
    const int64_t n = nb * 32 + n_l;

    float v[ITERS][kPerThread];
    int nvalid[ITERS];  // valid elements of this thread's (prefix), -1: column beyond N, or group beyond Kg
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
        const int64_t kb = kb0 + warp / STEPS + it * (GB / ITERS);
        const int64_t k = kb * G + seg_lane * kPerThread;
        const float* src = w + n * K + k;
        const int cnt = (n < N && kb < Kg) ? (int)min((int64_t)kPerThread, max((int64_t)0, K - k)) : -1;
        if (cnt == kPerThread && vec_ok == 2) {
            ldg_v8(src, v[it]);
            ldg_v8(src + 8, v[it] + 8);
        } else if (cnt == kPerThread && vec_ok) {
#pragma unroll
            for (int i = 0; i < kPerThread / 4; i++) {
                const float4 a = __ldg(reinterpret_cast<const float4*>(src) + i);
                v[it][4 * i] = a.x, v[it][4 * i + 1] = a.y, v[it][4 * i + 2] = a.z, v[it][4 * i + 3] = a.w;
            }
        } else if (cnt == kPerThread && n * K + k >= 4 && n * K + k + 20 <= N * K) {  // (the pieces lie inside the matrix)
            ldg_any16(src, v[it]);
        } else {
#pragma unroll
            for (int j = 0; j < kPerThread; j++) v[it][j] = (j < cnt) ? __ldg(src + j) : 0.0f;
        }
        nvalid[it] = cnt;
    }

#pragma unroll
    for (int it = 0; it < ITERS; it++) {
        const int kb_l = warp / STEPS + it * (GB / ITERS);
        const int cnt = nvalid[it];
        const float* x = v[it];
        float vmin = min3(x[0], x[1], x[2]), vmax = max3(x[0], x[1], x[2]);
#pragma unroll
        for (int j = 3; j + 1 < kPerThread; j += 2) vmin = min3(vmin, x[j], x[j + 1]), vmax = max3(vmax, x[j], x[j + 1]);
        vmin = min3(vmin, x[15], x[15]), vmax = max3(vmax, x[15], x[15]);
#pragma unroll
        for (int off = 1; off < SEG; off <<= 1) {
            const float a = __shfl_xor_sync(0xffffffffu, vmin, off), b = __shfl_xor_sync(0xffffffffu, vmax, off);
            vmin = min3(vmin, a, a), vmax = max3(vmax, b, b);
        }
        float d = scale_of(QTYPE, vmin, vmax);
        uint32_t word[2];
        // (the value of a minimum does not depend on the order of the scan, only the sign of a zero does)
        if (__all_sync(0xffffffffu, cnt == kPerThread && vmin != 0.0f && vmax != 0.0f && d >= 0x1p-100f && d <= 0x1p100f)) {
            const float id = __frcp_rn(d);
            word[0] = codes_of<QTYPE>(x, vmin, id), word[1] = codes_of<QTYPE>(x + 8, vmin, id);
        } else {
            // missing values, zeros as extremes, NaN, infinities, scales near the ends of the range
            MinMax mm;
            mm.has = cnt > 0;
            mm.vmin = mm.vmax = x[0];
#pragma unroll
            for (int j = 1; j < kPerThread; j++)
                if (j < cnt) mm_take(mm, x[j]);
            // ordered segmented reduction: lane i absorbs lane i+off (later k)
#pragma unroll
            for (int off = 1; off < SEG; off <<= 1) {
                float rmin = __shfl_down_sync(0xffffffffu, mm.vmin, off, SEG);
                float rmax = __shfl_down_sync(0xffffffffu, mm.vmax, off, SEG);
                int rhas = __shfl_down_sync(0xffffffffu, mm.has, off, SEG);
                if (seg_lane + off < SEG && rhas) {
                    if (mm.vmax < rmax) mm.vmax = rmax;
                    if (mm.vmin > rmin) mm.vmin = rmin;
                }
            }
            vmin = __shfl_sync(0xffffffffu, mm.vmin, 0, SEG);
            vmax = __shfl_sync(0xffffffffu, mm.vmax, 0, SEG);
            d = scale_of(QTYPE, vmin, vmax);
            const float id = inv_or_zero(d);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                word[h] = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (8 * h + j < cnt) {
                        const float e = x[8 * h + j];
                        const int q = QTYPE == 1 ? min(15, __float2int_rz(__fadd_rz(__fmul_rn(__fsub_rn(e, vmin), id), 0.5f)))
                                                 : min(7, max(round_half_away(__fmul_rn(e, id)), -7)) & 0xF;
                        word[h] += (uint32_t)q * place(j);
                    }
                }
            }
        }
        uint32_t* block = stage + kb_l * STAGE;
        block[(2 * seg_lane) * kRowWords + n_l] = word[0];
        block[(2 * seg_lane + 1) * kRowWords + n_l] = word[1];
        if (seg_lane == 0) {
            uint16_t* tail = reinterpret_cast<uint16_t*>(block + (G / 8) * kRowWords);
            const bool live = cnt >= 0;  // cnt==0 cannot occur at seg_lane 0 of an existing group
            tail[n_l] = live ? f2h_rn(d) : (uint16_t)0;
            if (QTYPE == 1) tail[32 + n_l] = live ? f2h_rn(vmin) : (uint16_t)0;
        }
    }
    __syncthreads();

    constexpr int N16 = BS / 16;  // 16-byte pieces of a block, eight to a staged row
    const int n16 = (int)min((int64_t)GB, Kg - kb0) * N16;
    uint4* dst = reinterpret_cast<uint4*>(out + (nb * Kg + kb0) * (int64_t)BS);
    for (int i = threadIdx.x; i < n16; i += kPackThreads) {
        const int kb_l = i / N16, o = i % N16;
        dst[i] = *reinterpret_cast<const uint4*>(stage + kb_l * STAGE + (o >> 3) * kRowWords + (o & 7) * 4);
    }
}

template <int G, int QTYPE>
__global__ void __launch_bounds__(256) dequant_kernel(const uint8_t* __restrict__ wq, int64_t nblocks, int64_t Kg,
                                                      int nibble_signed, float* __restrict__ out) {
    // one thread per 32-bit word: column n, 8 consecutive k (ops/op_fc.hpp:124-149, get() :49-61 / :95-106)
    constexpr int BS = block_bytes(QTYPE, G);
    constexpr int WPB = G * 4;  // words per block
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= nblocks * WPB) return;
    const int64_t blk = gid / WPB;
    const int wi = (int)(gid % WPB);
    const int k8 = wi / 32, n = wi % 32;
    const uint8_t* b = wq + blk * BS;
    const uint32_t word = *reinterpret_cast<const uint32_t*>(b + k8 * 128 + n * 4);
    const float d = h2f(*reinterpret_cast<const uint16_t*>(b + 16 * G + 2 * n));
    const float m = QTYPE ? h2f(*reinterpret_cast<const uint16_t*>(b + 16 * G + 64 + 2 * n)) : 0.0f;
    const int64_t nb = blk / Kg, kb = blk % Kg;
    float* dst = out + (nb * 32 + n) * (Kg * G) + kb * G + k8 * 8;
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        int q = (word >> (8 * (j & 3) + 4 * (j >> 2))) & 0xF;
        if (QTYPE == 0 && nibble_signed && q >= 8) q -= 16;
        const float p = __fmul_rn(d, (float)q);  // exact: 11-bit x 4-bit
        r[j] = QTYPE ? __fadd_rn(p, m) : p;
    }
    reinterpret_cast<float4*>(dst)[0] = make_float4(r[0], r[1], r[2], r[3]);
    reinterpret_cast<float4*>(dst)[1] = make_float4(r[4], r[5], r[6], r[7]);
}

}  // namespace

int launch_pack(const float* w, int64_t N, int64_t K, int qtype, int G, uint8_t* wq, cudaStream_t s) {
    const int64_t Ng = (N + 31) / 32, Kg = (K + G - 1) / G;
    if (Ng == 0 || Kg == 0) return Q4FC_OK;
    const int GB = kTileK / G;
    const int64_t tiles_k = (Kg + GB - 1) / GB;
    if (Ng * tiles_k > 0x7fffffffLL || tiles_k > 0x7fffffffLL) {
        set_error("pack: %lld x %lld tiles exceed the grid limit", (long long)Ng, (long long)tiles_k);
        return Q4FC_ELIMIT;
    }
    // widest load that every row's start allows: 2 = 32 bytes, 1 = 16, 0 = 4
    const uintptr_t wa = reinterpret_cast<uintptr_t>(w);
    const int vec_ok = (K % 8 == 0 && (wa & 31) == 0) ? 2 : (K % 4 == 0 && (wa & 15) == 0) ? 1 : 0;
    dim3 grid((unsigned)(Ng * tiles_k));
#define Q4FC_PACK(GG, QQ) \
    pack_kernel<GG, QQ><<<grid, kPackThreads, 0, s>>>(w, N, K, Kg, (int)tiles_k, vec_ok, wq)
    if (G == 32 && qtype == 1) Q4FC_PACK(32, 1);
    else if (G == 128 && qtype == 1) Q4FC_PACK(128, 1);
    else if (G == 32 && qtype == 0) Q4FC_PACK(32, 0);
    else Q4FC_PACK(128, 0);
#undef Q4FC_PACK
    Q4FC_CUDA_OK(cudaGetLastError());
    return Q4FC_OK;
}

int launch_dequant(const uint8_t* wq, int64_t Ng, int64_t Kg, int qtype, int G, int nibble_signed, float* out,
                   cudaStream_t s) {
    const int64_t nblocks = Ng * Kg;
    if (nblocks == 0) return Q4FC_OK;
    const int64_t threads = nblocks * G * 4;
    const int64_t grid = (threads + 255) / 256;
    if (grid > 0x7fffffffLL) {
        set_error("dequant: tensor too large for one launch");
        return Q4FC_ELIMIT;
    }
#define Q4FC_DEQ(GG, QQ) dequant_kernel<GG, QQ><<<(unsigned)grid, 256, 0, s>>>(wq, nblocks, Kg, nibble_signed, out)
    if (G == 32 && qtype == 1) Q4FC_DEQ(32, 1);
    else if (G == 128 && qtype == 1) Q4FC_DEQ(128, 1);
    else if (G == 32 && qtype == 0) Q4FC_DEQ(32, 0);
    else Q4FC_DEQ(128, 0);
#undef Q4FC_DEQ
    Q4FC_CUDA_OK(cudaGetLastError());
    return Q4FC_OK;
}

}  // namespace q4fc
