// FC over many activation rows (prefill): dense int8 contraction on the 5th-generation tensor cores.  Replaces fc_Q4A
// (ops/op_fc.hpp:286-426) for B*M > 8 and, with FMT = kQ8C, FC_evaluate_Q8C (ext/llama_ext.cpp:232-371) where q8c.cu's own
// kernel has too much to do.
//
//   Q4:   y[m][n] = sum_kb  fp32(wd[n,kb]) * xs[m,kb] * I[m,n,kb]  (+ fp32(wm[n,kb]) * gsum[m,kb], Q4_1)
//   Q8C:  y[m][n] = wscale[n] * sum_kb xs[m,kb] * I[m,n,kb]
//   I[m,n,kb] = sum_{k in group kb} weight code(n,k) * activation code(m,k)      exact int32
//
// Two launches: quant_x_tile_kernel (quant_x.cu) writes codes, scales and group sums of all rows to the workspace; this
// kernel, or that of fc_prefill_wide.cu (128-row tiles of Q4 weights), started while that one runs (programmatic launch: its weight
// copies do not depend on it), runs the GEMM.
//
// One CTA computes 128 columns n x TM rows m, 64, or of Q8C weights also 128:
//   * operand A = weights: the packed blocks come in by bulk copies, are unpacked to one byte per weight in shared
//     memory, K-major rows of 128 bytes, in the 128-byte-swizzle canonical layout that tcgen05.mma reads;
//   * operand B = activation codes (int8), same layout, straight from the code matrix by TMA;
//   * D = int32 accumulators in tensor memory, lane = weight column, column = activation row.
// Every K group has its own pair of scales, so a group's MMA(s) (one K=32 instruction for group 32, four for group
// 128) write a fresh TMEM buffer (four of TM columns, three where the fourth's place holds sums), and the
// epilogue warps read the buffer back with
// tcgen05.ld, turn the exact integers into fp32, scale them and accumulate the tile in registers.
//
// What bounds it: the CUDA-core work per (m, n, group) -- one conversion, one mul, one or two fma -- against 32 or 128
// tensor MACs.  Everything else is arranged to stay behind that: the packed bytes are prefetched several stages ahead
// (a warp re-arms its own slot as soon as it has unpacked it), a lane unpacks one column so that both its 32-bit loads
// and its 128-bit stores are free of bank conflicts without selects, scales arrive in the layout in which the epilogue
// reads four rows per load, and weights, codes and scales have rings of their own, so that operands are released by the
// MMA and not by the epilogue.
//
// Sizes here and below are rows x K x N.
//
// Measured (whole call, quantizer included; unpacking straight from global memory without prefetch, one 128 x 128 tile per CTA
// whatever the row count, epilogue of 5 operations per integer -> this form -> with the last tiles divided, below, and scales read by
// shared-memory loads):
//   4096 -> 11008   Q4_1 g32, 37 rows 123.7 -> 41.0 -> 36.0 us   Q8C, 256 rows 296 -> 151 -> 99 us (233 TOPS)
// With 128-row tiles of Q4 weights, before they had a kernel of their own: Q4_0 g32, 512 rows 186 us; Q4_1 g128, 2048 rows 296.
// A group of 32 k takes about 1000 cycles for 128 x 128 integers, of which the MMA needs 64: the epilogue's chain of load,
// convert, scale is latency-bound with the 16 warps that the registers allow.  Tried and dropped: handing registers
// between roles with setmaxnreg (spills around it; 260 us for the 512-row case), both chunks in registers at once
// (320 us), the add-a-constant conversion instead of I2F (30 % more issue slots), scalar instead of packed fp32 (5 % slower), and
// this file's work in the form of fc_prefill_wide.cu (Q8C, 256 rows: 102; 64-row tiles, 12 x 11008 x 4096: 27.4 -> 31).
//
// Warp roles: epilogue (warp % 4 = TMEM lane quarter, warp / 4 = which 16-row chunks), 4 unpacking warps (one stripe
// each), one MMA issuer, one loader.  Every wait is bounded: when a wait runs out the CTA sets the status word, every
// role leaves its loop, TMEM is freed and the kernel returns.
//
// Q8C sums K in two levels (FOLD): the 8-row kernel of q8c.cu adds chains of a few groups, and one chain over all of K is
// less exact than that (K = 4096: 2.0e-7 of the result in the 2-norm, with 8 warps' chains 9.6e-8; K = 11008: 3.3e-7 and
// 1.3e-7).  After 8 groups, or 12 where a CTA has more than 64, a thread moves its running sums to a second place and keeps
// what that addition rounds off: 6.5e-8 to 7.5e-8 for K from 512 to 11008, below the 8-warp sums at every size tried.  It
// cost 131 -> 151 us at 256 rows x 4096 x 11008 (before the last tiles were divided) and 33 -> 35 at 37 rows; every 16 groups 146
// us and 8.3e-8, at K = 3001 not below the 8-warp sums.  (Staggering the moves over the warps: 156; as an outer loop around the groups' loop: 157.)
//
// Q4 sums K in one chain for each CTA; where few CTAs share it the sums move to a second place in between, so that no chain is longer
// than with many (see fold_of).
//
// Few tiles, or the last of many: a cluster of `split` CTAs shares a tile and divides its K stages; the partial tiles meet in shared memory
// and are added in rank order (fixed order, no atomics).  So the outputs of one call can be sums in two orders: equal rows of x, or
// equal columns of W, in whole rounds and in the remainder may differ in the last place.
#include <cooperative_groups.h>

#include <atomic>
#include <cfloat>
#include <mutex>

#include "prefill_common.cuh"

namespace cg = cooperative_groups;

namespace q4fc {
namespace {

constexpr int kStageK = 128;   // k per shared-memory stage (one 128-byte swizzle row)
constexpr int kTmemBufs = 4;   // of a tile's columns each
constexpr int kProdWarps = 4;  // one stripe of the tile each
constexpr int kMaxSplit = 8;
constexpr int64_t kMaxTileRows = 65535;  // rows of tiles, a grid's y

// FOLD: Q8C, the K groups of a running sum; Q4, whether the sums move after p.fold stages (see fold_of), kFewRows or kManyRows of a
// 64-row tile in use
enum { kFewRows = 1, kManyRows = 2 };
template <int FMT, int G, int TM, int FOLD>
struct PrefillShape {
    static constexpr int kBlock = FMT == kQ8C ? 1024 : block_bytes(FMT == kQ4_1, G);
    static constexpr int kGroups = kStageK / G;           // K groups per stage: 4 (group 32) or 1 (group 128)
    static constexpr int kSums = FMT == kQ4_1 ? 2 : 1;    // per group and row: scale (and group sum)
    static constexpr int kEpiWarps = TM / 8;              // 32 rows of the tile per warp and TMEM lane quarter
    static constexpr int kThreads = (kEpiWarps + kProdWarps + 2) * 32;
    static constexpr int kLoadWidth = TM == 128 ? 16 : 8; // rows a thread takes from tensor memory at a time
    static_assert(TM == 64 || FMT == kQ8C, "128-row tiles of Q4 weights: fc_prefill_wide.cu");
    static constexpr int kA = TM == 128 ? 3 : 2;          // stages of unpacked weights
    static constexpr int kB = FMT == kQ8C || (TM == 64 && G == 32) ? 3 : 4;    // stages of activation codes
    static constexpr int kRaw = FMT == kQ8C || (TM == 64 && G == 32) ? 3 : 4;  // stages of packed bytes
    static constexpr int kScs = 4;                        // stages of scales
    // Buffers of integers in the kTmemBufs x TM columns.  Sums that move, of 64-row tiles, take the last one's place, or where at most
    // 48 rows are in use the last quarters of the buffers, which no MMA then writes.
    static constexpr int kBufs = TM == 64 && FOLD > (FMT == kQ8C ? 0 : kFewRows) ? kTmemBufs - 1 : kTmemBufs;
    static constexpr int kSumCol = kBufs == kTmemBufs ? 48 : kBufs * TM;      // of the first 16 rows' sums
    static constexpr int kSumStep = kBufs == kTmemBufs ? TM : 16;             // from 16 rows to the next 16
    static constexpr int kRawStripe = kGroups * kBlock;   // packed bytes of one stripe in a stage
    static constexpr int kABytes = kTileN * kStageK, kBBytes = TM * kStageK;
    static constexpr int kXscBytes = kGroups * kSums * TM * 4;                // [group][scale | sum][row] fp32
    static constexpr int kWscBytes = FMT == kQ8C ? 0 : kGroups * kTileN * 4;  // [group][n] {wd, wm} fp16
    static constexpr int kScBytes = kXscBytes + kWscBytes;
    static constexpr int kBOff = kA * kABytes;
    static constexpr int kRawOff = kBOff + kB * kBBytes;
    static constexpr int kScOff = kRawOff + kRaw * 4 * kRawStripe;
    static constexpr int kBarOff = kScOff + kScs * kScBytes;
    static constexpr int kSumOff = kBarOff + 512;
    static constexpr int kSmem = kSumOff + (FMT == kQ8C && TM == 128 ? TM * kTileN * 4 : 0) + 1024 /*alignment slack*/;
    static_assert(TM == 128 || kSmem <= 113 * 1024, "two CTAs on an SM");
    static_assert(TM * kTileN * 4 <= kRawOff, "the partial tile of a K split takes the operand stages' place");
};

// ---- PTX helpers -------------------------------------------------------------
// bounded wait: gives up after kWaitLimitNs, or as soon as another role has raised the abort flag
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0 = 0;
#pragma unroll 1
    for (uint32_t i = 1;; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63) == 0) {
            if (*abort_flag) return false;
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > kWaitLimitNs) break;
        }
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ uint64_t fsub2(uint64_t a, uint64_t b) { return ffma2(b, 0xBF800000BF800000ull, a); }
__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
        : "memory");
}
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tc_st(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.b16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void lds128(uint32_t addr, uint64_t& a, uint64_t& b) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint64_t a, uint64_t b) {
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(addr), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// acc[P .. P + W/2) += scaled integers of W rows (+ wm * their group sums); `xs`: the rows' scales, the group sums
// follow at xs + TM
template <int FMT, int G, int TM, int P, int W>
__device__ __forceinline__ void accumulate(uint64_t (&acc)[8], const uint32_t (&v)[W], const float* xs, uint64_t wd2,
                                           uint64_t wm2) {
#pragma unroll
    for (int j = 0; j < W / 4; j++) {
        const ulonglong2 x4 = *reinterpret_cast<const ulonglong2*>(xs + 4 * j);
        const uint64_t i01 = pack2(__int2float_rn((int)v[4 * j]), __int2float_rn((int)v[4 * j + 1]));
        const uint64_t i23 = pack2(__int2float_rn((int)v[4 * j + 2]), __int2float_rn((int)v[4 * j + 3]));
        uint64_t &a = acc[P + 2 * j], &b = acc[P + 2 * j + 1];
        // The column's scale, fp16, and the integer first, whose product rounds off less than that of the scales: 3 to 4 % less error
        // against 64 bits, and 0.5 % less time.  (Not for Q4_0 with group 32, where up to 32 rows then take 0.8 % longer.)
        constexpr bool kIntegerFirst = FMT == kQ4_1 || G == 128;
        a = FMT == kQ8C ? ffma2(x4.x, i01, a) : kIntegerFirst ? ffma2(x4.x, fmul2(wd2, i01), a) : ffma2(fmul2(wd2, x4.x), i01, a);
        b = FMT == kQ8C ? ffma2(x4.y, i23, b) : kIntegerFirst ? ffma2(x4.y, fmul2(wd2, i23), b) : ffma2(fmul2(wd2, x4.y), i23, b);
        if (FMT == kQ4_1) {
            const ulonglong2 g4 = *reinterpret_cast<const ulonglong2*>(xs + TM + 4 * j);
            a = ffma2(wm2, g4.x, a);
            b = ffma2(wm2, g4.y, b);
        }
    }
}

// ---- Q8C: sums in two levels --------------------------------------------------------------------------------------------
// `sum` += `run`, and what the addition rounds off stays in `run` and starts the next running sum (T. J. Dekker, Numer.
// Math. 18, 1971: exact where |sum| >= |run|; elsewhere a rounding of the smaller `run` is lost).
__device__ __forceinline__ uint64_t move_sum(uint64_t sum, uint64_t& run) {
    const uint64_t s = fadd2(sum, run);
    run = fsub2(run, fsub2(s, sum));
    return s;
}
__device__ __forceinline__ void finite_or_zero(uint64_t& v) {
    float lo, hi;
    unpack2(v, lo, hi);
    v = pack2(fabsf(lo) <= FLT_MAX ? lo : 0.0f, fabsf(hi) <= FLT_MAX ? hi : 0.0f);
}
// Sixteen rows of a thread's running sums into the sums behind `at`: 128-row tiles keep them in shared memory (a thread's
// own 16-byte places), 64-row tiles, whose shared memory is full, in the last of their four TMEM buffers.
template <int TM, int THREADS>
__device__ __forceinline__ void fold(uint64_t (&run)[8], uint32_t at, bool first) {
    uint64_t odd = 0;  // not finite where a sum has left the finite numbers
    if constexpr (TM == 128) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint64_t a = 0, b = 0;
            if (!first) lds128(at + j * THREADS * 16, a, b);
            a = move_sum(a, run[2 * j]), b = move_sum(b, run[2 * j + 1]);
            odd = fadd2(odd, fadd2(run[2 * j], run[2 * j + 1]));
            sts128(at + j * THREADS * 16, a, b);
        }
    } else {
        tc_wait_st();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t v[8] = {};
            if (!first) {
                tc_ld(at + 8 * h, v);
                tc_wait_ld();
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint64_t a = pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                a = move_sum(a, run[4 * h + j]);
                odd = fadd2(odd, run[4 * h + j]);
                float lo, hi;
                unpack2(a, lo, hi);
                v[2 * j] = __float_as_uint(lo), v[2 * j + 1] = __float_as_uint(hi);
            }
            tc_st(at + 8 * h, v);
        }
    }
    float lo, hi;
    unpack2(odd, lo, hi);
    if (!(fabsf(lo) <= FLT_MAX && fabsf(hi) <= FLT_MAX)) {
#pragma unroll
        for (int j = 0; j < 8; j++) finite_or_zero(run[j]);
    }
}
template <int TM, int THREADS>
__device__ __forceinline__ void unfold(uint64_t (&run)[8], uint32_t at) {  // `run` += the sums behind `at`
    if constexpr (TM == 128) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint64_t a, b;
            lds128(at + j * THREADS * 16, a, b);
            run[2 * j] = fadd2(a, run[2 * j]), run[2 * j + 1] = fadd2(b, run[2 * j + 1]);
        }
    } else {
        tc_wait_st();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t v[8];
            tc_ld(at + 8 * h, v);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 4; j++)
                run[4 * h + j] = fadd2(pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), run[4 * h + j]);
        }
    }
}


// Q4 where sums move: the running sums of a thread's rows (sixteen, or `two` times sixteen) and the sums behind `at` added, into there,
// and the running sums start anew; the `last` time into the running sums.  One piece of code for both: a CTA runs it once or twice,
// and what it takes is its instructions' way to the SM (0.3 us for both; in front of the groups' loop's own branches 1 us).
__device__ __forceinline__ void merge_sums(uint64_t (&run)[2][8], uint32_t at, uint32_t step, bool two, bool last) {
    tc_wait_st();
    auto add = [&](uint64_t (&r)[8], uint32_t at) {
        uint32_t v[16];
        tc_ld(at, v);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; j++) r[j] = fadd2(pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), r[j]);
    };
    auto store = [&](uint64_t (&r)[8], uint32_t at) {
        uint32_t v[16];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            float lo, hi;
            unpack2(r[j], lo, hi);
            v[2 * j] = __float_as_uint(lo), v[2 * j + 1] = __float_as_uint(hi);
            r[j] = 0;
        }
        q4fc::tc_st(at, v);
    };
    add(run[0], at);
    if (two) add(run[1], at + step);
    if (last) return;
    store(run[0], at);
    if (two) store(run[1], at + step);
}

template <int FMT, int G, int TM, int FOLD>
__global__ void __launch_bounds__(PrefillShape<FMT, G, TM, FOLD>::kThreads, TM == 128 ? 1 : 2)
    fc_prefill_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap codes_map) {
    using S = PrefillShape<FMT, G, TM, FOLD>;
    constexpr int BS = S::kBlock;
    constexpr int GPS = S::kGroups;
    constexpr int MMAS = G / 32;  // K=32 instructions per group
    constexpr int CGN = S::kEpiWarps / 4;
    constexpr int kUnpackWarp = S::kEpiWarps, kMmaWarp = kUnpackWarp + kProdWarps;
    constexpr bool kMoves = FMT != kQ8C && FOLD > 0;

    extern __shared__ uint8_t smem_raw[];
    // (the same offset in every CTA of a cluster: the dynamic shared memory starts at the same address)
    // (An offset, and no cast through an integer behind which every load of a scale is a generic one: 37 rows x 4096 x 11008
    // 39.1 -> 36.3 us, 200 x 4096 x 4096, group 128, 26.8 -> 25.5, Q8C, 512 x 4096 x 4096, 86.5 -> 82.0.)
    uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
    uint8_t* bars = smem + S::kBarOff;
    const uint32_t smem0 = smem_u32(smem);
    const uint32_t bar_raw = smem0 + S::kBarOff;  // [raw stage][stripe]
    const uint32_t bar_afull = bar_raw + 8 * 4 * S::kRaw, bar_aempty = bar_afull + 8 * S::kA;
    const uint32_t bar_bfull = bar_aempty + 8 * S::kA, bar_bempty = bar_bfull + 8 * S::kB;
    const uint32_t bar_sfull = bar_bempty + 8 * S::kB, bar_sempty = bar_sfull + 8 * S::kScs;
    const uint32_t bar_tfull = bar_sempty + 8 * S::kScs, bar_tempty = bar_tfull + 8 * kTmemBufs;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 496);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 500);
    [[maybe_unused]] volatile int* noted = reinterpret_cast<volatile int*>(bars + 504);  // kMoves: the CTA's groups, and rows
    static_assert(8 * (4 * S::kRaw + 2 * S::kA + 2 * S::kB + 2 * S::kScs + 2 * kTmemBufs) <= 496, "barriers");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cs = p.split, rank = (int)(blockIdx.x % cs);
    int n_tile = (int)(blockIdx.x / cs) + p.n_off, m_tile = (int)blockIdx.y + p.m_off;
    if (n_tile >= p.n_tiles) n_tile -= p.n_tiles, m_tile++;
    if (m_tile > p.m_end || (m_tile == p.m_end && n_tile >= p.n_end)) return;  // (the whole cluster)
    const int64_t n0 = (int64_t)n_tile * kTileN, m0 = (int64_t)m_tile * TM;
    const int live = (int)min((int64_t)TM, p.rows - m0);  // rows of this tile that exist
    const int nstage = (p.Kg + GPS - 1) / GPS;
    const int it0 = (int)((int64_t)nstage * rank / cs), it1 = (int)((int64_t)nstage * (rank + 1) / cs);
    const int iters = it1 - it0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 4 * S::kRaw; i++) mbar_init(bar_raw + 8 * i, 1);
        for (int i = 0; i < S::kA; i++) {
            mbar_init(bar_afull + 8 * i, kProdWarps);
            mbar_init(bar_aempty + 8 * i, 1);  // tcgen05.commit
        }
        for (int i = 0; i < S::kB; i++) {
            mbar_init(bar_bfull + 8 * i, 1);
            mbar_init(bar_bempty + 8 * i, 1);  // tcgen05.commit
        }
        for (int i = 0; i < S::kScs; i++) {
            mbar_init(bar_sfull + 8 * i, kProdWarps + 1);  // unpacking warps + the loader's expect_tx
            mbar_init(bar_sempty + 8 * i, S::kEpiWarps);
        }
        for (int i = 0; i < kTmemBufs; i++) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, S::kEpiWarps);
        }
        *abort_flag = 0;
        if (kMoves) noted[0] = min(p.Kg, it1 * GPS) - it0 * GPS, noted[1] = live;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"((uint32_t)(kTmemBufs * TM))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < kUnpackWarp) {
        // =================== epilogue: 32 lanes x (16 + 16) rows per warp ===================
        uint64_t acc[2][8];  // 2 x 16 rows as packed pairs
        const int quarter = warp & 3, cgrp = warp >> 2;
        const int nrow = quarter * 32 + lane;  // tile column n handled by this thread (= TMEM lane)
        if (iters == 0) pdl_wait_prior_grid();  // no K group: nothing else orders the stores behind earlier work
        // chunks of 16 rows are dealt out to the warps of a quarter in turn, so that few rows still occupy all of them
        const bool live0 = cgrp * 16 < live, live1 = (cgrp + CGN) * 16 < live;
#pragma unroll
        for (int i = 0; i < 8; i++) acc[0][i] = acc[1][i] = 0ull;
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + cgrp * 16;
        // the sums that FOLD K groups at a time are moved to
        constexpr int kEpi = S::kEpiWarps * 32;
        const uint32_t sum0 = TM == 128 ? smem0 + S::kSumOff + threadIdx.x * 16 : taddr + S::kBufs * TM;
        const uint32_t sum1 = sum0 + (TM == 128 ? 4 * 16 * kEpi : CGN * 16);
        const int groups = min(p.Kg, it1 * GPS) - it0 * GPS;
        // groups g .. end - 1 into the running sums; false when a wait ran out
        auto add_groups = [&](int g, int end) {
#pragma unroll 1
            for (; g < end; g++) {
                const int i = g / GPS, sl = i % S::kScs, gi = g % GPS, b = g % S::kBufs;
                if (gi == 0 && !wait_or_abort(bar_sfull + 8 * sl, (i / S::kScs) & 1, abort_flag)) return false;
                const uint8_t* sc = smem + S::kScOff + sl * S::kScBytes;
                const float* xs = reinterpret_cast<const float*>(sc) + gi * (S::kSums * TM) + cgrp * 16;
                uint64_t wd2 = 0, wm2 = 0;
                if constexpr (FMT != kQ8C) {
                    const uint32_t w = reinterpret_cast<const uint32_t*>(sc + S::kXscBytes)[gi * kTileN + nrow];
                    const float wd = h2f((uint16_t)w), wm = h2f((uint16_t)(w >> 16));
                    wd2 = pack2(wd, wd), wm2 = pack2(wm, wm);
                }
                if (!wait_or_abort(bar_tfull + 8 * b, (g / S::kBufs) & 1, abort_flag)) return false;
                tc_fence_after();
                // W integers at a time: what the two chunks would take together is what the register file has left, and the
                // compiler then serialises the arithmetic (37 rows, one CTA an SM: 84 us with W = 16 in 72 registers, 78 with 8)
                auto release = [&] {  // the buffer can be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_tempty + 8 * b);
                };
                constexpr int W = S::kLoadWidth;
                uint32_t v[W];
                if (live0) {
                    tc_ld(taddr + b * TM, v);
                    tc_wait_ld();
                    accumulate<FMT, G, TM, 0, W>(acc[0], v, xs, wd2, wm2);
                    if constexpr (W == 8) {
                        tc_ld(taddr + b * TM + 8, v);
                        tc_wait_ld();
                        accumulate<FMT, G, TM, 4, W>(acc[0], v, xs + 8, wd2, wm2);
                    }
                }
                if (live1) {
                    tc_ld(taddr + b * TM + CGN * 16, v);
                    tc_wait_ld();
                    if constexpr (W == 8) {
                        accumulate<FMT, G, TM, 0, W>(acc[1], v, xs + CGN * 16, wd2, wm2);
                        tc_ld(taddr + b * TM + CGN * 16 + 8, v);
                        tc_wait_ld();
                    }
                }
                release();
                if (live1) accumulate<FMT, G, TM, W == 8 ? 4 : 0, W>(acc[1], v, xs + CGN * 16 + 16 - W, wd2, wm2);
                if (gi == GPS - 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_sempty + 8 * sl);  // done with the stage's scales
                }
                if constexpr (FMT == kQ8C && FOLD > 0)
                    if (g % FOLD == FOLD - 1) {
                        if (live0) fold<TM, kEpi>(acc[0], sum0, g == FOLD - 1);
                        if (live1) fold<TM, kEpi>(acc[1], sum1, g == FOLD - 1);
                    }
            }
            return true;
        };
        if constexpr (!kMoves) {
            add_groups(0, groups);
        } else {
            const uint32_t kZero[16] = {};
            const uint32_t first = taddr + S::kSumCol + cgrp * (S::kSumStep - 16);
            q4fc::tc_st(first, kZero);
            if (live1) q4fc::tc_st(first + CGN * S::kSumStep, kZero);
            // A loop around the groups' loop, which finds anew what it needs, so that the groups' loop keeps its registers
            // (16 x 2816 x 3584, group 32: moving nothing 12.8 us, so 13.5, as a branch in the groups' loop 14.8).
            int end = 0;
#pragma unroll 1
            do {
                const int g = end;
                end = min(g + p.fold * GPS, noted[0]);
                if (!add_groups(g, end)) break;
                const uint32_t at = *reinterpret_cast<volatile uint32_t*>(tmem_slot) + ((threadIdx.x & 96u) << 16) + S::kSumCol;
                const uint32_t w = threadIdx.x >> 7;
                merge_sums(acc, at + w * S::kSumStep, CGN * S::kSumStep, (int)(w + CGN) * 16 < noted[1], end >= noted[0]);
            } while (end < noted[0]);
        }
        if (FMT == kQ8C && groups >= FOLD) {
            if (live0) unfold<TM, kEpi>(acc[0], sum0);
            if (live1) unfold<TM, kEpi>(acc[1], sum1);
        }
        if (cs == 1) {
            const int64_t n = n0 + nrow;
            if (n < p.N && !*abort_flag) {
                const float ws = FMT == kQ8C ? __ldg(p.wscales + n) : 1.0f;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int mc = (cgrp + h * CGN) * 16;
                    float* dst = p.y + (m0 + mc) * p.ldy + n;
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        float lo, hi;
                        unpack2(acc[h][j], lo, hi);
                        if (FMT == kQ8C) lo = __fmul_rn(ws, lo), hi = __fmul_rn(ws, hi);
                        if (mc + 2 * j < live) *dst = lo;
                        dst += p.ldy;
                        if (mc + 2 * j + 1 < live) *dst = hi;
                        dst += p.ldy;
                    }
                }
            }
        } else if (!*abort_flag) {
            // this CTA's partial tile; every operand of this CTA has been consumed (all groups' integers were seen)
            float* red = reinterpret_cast<float*>(smem);
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int m = (cgrp + h * CGN) * 16 + 2 * j;
                    float lo, hi;
                    unpack2(acc[h][j], lo, hi);
                    red[m * kTileN + nrow] = lo, red[(m + 1) * kTileN + nrow] = hi;
                }
        }
    } else if (warp < kMmaWarp) {
        // =================== unpacking: one stripe per warp, one column per lane ===================
        const int pw = warp - kUnpackWarp;
        const int nb = n_tile * 4 + pw;
        const bool stripe_live = nb < p.Ng;  // (columns beyond the weights: nothing is read, nothing is stored)
        const uint8_t* stripe = p.wq + (int64_t)nb * p.Kg * BS;
        auto issue_raw = [&](int i) {
            const int it = it0 + i, slot = (i % S::kRaw) * 4 + pw;
            const uint32_t bytes = (uint32_t)(min(GPS, p.Kg - it * GPS) * BS);
            mbar_expect_tx(bar_raw + 8 * slot, bytes);
            bulk_g2s(smem0 + S::kRawOff + slot * S::kRawStripe, stripe + (int64_t)it * GPS * BS, bytes, bar_raw + 8 * slot);
        };
        if (stripe_live && lane == 0) {
#pragma unroll 1
            for (int i = 0; i < min(S::kRaw, iters); i++) issue_raw(i);
        }
        const uint32_t row = (uint32_t)(pw * 32 + lane);
        const uint32_t row_off = (row >> 3) * 1024 + (row & 7) * 128, sw = (row & 7) << 4;
#pragma unroll 1
        for (int i = 0; i < iters; i++) {
            const int s = i % S::kA, sl = i % S::kScs, rs = (i % S::kRaw) * 4 + pw;
            const int ng = min(GPS, p.Kg - (it0 + i) * GPS);
            if (stripe_live && !wait_or_abort(bar_raw + 8 * rs, (i / S::kRaw) & 1, abort_flag)) break;
            if (!wait_or_abort(bar_aempty + 8 * s, ((i / S::kA) & 1) ^ 1, abort_flag)) break;
            const uint32_t dst = smem0 + s * S::kABytes + row_off;
            const uint32_t src = smem0 + S::kRawOff + rs * S::kRawStripe + lane * 4;
            if (stripe_live) {
                // 16 words at a time: the loads in one batch, then the stores
                // (groups beyond Kg: stale bytes that no MMA reads)
                if constexpr (FMT == kQ8C) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        uint32_t w[16];
#pragma unroll
                        for (int c = 0; c < 16; c++) w[c] = lds32(src + (h * 16 + c) * 128);
#pragma unroll
                        for (int c = 0; c < 4; c++)
                            sts128(dst + ((uint32_t)((h * 4 + c) << 4) ^ sw), w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
                    }
                } else {
                    uint32_t w[16];
#pragma unroll
                    for (int c = 0; c < 16; c++) w[c] = lds32(src + (G == 128 ? c * 128 : (c / 4) * BS + (c % 4) * 128));
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        uint32_t lo0, hi0, lo1, hi1;
                        unpack_nibbles<FMT == kQ4_0Signed>(w[2 * c], lo0, hi0);
                        unpack_nibbles<FMT == kQ4_0Signed>(w[2 * c + 1], lo1, hi1);
                        sts128(dst + ((uint32_t)(c << 4) ^ sw), lo0, hi0, lo1, hi1);
                    }
                }
            }
            if (!wait_or_abort(bar_sempty + 8 * sl, ((i / S::kScs) & 1) ^ 1, abort_flag)) break;
            if constexpr (FMT != kQ8C) {
                uint32_t* wsc = reinterpret_cast<uint32_t*>(smem + S::kScOff + sl * S::kScBytes + S::kXscBytes);
                if (stripe_live) {
#pragma unroll
                    for (int gi = 0; gi < GPS; gi++)
                        if (gi < ng) {
                            const uint32_t tail = src - lane * 2 + gi * BS + 16 * G;
                            uint32_t w = lds16(tail);
                            if (FMT == kQ4_1) w |= lds16(tail + 64) << 16;
                            wsc[gi * kTileN + row] = w;
                        }
                }
            }
            fence_proxy_async();  // generic-proxy stores above -> visible to the tensor core's async proxy
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar_afull + 8 * s);
                mbar_arrive(bar_sfull + 8 * sl);
                if (stripe_live && i + S::kRaw < iters) issue_raw(i + S::kRaw);  // this warp has read the slot
            }
        }
    } else if (warp == kMmaWarp) {
        // =================== MMA issue: one lane ===================
        if (elect_one()) {
            // instruction descriptor: D = s32, A = u8 (s8 where codes are signed), B = s8, both K-major, M = 128,
            // N = the tile's existing rows rounded up to 16
            const uint32_t ncols = (uint32_t)((live + 15) & ~15);
            const uint32_t idesc = (2u << 4) | ((FMT == kQ4_0Signed || FMT == kQ8C ? 1u : 0u) << 7) | (1u << 10) |
                                   ((ncols >> 3) << 17) | ((uint32_t)(kTileN >> 4) << 24);
            const uint64_t desc0 = make_desc(smem0);  // (the start address counts 16-byte units from bit 0)
            int gcount = 0;
            bool ok = true;
#pragma unroll 1
            for (int i = 0; i < iters && ok; i++) {
                const int sa = i % S::kA, sb = i % S::kB;
                if (!wait_or_abort(bar_afull + 8 * sa, (i / S::kA) & 1, abort_flag) ||
                    !wait_or_abort(bar_bfull + 8 * sb, (i / S::kB) & 1, abort_flag)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint64_t a_desc = desc0 + (uint64_t)(sa * (S::kABytes / 16));
                const uint64_t b_desc = desc0 + (uint64_t)((S::kBOff + sb * S::kBBytes) / 16);
                const int ng = min(GPS, p.Kg - (it0 + i) * GPS);
#pragma unroll 1
                for (int gi = 0; gi < ng; gi++, gcount++) {
                    const int b = gcount % S::kBufs;
                    const uint64_t ad = a_desc + (uint64_t)(gi * (G / 16)), bd = b_desc + (uint64_t)(gi * (G / 16));
                    if (!wait_or_abort(bar_tempty + 8 * b, ((gcount / S::kBufs) & 1) ^ 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < MMAS; ks++) {
                        tc_mma_i8(tmem_base + b * TM, ad + ks * 2, bd + ks * 2, idesc, ks > 0 ? 1u : 0u);
                    }
                    tc_commit(bar_tfull + 8 * b);  // the group's integers are complete in TMEM
                }
                tc_commit(bar_aempty + 8 * sa);  // the stage's operands have been consumed
                tc_commit(bar_bempty + 8 * sb);
            }
            // the last commits' arrivals land before this CTA's shared memory can be handed on
            if (ok && iters > 0) {
                wait_or_abort(bar_aempty + 8 * ((iters - 1) % S::kA), ((iters - 1) / S::kA) & 1, abort_flag);
                wait_or_abort(bar_bempty + 8 * ((iters - 1) % S::kB), ((iters - 1) / S::kB) & 1, abort_flag);
            }
        }
    } else {
        // =================== loader: codes and scales of the rows ===================
        if (elect_one()) {
            // The quantizer's results are complete.  (It has let this launch, or the one whose remainder this one does, begin only
            // when everything in front of it was complete.)  A remainder has the quantizer two launches in front of it and does not
            // wait yet for the one between, of whose tiles it reads and writes none.  Why it sees codes and scales all the same:
            // every CTA of that launch has passed its wait, behind which the quantizer's stores are performed and visible to it;
            // a fence at GPU scope, which hands on what a thread has observed, stands between that wait and the release without
            // which the remainder cannot begin, and its counterpart, for the copies too, in front of the first read here.
            // (Waiting here instead: 512 rows x 4096 x 11008 186 -> 188 us, 37 x 4096 x 38000 103 -> 107, 129 x 2080 x 9500 52 -> 59.)
            if (p.part == kRemainder)
                fence_gpu_and_copies();
            else
                pdl_wait_prior_grid();
            if (p.part == kWhole) pdl_launch_dependents();
#pragma unroll 1
            for (int i = 0; i < iters; i++) {
                const int s = i % S::kB, sl = i % S::kScs, it = it0 + i;
                if (!wait_or_abort(bar_bempty + 8 * s, ((i / S::kB) & 1) ^ 1, abort_flag)) break;
                mbar_expect_tx(bar_bfull + 8 * s, S::kBBytes);
                // rows and k beyond the matrix read 0
                tma_load_2d(smem0 + S::kBOff + s * S::kBBytes, &codes_map, bar_bfull + 8 * s, it * kStageK, (int)m0);
                if (!wait_or_abort(bar_sempty + 8 * sl, ((i / S::kScs) & 1) ^ 1, abort_flag)) break;
                const uint32_t bytes = (uint32_t)(min(GPS, p.Kg - it * GPS) * S::kSums * TM * 4);
                mbar_expect_tx(bar_sfull + 8 * sl, bytes);
                bulk_g2s(smem0 + S::kScOff + sl * S::kScBytes,
                         p.sc + ((int64_t)m_tile * p.Kg + (int64_t)it * GPS) * (S::kSums * TM), bytes, bar_sfull + 8 * sl);
                if (p.part == kFirst && i == S::kB - 1) {  // (in front of the first copies the fence costs 2048 rows 297 -> 303 us)
                    fence_gpu_and_copies();
                    pdl_launch_dependents();
                }
            }
            if (p.part == kRemainder) {  // (its end stands for that of the launch in front too)
                pdl_wait_prior_grid();
                pdl_launch_dependents();
            }
        }
    }
    __syncwarp();
    if (cs > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        if (warp < kUnpackWarp && !*abort_flag) {
            // rows rank, rank + cs, ... of the tile: the partial sums of all ranks in rank order
            const float* red = reinterpret_cast<const float*>(smem);
#pragma unroll 1
            for (int m = rank + cs * warp; m < live; m += cs * S::kEpiWarps) {
                uint64_t sum[2] = {}, rest[2] = {};  // columns lane, lane + 32 and lane + 64, lane + 96
#pragma unroll 1
                for (int q = 0; q < cs; q++) {
                    const float* src = cluster.map_shared_rank(red, q) + m * kTileN + lane;
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        const uint64_t v = pack2(src[64 * c], src[64 * c + 32]);
                        if (FMT == kQ8C) {
                            uint64_t r = fadd2(v, rest[c]);
                            sum[c] = move_sum(sum[c], r);
                            finite_or_zero(r);
                            rest[c] = r;
                        } else {
                            sum[c] = q ? fadd2(sum[c], v) : v;
                        }
                    }
                }
                float out[4];
#pragma unroll
                for (int c = 0; c < 2; c++) unpack2(FMT == kQ8C ? fadd2(sum[c], rest[c]) : sum[c], out[2 * c], out[2 * c + 1]);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int64_t n = n0 + lane + 32 * c;
                    if (n < p.N)
                        p.y[(m0 + m) * p.ldy + n] = FMT == kQ8C ? __fmul_rn(__ldg(p.wscales + n), out[c]) : out[c];
                }
            }
        }
        __syncwarp();
        cluster.sync();  // nobody leaves while its partial tile is being read
    }

    // ---- teardown: everyone meets, then the allocating warp frees TMEM
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0 && (atomicCAS(p.status, 0, 0x50524546) & ~kStatusBadId) == 0)  // 'PREF': a bounded wait ran out
            atomicOr(p.status, 0x50524546);
        // copies that may still be in flight land before the shared memory is handed to another CTA
#pragma unroll 1
        for (int i = 0; i < 64; i++) __nanosleep(32000);
    }
    if (warp == kMmaWarp) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"((uint32_t)(kTmemBufs * TM))
                     : "memory");
    }
}

// cuTensorMapEncodeTiled, looked up once through the runtime (the driver library is not linked)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
    // a function-local static is initialised once, also when several host threads arrive together
    static const EncodeTiledFn fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(sym);
        cudaGetLastError();
        return static_cast<EncodeTiledFn>(nullptr);
    }();
    return fn;
}

// the code matrix, rows of `row_bytes`, as a 2-D tensor; boxes of 128 bytes x `tile` rows land in the
// 128-byte-swizzle layout that the MMA descriptors describe; out-of-range rows and k read as 0
int make_codes_map(CUtensorMap* map, const int8_t* codes, int64_t rows, int64_t row_bytes, int tile) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) {
        set_error("fc_prefill: cuTensorMapEncodeTiled is not available from this driver");
        return Q4FC_ECUDA;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)kStageRow, (cuuint32_t)tile};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(codes), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("fc_prefill: cuTensorMapEncodeTiled failed with %d (%lld rows of %lld bytes)", (int)r, (long long)rows,
                  (long long)row_bytes);
        return Q4FC_ECUDA;
    }
    return Q4FC_OK;
}

template <int FMT, int G, int TM, int FOLD = 0>
int launch_prefill_variant(const PrefillParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t s) {
    using S = PrefillShape<FMT, G, TM, FOLD>;
    static std::atomic<bool> attr_done[64] = {};  // set once per device; a second setter repeats the same call
    int dev = 0;
    Q4FC_CUDA_OK(cudaGetDevice(&dev));
    auto* fn = fc_prefill_kernel<FMT, G, TM, FOLD>;
    if (dev >= 64 || !attr_done[dev]) {
        Q4FC_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem));
        Q4FC_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        if (dev < 64) attr_done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(S::kThreads);
    cfg.dynamicSmemBytes = S::kSmem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    // starts beside the quantizer in front of it and waits for that one's results where it needs them
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    Q4FC_CUDA_OK(cudaLaunchKernelEx(&cfg, fn, p, map));
    return Q4FC_OK;
}

template <int FMT, int G>
int launch_prefill_tile(int tile, const PrefillParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t s) {
    if (tile == 128) return launch_prefill_wide(FMT, G, p, map, grid, s);
    if (p.fold == 0) return launch_prefill_variant<FMT, G, 64>(p, map, grid, s);
    return p.rows <= 48 ? launch_prefill_variant<FMT, G, 64, kFewRows>(p, map, grid, s)
                        : launch_prefill_variant<FMT, G, 64, kManyRows>(p, map, grid, s);
}

// tiles first .. end - 1, K divided by p.split
int launch_tiles(int fmt, int G, int tile, PrefillParams p, const CUtensorMap& map, int64_t first, int64_t end, cudaStream_t s) {
    const int64_t wide = end - first < p.n_tiles ? end - first : p.n_tiles;
    p.n_off = (int)(first % p.n_tiles), p.m_off = (int)(first / p.n_tiles);
    p.n_end = (int)(end % p.n_tiles), p.m_end = (int)(end / p.n_tiles);
    const dim3 grid((unsigned)(wide * p.split), (unsigned)((end - first + wide - 1) / wide));
    if (fmt == kQ8C) {
        const bool many = p.Kg > 64 * p.split;  // K groups of a CTA: see the file's head
        if (tile == 128)
            return many ? launch_prefill_variant<kQ8C, 32, 128, 12>(p, map, grid, s)
                        : launch_prefill_variant<kQ8C, 32, 128, 8>(p, map, grid, s);
        return many ? launch_prefill_variant<kQ8C, 32, 64, 12>(p, map, grid, s)
                    : launch_prefill_variant<kQ8C, 32, 64, 8>(p, map, grid, s);
    }
    if (fmt == kQ4_1 && G == 32) return launch_prefill_tile<kQ4_1, 32>(tile, p, map, grid, s);
    if (fmt == kQ4_1) return launch_prefill_tile<kQ4_1, 128>(tile, p, map, grid, s);
    if (fmt == kQ4_0 && G == 32) return launch_prefill_tile<kQ4_0, 32>(tile, p, map, grid, s);
    if (fmt == kQ4_0) return launch_prefill_tile<kQ4_0, 128>(tile, p, map, grid, s);
    if (G == 32) return launch_prefill_tile<kQ4_0Signed, 32>(tile, p, map, grid, s);
    return launch_prefill_tile<kQ4_0Signed, 128>(tile, p, map, grid, s);
}

// scales and group sums of a format, padded to whole row tiles of either size
size_t scale_bytes(int64_t rows, int64_t Kg, int sums) { return (size_t)((rows + 127) / 128 * 128) * Kg * sums * 4; }

// Clusters of 1 .. kMaxSplit CTAs that run at once, one CTA on an SM and two.  Cards differ in where their SMs lie (clusters of three and
// five CTAs: 42 and 24 on one B200, 45 and 26 on another), so the runtime is asked; for an empty kernel, since of a
// 64-row tile's own kernel it counts one CTA on an SM where two run.
__global__ void cluster_room_kernel() {}
struct ClusterRoom {
    int one[kMaxSplit], two[kMaxSplit];
};
const ClusterRoom& cluster_room(const DeviceInfo* di) {
    static std::atomic<bool> known[64] = {};
    static ClusterRoom rooms[64];
    static std::mutex mutex;
    ClusterRoom& room = rooms[di->index];
    if (known[di->index].load(std::memory_order_acquire)) return room;
    std::lock_guard<std::mutex> lock(mutex);
    if (known[di->index].load(std::memory_order_relaxed)) return room;
    for (int places = 1; places <= 2; places++)
        for (int c = 1; c <= kMaxSplit; c++) {
            const int smem = places == 1 ? di->max_smem_optin : 113 * 1024;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(c * di->sm_count)), cfg.blockDim = dim3(64), cfg.dynamicSmemBytes = (size_t)smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)c, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr, cfg.numAttrs = 1;
            int n = 0;
            if (cudaFuncSetAttribute(cluster_room_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
                cudaFuncSetAttribute(cluster_room_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
                cudaOccupancyMaxActiveClusters(&n, cluster_room_kernel, &cfg) != cudaSuccess || n <= 0) {
                cudaGetLastError();
                n = places * di->sm_count / c * 7 / 8;  // a stand-in
                if (n < 1) n = 1;
            }
            (places == 1 ? room.one : room.two)[c - 1] = n;
        }
    known[di->index].store(true, std::memory_order_release);
    return room;
}
// Clusters of an odd number of CTAs find the last of their places late: by how much more the n-th takes (K = 4096, group 32, 64 rows, two
// places on an SM: by three up to 87 tiles 35 us, 90 41, 93 54; 128 rows, one place, up to 43 tiles 30 us, 44 33, 45 38).
float late(int n, int room, int c, float most) {
    const int last = room / 14 > 0 ? room / 14 : 1;
    return c > 1 && c % 2 == 1 && n > room - last ? 1.0f + most * (float)(n - (room - last)) / (float)last : 1.0f;
}

// How tiles of `tile` rows go over the SMs.
struct TilePlan {
    int tile = 0;
    int tiles = 0, split = 1;          // K divided over clusters of `split` CTAs ...
    int left = 0, left_split = 1;      // ... and of the last `left` tiles, in a launch of their own, over `left_split`
    float cost = 0;                    // us
};
// What a stage of 128 k takes, us: a 64-row tile's alone on an SM, and for each 16 rows in use; with a second CTA on the SM; a
// tile's of the wide kernel.  These and the constants in plan_tiles are fitted to the times of 844 calls of 9 to 2048 rows, each in both
// tiles and with every division of K.  What they choose took 0.3 % longer than the best of these in the mean, at most 12 % (rules of their own
// for at most 64 rows, for more and between the tiles, by the clusters that one card holds at once: 2 %, of Q8C 4 %, at most 53 %).
struct StageCost {
    float alone, alone_rows, shared, shared_rows, wide;
};
constexpr StageCost kStageQ4[2][2] = {  // group 128 and 32, each Q4_0 and Q4_1
    {{0.51f, 0.04f, 0.62f, 0.07f, 0.57f}, {0.44f, 0.06f, 0.59f, 0.11f, 0.64f}},
    {{0.97f, 0.20f, 1.16f, 0.29f, 1.65f}, {1.11f, 0.24f, 1.29f, 0.38f, 2.20f}}};
constexpr StageCost kStageQ8C = {0.95f, 0.20f, 1.06f, 0.29f, 0};

// The last tiles of many: K divided over clusters where that takes less than a round more.  In stages: rounds x (stages of a CTA +
// start-up and adding).  (11008 columns, K = 4096: 512 rows, group 32, 48 of 344 tiles left, undivided 177 us, by two 156, by three,
// which takes two rounds, 174; 256 rows, Q8C, 24 of 172, 148 -> 100; 100 rows x 20000, group 32, 18 of 314, 174 -> 106.  Divided where
// this sum says no: 1024 x 4096 x 4096, 108 of 256 left, 125 -> 137.)
int split_of_left(int left, const int* room, int most, int nstage, int startup) {
    float best = (float)nstage;  // undivided, in the launch of the others
    int split = 1;
    for (int c = 2; c <= most; c++) {
        const int full = (left - 1) / room[c - 1], rest = left - full * room[c - 1];
        const float cost = ((float)full + late(rest, room[c - 1], c, 0.25f)) * (float)((nstage + c - 1) / c + startup);
        if (cost < best) best = cost, split = c;
    }
    return split;
}
// Into how many running sums the K of a tile is divided at least (see fold_of).
int least_parts(int n_tiles, int64_t rows, int nstage, int sms) {
    const int64_t tiles = n_tiles * ((rows + 63) / 64);
    const int most = nstage / 4 < kMaxSplit ? nstage / 4 : kMaxSplit;
    return 2 * sms / tiles < most ? (int)(2 * sms / tiles) : most;
}
TilePlan plan_tiles(int tile, int fmt, int G, int n_tiles, int64_t rows, int nstage, const ClusterRoom& at_once, int sms) {
    const bool q8c = fmt == kQ8C, wide = tile == 128 && !q8c;
    const StageCost& stage = q8c ? kStageQ8C : kStageQ4[G == 32][fmt == kQ4_1];
    const int m_tiles = (int)((rows + tile - 1) / tile);
    TilePlan t;
    t.tile = tile, t.tiles = n_tiles * m_tiles;
    const int places = (tile == 128 ? 1 : 2) * sms, most = nstage / 4 < 1 ? 1 : nstage / 4 < kMaxSplit ? nstage / 4 : kMaxSplit;
    const bool few = t.tiles < places;
    const int* room = tile == 128 ? at_once.one : at_once.two;
    // 64-row tiles: 16-row pieces in use, of the fullest tile and in the mean
    const float fullest = rows < 64 ? (float)((rows + 15) / 16) : 4.0f, mean = (float)((rows + 15) / 16) / (float)m_tiles;
    const float alone = stage.alone + stage.alone_rows * fullest;
    const float shared = stage.shared + stage.shared_rows * (few && m_tiles > 1 ? 0.5f * (mean + fullest) : mean);
    // the wide kernel: a tile with fewer rows takes other code, and what it lets stand saves it little (129 to 256 rows x 6144 x
    // 18944, two rounds, the second of tiles with 1, 33, 65, 97 and 128 rows: Q4_0 group 32 68, 78, 90, 95 and 83 us, Q4_1 group
    // 128 29, 30, 33, 37 and 39)
    const int last = (int)((rows - (int64_t)(m_tiles - 1) * tile + 15) / 16);
    const float partial = last == 8 ? 1.0f : 0.75f + 0.05f * (float)last;
    // n tiles, K divided by c: rounds x (start + stages)
    auto launch = [&](int n, int c) {
        const float stages = (float)((nstage + c - 1) / c);
        const int full = (n - 1) / room[c - 1], rest = n - full * room[c - 1];
        if (wide) {
            const float used = full > 0 ? ((float)(m_tiles - 1) + partial) / (float)m_tiles : m_tiles > 1 && partial < 1 ? 1.0f : partial;
            return (6.4f + stages * stage.wide * used) * ((float)full + late(rest, room[c - 1], c, 0.4f));
        }
        const float pair = 4.6f + stages * shared, one = 3.3f + stages * alone;
        if (rest > at_once.one[c - 1]) return pair * ((float)full + late(rest, room[c - 1], c, 0.5f));
        return pair * (float)full + one * (full == 0 ? late(rest, at_once.one[c - 1], c, 0.05f) : 1.0f);
    };
    const float clusters = wide ? 1.9f : 2.3f;  // their start, and adding their parts
    if (few) {
        // K is divided while a CTA keeps four stages
        const int parts = q8c ? 0 : least_parts(n_tiles, rows, nstage, sms);
        for (int c = 1; c <= most; c++) {
            if (wide && parts > 2 * c) continue;  // (whose sums move once)
            const float cost = launch(t.tiles, c) + (c > 1 ? clusters : 0.0f) + (parts > c ? 0.8f : 0.0f);
            if (t.cost == 0 || cost <= t.cost) t.split = c, t.cost = cost;
        }
    } else {
        if (t.tiles % places != 0) t.left_split = split_of_left(t.tiles % places, room, most, nstage, G == 128 ? 8 : 4);
        if (t.left_split > 1) t.left = t.tiles % places;
        t.cost = launch(t.tiles - t.left, 1) + (t.left > 0 ? launch(t.left, t.left_split) + clusters : 0.0f);
    }
    if (wide) t.cost -= 0.6f;
    return t;
}

// Stages of a running sum (Q4), 0: all of a CTA's.  The rounding error of a sum grows with the root of its terms, so that a division of
// K into few parts, where it is the fastest, would be less exact than one into many (49 x 10740 x 9384, group 32: by two 2.38e-7 of
// the result in the 2-norm, by four 1.80e-7).  So no running sum is longer than if K were divided as often as fills two places on every
// SM, and the parts of a CTA are added as those of several would be.
int fold_of(int split, int parts, int nstage) {
    if (parts <= split) return 0;
    const int fold = (nstage + parts - 1) / parts;
    return fold < (nstage + split - 1) / split ? fold : 0;
}

// The wide kernel's codes are fp16 (group 32), twice the bytes.
bool wide_codes_f16(int G) { return G == 32; }
// Quantizer and GEMM; `codes` and `sc` are scratch for [rows][Kg * G] codes of a byte, or two bytes where `wide` allows the wide kernel
// and wide_codes_f16() says so, and for scale_bytes().
int launch_gemm(int fmt, int G, const float* x, int64_t rows, int64_t K, int64_t ldx, int8_t* codes, float* sc, bool wide,
                PrefillParams p, cudaStream_t s) {
    const DeviceInfo* di = device_info();
    if (!di) return Q4FC_ECUDA;
    p.rows = rows, p.sc = sc;
    const int64_t Kp = (int64_t)p.Kg * G;
    if (rows > 0x7fffffffLL || Kp > 0x7fffffffLL) {
        set_error("fc_prefill: rows=%lld or K=%lld beyond the 2^31 coordinate range", (long long)rows, (long long)K);
        return Q4FC_ELIMIT;
    }
    const int64_t all_columns = (p.N + kTileN - 1) / kTileN;
    if (all_columns > 0x7fffffffLL / kMaxSplit || (rows + 63) / 64 > 0x7fffffffLL / kMaxSplit / all_columns) {
        set_error("fc_prefill: %lld rows x %lld columns exceed the grid limit", (long long)rows, (long long)p.N);
        return Q4FC_ELIMIT;
    }
    const int n_tiles = (int)all_columns, nstage = (int)((Kp + kStageK - 1) / kStageK), sms = di->sm_count;
    const ClusterRoom& room = cluster_room(di);
    // 128-row tiles unpack the weights half as often, 64-row tiles run two to an SM.
    TilePlan t;
    if (fmt == kQ8C) {
        // Q8C: the large tile as soon as such tiles occupy every SM (256 rows x 4096 x 11008: 102 us and 108).
        const int tile = rows > 64 && n_tiles * ((rows + 127) / 128) >= sms ? 128 : 64;
        t = plan_tiles(tile, fmt, G, n_tiles, rows, nstage, room, sms);
    } else {
        t = plan_tiles(64, fmt, G, n_tiles, rows, nstage, room, sms);
        if (wide && Kp <= 0x3fffffffLL) {
            // The large tile too where its last tiles are divided, which takes less than the sum (they start beside the others'
            // ends: 129 rows x 2080 x 9500, Q4_0 group 32, 38 us, sum 50, and 45 in 64-row tiles; over 180 calls of many tiles
            // 0.04 % are lost).
            const TilePlan w = plan_tiles(128, fmt, G, n_tiles, rows, nstage, room, sms);
            if (w.cost < t.cost || w.left > 0 || rows > kMaxTileRows * 64) t = w;
        }
    }
    const int tile = t.tile, tiles = t.tiles, split = t.split, left = t.left;
    if (rows > kMaxTileRows * tile) {
        set_error("fc_prefill: %lld rows exceed the grid limit", (long long)rows);
        return Q4FC_ELIMIT;
    }
    p.n_tiles = n_tiles;
    const bool f16 = fmt != kQ8C && tile == 128 && wide_codes_f16(G);
    if (int rc = launch_quant_x_tile(x, rows, K, ldx, G, fmt == kQ4_1, tile, f16, codes, sc, s)) return rc;
    CUtensorMap map = {};
    if (Kp > 0)  // (no K group: no stage reads the map)
        if (int rc = make_codes_map(&map, codes, rows, f16 ? 2 * Kp : Kp, tile)) return rc;
    p.split = split, p.part = left == 0 ? kWhole : kFirst;
    p.fold = fmt == kQ8C || left > 0 ? 0 : fold_of(split, least_parts(n_tiles, rows, nstage, sms), nstage);
    if (int rc = launch_tiles(fmt, G, tile, p, map, 0, tiles - left, s)) return rc;
    if (left == 0) return Q4FC_OK;
    p.split = t.left_split, p.part = kRemainder;
    return launch_tiles(fmt, G, tile, p, map, tiles - left, tiles, s);
}

// workspace: [status 256][what the decode kernels keep between calls: decode_prequant_offset() bytes]
//            [codes of all rows, 256-aligned][scales and group sums]
// The quantized activations start where the decode path's own quantizer scratch starts: calls on one
// workspace are ordered, so the two can share that space, and neither lands on the stream-K stripe
// counters, which must stay zero between calls.
struct WsLayout {
    size_t codes, sc, total;
};
WsLayout ws_layout(int64_t rows, int64_t Kg, int G, bool wide) {
    WsLayout l;
    l.codes = decode_prequant_offset();
    l.sc = align_up(l.codes + (size_t)rows * Kg * G * (wide && wide_codes_f16(G) ? 2 : 1), 256);
    l.total = align_up(l.sc + scale_bytes(rows, Kg, 2), 256);
    return l;
}
bool may_be_wide(int64_t rows) { return rows > 64; }

}  // namespace

size_t prefill_workspace_bytes(int64_t rows, int64_t K, int64_t N, int qtype, int G) {
    (void)N, (void)qtype;
    return ws_layout(rows, (K + G - 1) / G, G, may_be_wide(rows)).total;
}

int launch_fc_prefill(const float* x, int64_t rows, int64_t K, int64_t ldx, const uint8_t* wq, int64_t Ng,
                      int64_t Kg, int qtype, int G, int64_t N, float* y, int64_t ldy, void* ws, size_t ws_bytes,
                      unsigned flags, cudaStream_t s) {
    if (rows == 0 || N == 0) return Q4FC_OK;
    // A workspace without room for fp16 codes (of a size from when there were none, say) does for 64-row tiles.
    bool wide = may_be_wide(rows);
    if (wide && ws_bytes < ws_layout(rows, Kg, G, true).total && rows <= kMaxTileRows * 64) wide = false;
    const WsLayout l = ws_layout(rows, Kg, G, wide);
    if (ws == nullptr || ws_bytes < l.total) {
        set_error("fc_prefill: workspace of %zu bytes given, %zu needed", ws_bytes, l.total);
        return Q4FC_EWORKSPACE;
    }
    uint8_t* base = static_cast<uint8_t*>(ws);
    PrefillParams p = {};
    p.wq = wq, p.y = y, p.status = reinterpret_cast<int*>(base);
    p.N = N, p.ldy = ldy, p.Ng = (int)Ng, p.Kg = (int)Kg;
    const bool sgn = (flags & Q4FC_FLAG_NIBBLE_SIGNED) && qtype == 0;
    // the reference's 1/16 activation scale of Q4_0 pairs with its x16 nibble shift; neither is materialised
    return launch_gemm(qtype == 1 ? kQ4_1 : sgn ? kQ4_0Signed : kQ4_0, G, x, rows, K, ldx,
                       reinterpret_cast<int8_t*>(base + l.codes), reinterpret_cast<float*>(base + l.sc), wide, p, s);
}

size_t q8c_prefill_scale_bytes(int64_t rows, int64_t Kg) { return scale_bytes(rows, Kg, 1); }

int launch_q8c_prefill(const float* x, int64_t rows, int64_t K, int64_t ldx, const int8_t* wq, const float* wscales,
                       int64_t Ng, int64_t Kg, int64_t N, float* y, int64_t ldy, int8_t* codes, float* sc, cudaStream_t s) {
    PrefillParams p = {};
    p.status = ring_status_word();
    if (!p.status) return Q4FC_ECUDA;
    p.wq = reinterpret_cast<const uint8_t*>(wq), p.wscales = wscales, p.y = y;
    p.N = N, p.ldy = ldy, p.Ng = (int)Ng, p.Kg = (int)Kg;
    return launch_gemm(kQ8C, 32, x, rows, K, ldx, codes, sc, false, p, s);
}

}  // namespace q4fc
