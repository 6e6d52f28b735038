// FC over many activation rows (prefill) in 128-row tiles of Q4 weights: see fc_prefill.cu for the formula, the launches around
// it, the remainder and the division of K, which are the same.
//
// What the 64-row kernel's roles do in warps of their own, and wait for one another over, eight warps do in one stream here: a warp
// takes the sums of its 32 columns x 64 rows from tensor memory, scales them, and unpacks its share of the weights three stages
// ahead, so that arithmetic, loads and unpacking fill one another's latencies.  Beside them one thread issues the MMAs and one the
// copies.  Ten warps, three a scheduler, leave a thread 168 registers: 64 sums and two chunks of 16 rows, one on its way from tensor
// memory while the other is scaled.
//   * A = weights, in tensor memory (four stages).  Group 32: as fp16, where a nibble's own bits are the number n x 2^-24: unpacking
//     is five logic operations for eight weights.  Group 128: int8.
//   * B = activation codes, fp16 (see launch_quant_x_tile) or int8, from the code matrix by TMA.
//   * D = three buffers of 128 columns: with fp16 operands fp32 numbers n x code x 2^-16 summed without rounding (below 2^24 units),
//     so that nothing converts them, with int8 integers (group 128's MMAs alone would take 512 cycles with fp16).
//
// Measured (whole calls, rows x K x N, in the 64-row kernel's form before -> here):
//   512 x 4096 x 11008, Q4_0 g32 186 -> 148 us (312 TOPS), Q4_1 g32 235 -> 196;  2048 rows, Q4_1 g128 296 -> 274 (674 TOPS)
//   one round of 148 tiles, K = 4096 (the quantizer included): Q4_0 g32 76 -> 60 us, Q4_1 g32 96 -> 78, Q4_1 g128 33 -> 31
// A K group of 32 takes 790 cycles (from K = 2048 to 8192), in which a scheduler issues 400 instructions.  What bounds it: the
// latencies of two warps a scheduler that meet at the same buffers.  The FMA pipe has 330 cycles to do (a packed multiplication 2.4, a
// packed fma with three register operands 2.8), broadcasting the scales takes shared memory 260, the MMAs 128; an epilogue
// alone, without unpacking and with a constant for the column's scale, takes 435.  That total moves little with its parts
// (without unpacking -4 %, without tensor loads -10 %, without the scales' loads 0).  Tried and dropped: sixteen warps of 32 rows, 96
// registers (512 rows 169 us); chunks of 32 rows (179); unpacking in four warps of their own, of which one issues the MMAs and one
// the copies (186), with these in two more warps and 128 registers (302: the loads no longer overlap); scalar fmas (+11 %);
// registers handed between roles with setmaxnreg (249, and an illegal instruction under load that reading did not explain).

#include <cooperative_groups.h>

#include <atomic>
#include <type_traits>

#include "prefill_common.cuh"

namespace cg = cooperative_groups;

namespace q4fc {
namespace {

constexpr int TM = 128;        // rows of a tile
constexpr int kTmemBufs = 3;   // accumulators, of TM columns each
constexpr int kA = 4, kAColumns = 32;  // stages of unpacked weights, and the TMEM columns of one
constexpr int kEpiWarps = 8;
constexpr int kThreads = (kEpiWarps + 2) * 32;  // three warps a scheduler leave a thread 168 registers
constexpr int W = 16, kChunks = TM / 2 / W;     // rows a thread takes from tensor memory at a time
constexpr float kWdScale = 1024.0f;             // see launch_quant_x_tile
static_assert(kTmemBufs * TM + kA * kAColumns == 512, "all of an SM's tensor memory");

template <int FMT, int G>
struct WideShape {
    static constexpr bool kF16 = G == 32;                 // operands of the MMA: fp16, else int8
    static constexpr int kBlock = block_bytes(FMT == kQ4_1, G);
    static constexpr int kGroups = kF16 ? 2 : 1;          // K groups per stage (64 or 128 k)
    static constexpr int kMmas = 4 / kGroups;             // per group, each of 32 bytes of a row
    static constexpr int kSums = FMT == kQ4_1 ? 2 : 1;    // per group and row: scale (and group sum)
    static constexpr int kB = 4;                          // stages of activation codes
    static constexpr int kSlots = 8;                      // stages of packed bytes and of the rows' scales
    static constexpr int kAhead = kSlots - kB - 2;        // these are asked for so many stages in front of the codes
    static constexpr int kRawStripe = kGroups * kBlock;   // packed bytes of one stripe in a stage
    static constexpr int kBBytes = TM * kStageRow;
    static constexpr int kRawBytes = 4 * kRawStripe;
    static constexpr int kXscBytes = kGroups * kSums * TM * 4;  // [group][scale | sum][row] fp32
    static constexpr int kSlotBytes = kRawBytes + kXscBytes;
    static constexpr int kSlotOff = kB * kBBytes;
    static constexpr int kBarOff = kSlotOff + kSlots * kSlotBytes;
    static constexpr int kSumOff = kBarOff + 512;
    // where the sums move (FOLD), their second place is behind the barriers
    template <bool FOLD>
    static constexpr int kSmem = kSumOff + (FOLD ? TM * kTileN * 4 : 0) + 1024 /*alignment slack*/;
    static_assert(kSmem<true> <= 227 * 1024, "one CTA on an SM");
    static_assert(TM * kTileN * 4 <= kSlotOff, "the partial tile of a K split takes the place of the codes");
};

// Bounded waits of one thread, or of a whole warp that stays together: they give up after kWaitLimitNs, or as soon as another
// role has raised the abort flag.  What they do when the phase has not ended stands apart, as short as it can be: it is in the
// middle of every role's loop, and the loops together are to stay in the instruction cache.
__device__ __forceinline__ uint32_t globaltimer_low() {
    uint32_t t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}
__device__ __noinline__ bool wait_longer(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
    const uint32_t t0 = globaltimer_low();
    uint32_t aborted = 0;
    do {
        if (mbar_try_wait(bar, parity)) return true;
        asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(aborted) : "r"(abort_flag) : "memory");
    } while (!aborted && globaltimer_low() - t0 < (uint32_t)kWaitLimitNs);
    asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(abort_flag), "r"(1) : "memory");
    return false;
}
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
    if (__builtin_expect(mbar_try_wait(bar, parity), 1)) return true;
    return wait_longer(bar, parity, abort_flag);
}
// Has the phase ended?  Does not wait.  (An answer takes 60 cycles: ask early.)
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}"
        : "=r"(ok)
        : "r"(bar), "r"(parity));
    return ok;
}
// (the lanes of a warp may get different answers, and what follows wants them together)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
    if (__builtin_expect(__all_sync(0xffffffffu, mbar_try_wait(bar, parity)), 1)) return true;
    return __all_sync(0xffffffffu, wait_longer(bar, parity, abort_flag));
}
// D (+)= A x B, A in tensor memory, 32 bytes of K per row
template <bool F16>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
    if constexpr (F16)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accum)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accum)
            : "memory");
}
#define Q4FC_R4(op, v, i) op(v[i]), op(v[i + 1]), op(v[i + 2]), op(v[i + 3])
#define Q4FC_R16(op, v, i) Q4FC_R4(op, v, i), Q4FC_R4(op, v, i + 4), Q4FC_R4(op, v, i + 8), Q4FC_R4(op, v, i + 12)
// W columns of this warp's lanes; the registers hold them behind tc_wait_ld() of the same array
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : Q4FC_R16("=r", r, 0)
        : "r"(taddr));
}
// (the registers pass through, so that nothing that reads them can come before the wait)
__device__ __forceinline__ void tc_wait_ld(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : Q4FC_R16("+r", r, 0));
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// The same as fp16: a nibble's bits in the lowest places of an fp16 are the number nibble x 2^-24, four places further up
// 16 times that, so there is nothing to convert.  k = 0,2 | 4,6 | 1,3 | 5,7; the codes of k = 4..7 are 16 times smaller
// (quant_x_tile_kernel).
template <bool SIGNED>
__device__ __forceinline__ void unpack_nibbles_f16(uint32_t word, uint32_t* o) {
    if (SIGNED) word ^= 0x88888888u;  // n + 8 of the signed n
    const uint32_t odd = word >> 8;
    o[0] = word & 0x000F000Fu, o[1] = word & 0x00F000F0u, o[2] = odd & 0x000F000Fu, o[3] = odd & 0x00F000F0u;
    if (SIGNED) {
        o[0] = hadd2(o[0], 0x80088008u), o[1] = hadd2(o[1], 0x80808080u);
        o[2] = hadd2(o[2], 0x80088008u), o[3] = hadd2(o[3], 0x80808080u);
    }
}
// acc += scaled sums of W rows (+ wm * their group sums); `xs`: the rows' scales, the group sums follow at xs + TM
template <int FMT, bool F16>
__device__ __forceinline__ void accumulate(uint64_t (&acc)[W / 2], const uint32_t (&v)[W], const float* xs, uint64_t wd2,
                                           uint64_t wm2) {
    auto number = [&](int i) { return F16 ? __uint_as_float(v[i]) : __int2float_rn((int)v[i]); };
#pragma unroll
    for (int j = 0; j < W / 4; j++) {
        const ulonglong2 x4 = *reinterpret_cast<const ulonglong2*>(xs + 4 * j);
        const uint64_t i01 = pack2(number(4 * j), number(4 * j + 1)), i23 = pack2(number(4 * j + 2), number(4 * j + 3));
        uint64_t &a = acc[2 * j], &b = acc[2 * j + 1];
        // which factor comes first decides which operands stay at hand: a group of one round's tiles, Q4_1, 128 k 736 and 718 ns, 32 k
        // 549 and 563
        a = F16 ? ffma2(wd2, fmul2(x4.x, i01), a) : ffma2(x4.x, fmul2(wd2, i01), a);
        b = F16 ? ffma2(wd2, fmul2(x4.y, i23), b) : ffma2(x4.y, fmul2(wd2, i23), b);
        if (FMT == kQ4_1) {
            const ulonglong2 g4 = *reinterpret_cast<const ulonglong2*>(xs + TM + 4 * j);
            a = ffma2(wm2, g4.x, a);
            b = ffma2(wm2, g4.y, b);
        }
    }
}

// FOLD: the running sums move to a second place, once, after p.fold stages of 128 k (0.9 us with adding them at the end; see fold_of in
// fc_prefill.cu)
template <int FMT, int G, bool FOLD>
__global__ void __launch_bounds__(kThreads, 1) fc_prefill_wide_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap codes_map) {
    using S = WideShape<FMT, G>;
    constexpr int BS = S::kBlock;
    constexpr int GPS = S::kGroups;
    constexpr int kMmaWarp = kEpiWarps;

    extern __shared__ uint8_t smem_raw[];
    // (the same offset in every CTA of a cluster: the dynamic shared memory starts at the same address)
    // (an offset, and no cast through an integer: shared-memory loads and stores)
    uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
    uint8_t* bars = smem + S::kBarOff;
    const uint32_t smem0 = smem_u32(smem);
    const uint32_t bar_raw = smem0 + S::kBarOff, bar_scales = bar_raw + 8 * S::kSlots, bar_free = bar_scales + 8 * S::kSlots;
    const uint32_t bar_a = bar_free + 8 * S::kSlots;
    const uint32_t bar_bfull = bar_a + 8 * kA, bar_bempty = bar_bfull + 8 * S::kB;
    const uint32_t bar_tfull = bar_bempty + 8 * S::kB, bar_tempty = bar_tfull + 8 * kTmemBufs;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 496);
    volatile int* aborted = reinterpret_cast<volatile int*>(bars + 500);
    const uint32_t abort_flag = smem0 + S::kBarOff + 500;
    static_assert(8 * (3 * S::kSlots + kA + 2 * S::kB + 2 * kTmemBufs) <= 496, "barriers");

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
        for (int i = 0; i < S::kSlots; i++) {
            mbar_init(bar_scales + 8 * i, 1);
            mbar_init(bar_free + 8 * i, kEpiWarps);
        }
        for (int i = 0; i < kA; i++) mbar_init(bar_a + 8 * i, kEpiWarps);
        for (int i = 0; i < S::kB; i++) {
            mbar_init(bar_bfull + 8 * i, 1);
            mbar_init(bar_bempty + 8 * i, 1);  // tcgen05.commit
        }
        for (int i = 0; i < kTmemBufs; i++) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, kEpiWarps);
        }
        *aborted = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
    }
    if (warp == kMmaWarp + 1) {
        if (lane < S::kSlots) mbar_init(bar_raw + 8 * lane, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_proxy_async();
        __syncwarp();
        // The first stages' packed bytes, a lane per stage and stripe, while tensor memory is allocated and the warps meet.  (One thread,
        // behind that: 1398 rows x 694 x 25344, Q4_1 group 128, 135.2 us, so 130.7; 2048 x 4096 x 11008 279.0 and 277.1.)
        const int i = lane >> 2, j = lane & 3, stripes = min(4, p.Ng - n_tile * 4);
        if (i < min(S::kSlots / 2, iters) && j < stripes) {
            const uint32_t bytes = (uint32_t)(min(GPS, p.Kg - (it0 + i) * GPS) * BS), bar = bar_raw + 8 * i;
            if (j == 0) mbar_expect_tx(bar, bytes * stripes);
            bulk_g2s(smem0 + S::kSlotOff + i * S::kSlotBytes + j * S::kRawStripe,
                     p.wq + ((int64_t)(n_tile * 4 + j) * p.Kg + (int64_t)(it0 + i) * GPS) * BS, bytes, bar);
        }
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot, a_tmem = tmem_base + kTmemBufs * TM;

    if (warp < kEpiWarps) {
        // =================== epilogue: 32 lanes x 4 chunks of rows per warp ===================
        uint64_t acc[kChunks][W / 2];  // rows as packed pairs
        const int quarter = warp & 3, half = warp >> 2;
        const int nrow = quarter * 32 + lane;  // tile column n handled by this thread (= TMEM lane)
        if (iters == 0) pdl_wait_prior_grid();  // no K group: nothing else orders the stores behind earlier work
        // chunks are dealt out to the two warps of a quarter in turn, so that few rows still occupy both
        const int mine = min(kChunks, max(0, (live + W - 1) / W - half + 1) / 2);
#pragma unroll
        for (int c = 0; c < kChunks; c++)
#pragma unroll
            for (int i = 0; i < W / 2; i++) acc[c][i] = 0ull;
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * W;
        const int groups = min(p.Kg, it1 * GPS) - it0 * GPS;
        uint32_t v[2][W];
        uint32_t xs = 0;  // the group's scales, as an offset: the compiler keeps to shared-memory loads
        uint64_t wd2 = 0, wm2 = 0;
        // a thread's sums behind the barriers, in 16-byte places of its own: `then`(place, two pairs of rows) for each of them
        [[maybe_unused]] auto sums = [&](auto then) {
            ulonglong2* at = reinterpret_cast<ulonglong2*>(smem + S::kSumOff) + threadIdx.x;
#pragma unroll
            for (int j = 0; j < kChunks * W / 4; j++) {
                uint64_t(&a)[W / 2] = acc[j / (W / 4)];
                then(at[j * kEpiWarps * 32], a[2 * j % (W / 2)], a[2 * j % (W / 2) + 1]);
            }
        };
        auto scale = [&](int c) {
            accumulate<FMT, S::kF16>(acc[c], v[c & 1], reinterpret_cast<const float*>(smem + xs) + c * (2 * W), wd2, wm2);
        };
        // Weights: a warp unpacks half of its 32 columns' share of a stage, kA - 1 stages in front of the one it scales.  (The MMAs
        // that read that place before have ended: this warp has seen the sums of a later one.)
        constexpr int kLead = kA - 1;
        constexpr int kPerFold = 128 / (GPS * G);  // stages of 128 k
        const uint32_t share = quarter * S::kRawStripe + half * (S::kF16 ? BS : 1024) + lane * 4;
        constexpr int kWords = S::kF16 ? 4 : 8, kOut = 16 / kWords;
        uint32_t words[kWords];
        // behind the first or the second of the four chunks: 512 x 4096 x 11008, Q4_0 g32 154 and 150 us, Q4_1 g32 197 and 201; one round,
        // Q4_1 g128, 732 and 749 ns a group
        constexpr int kUnpackAt = G == 32 && FMT != kQ4_1 ? 1 : 0;
        auto load_words = [&](int slot) {
            const uint8_t* src = smem + S::kSlotOff + slot * S::kSlotBytes + share;
#pragma unroll
            for (int c = 0; c < kWords; c++) words[c] = *reinterpret_cast<const uint32_t*>(src + c * 128);
        };
        auto unpack = [&](int place) {
            uint32_t o[16];
#pragma unroll
            for (int c = 0; c < kWords; c++) {
                if constexpr (S::kF16)
                    unpack_nibbles_f16<FMT == kQ4_0Signed>(words[c], o + kOut * c);
                else
                    unpack_nibbles<FMT == kQ4_0Signed>(words[c], o[kOut * c], o[kOut * c + 1]);
            }
            tc_st(a_tmem + ((uint32_t)(quarter * 32) << 16) + place * kAColumns + 16 * half, o);
        };
        // ALL: every chunk has rows.  A chunk is scaled while the next one is on its way from tensor memory, a group's last beside the
        // next group's first, and the barriers are asked ahead of time; no branch divides what the compiler can so set side by side.
        auto run = [&](auto all) {
            constexpr bool ALL = decltype(all)::value;
            int b = 0, sl = 0;                   // buffer, slot of the stage
            uint32_t b_phase = 0, s_phase = 0;
            int usl = 0, place = 0;              // slot and place in tensor memory of the stage that is unpacked
            uint32_t u_phase = 0;
            auto next_unpacked = [&] {
                if (++usl == S::kSlots) usl = 0, u_phase ^= 1;
                if (++place == kA) place = 0;
            };
#pragma unroll 1
            for (int u = 0; u < min(kLead, iters); u++) {
                if (!warp_wait(bar_raw + 8 * usl, u_phase, abort_flag)) return;
                __syncwarp();
                load_words(usl);
                unpack(place);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_a + 8 * place);
                __syncwarp();
                next_unpacked();
            }
            bool full = false, stage = false;    // what was asked for ahead of time is there: the group's sums; the stage's scales and bytes
#pragma unroll 1
            for (int i = 0; i < iters; i++) {
#pragma unroll
                for (int gi = 0; gi < GPS; gi++) {
                    if (gi > 0 && i * GPS + gi >= groups) break;
                    const bool later = gi > 0 || i > 0;
                    if (!full && !warp_wait(bar_tfull + 8 * b, b_phase, abort_flag)) return;
                    if (gi == 0 && !stage) {
                        if (!warp_wait(bar_scales + 8 * sl, s_phase, abort_flag)) return;
                        if (i + kLead < iters && !warp_wait(bar_raw + 8 * usl, u_phase, abort_flag)) return;
                    }
                    __syncwarp();
                    tc_fence_after();
                    const uint32_t at = taddr + b * TM;
                    if (ALL || mine > 0) tc_ld(at, v[0]);
                    const uint32_t sc = S::kSlotOff + sl * S::kSlotBytes;
                    if (gi == 0) load_words(usl);  // (beyond the last stage: stale bytes that no MMA reads)
                    const uint8_t* tail = smem + sc + quarter * S::kRawStripe + gi * BS + 16 * G + lane * 2;
                    const uint16_t wd16 = *reinterpret_cast<const uint16_t*>(tail);
                    const uint16_t wm16 = FMT == kQ4_1 ? *reinterpret_cast<const uint16_t*>(tail + 64) : 0;
                    if (ALL && later) scale(kChunks - 1);  // of the group before
                    if constexpr (FOLD)
                        if (gi == 0 && i == p.fold * kPerFold)
                            sums([](ulonglong2& s, uint64_t& a, uint64_t& b) { s.x = a, s.y = b, a = b = 0; });
                    xs = sc + S::kRawBytes + (gi * (S::kSums * TM) + half * W) * 4;
                    const float wd = h2f(wd16) * (S::kF16 ? kWdScale : 1.0f), wm = h2f(wm16);
                    wd2 = pack2(wd, wd), wm2 = pack2(wm, wm);
                    const uint32_t freed = bar_tempty + 8 * b;
                    if (++b == kTmemBufs) b = 0, b_phase ^= 1;
                    const uint32_t place_now = place, before = sl == 0 ? S::kSlots - 1 : sl - 1;
                    if (gi == 0) next_unpacked();
                    if (gi == GPS - 1)
                        if (++sl == S::kSlots) sl = 0, s_phase ^= 1;
                    // asked now, answered behind the arithmetic
                    uint32_t next_full = 0, next_stage = 1;
                    auto ask = [&] {
                        next_full = mbar_test(bar_tfull + 8 * b, b_phase);
                        if (gi == GPS - 1) {
                            next_stage = mbar_test(bar_scales + 8 * sl, s_phase);
                            if (i + 1 + kLead < iters) next_stage &= mbar_test(bar_raw + 8 * usl, u_phase);
                        }
                    };
                    if (ALL || mine > 0) tc_wait_ld(v[0]);
#pragma unroll
                    for (int c = 0; c < kChunks - 1; c++) {
                        const bool some = ALL || c < mine, more = ALL || c + 1 < mine;
                        if (more) tc_ld(at + (c + 1) * (2 * W), v[(c + 1) & 1]);
                        if (c == 0) ask();
                        if (some) scale(c);
                        if (c == kUnpackAt && gi == 0) unpack(place_now);
                        if (more) tc_wait_ld(v[(c + 1) & 1]);
                    }
                    if (gi == 0) tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(freed);  // the buffer can be overwritten
                        if (gi == 0) {
                            if (i > 0) mbar_arrive(bar_free + 8 * before);  // done with the stage before
                            if (i + kLead < iters) mbar_arrive(bar_a + 8 * place_now);
                        }
                    }
                    __syncwarp();
                    full = __all_sync(0xffffffffu, next_full);
                    if (gi == GPS - 1) stage = __all_sync(0xffffffffu, next_stage);
                }
            }
            if (ALL && groups > 0) scale(kChunks - 1);
        };
        if (mine == kChunks)
            run(std::true_type{});
        else
            run(std::false_type{});
        if constexpr (FOLD)
            if (iters > p.fold * kPerFold) sums([](ulonglong2& s, uint64_t& a, uint64_t& b) { a = fadd2(s.x, a), b = fadd2(s.y, b); });
        if (cs == 1) {
            const int64_t n = n0 + nrow;
            if (n < p.N && !*aborted) {
#pragma unroll
                for (int h = 0; h < kChunks; h++) {
                    const int mc = (half + 2 * h) * W;
                    float* dst = p.y + (m0 + mc) * p.ldy + n;
#pragma unroll
                    for (int j = 0; j < W / 2; j++) {
                        float lo, hi;
                        unpack2(acc[h][j], lo, hi);
                        if (mc + 2 * j < live) *dst = lo;
                        dst += p.ldy;
                        if (mc + 2 * j + 1 < live) *dst = hi;
                        dst += p.ldy;
                    }
                }
            }
        } else if (!*aborted) {
            // This CTA's partial tile, in the place of the codes.  Only MMAs read those, and a warp that has seen the last sums knows them all
            // to have ended.
            float* red = reinterpret_cast<float*>(smem);
#pragma unroll
            for (int h = 0; h < kChunks; h++)
#pragma unroll
                for (int j = 0; j < W / 2; j++) {
                    const int m = (half + 2 * h) * W + 2 * j;
                    float lo, hi;
                    unpack2(acc[h][j], lo, hi);
                    red[m * kTileN + nrow] = lo, red[(m + 1) * kTileN + nrow] = hi;
                }
        }
    } else if (warp == kMmaWarp) {
        // =================== MMA issue: one lane ===================
        if (elect_one()) {
            // instruction descriptor: both operands K-major, M = 128, N = the tile's existing rows rounded up to 16;
            // D = f32, A and B = f16, or D = s32, A = u8 (s8 where codes are signed), B = s8
            const uint32_t ncols = (uint32_t)((live + 15) & ~15);
            const uint32_t types = S::kF16 ? 1u << 4 : (2u << 4) | ((FMT == kQ4_0Signed ? 1u : 0u) << 7) | (1u << 10);
            const uint32_t idesc = types | ((ncols >> 3) << 17) | ((uint32_t)(kTileN >> 4) << 24);
            const uint64_t desc0 = make_desc(smem0);  // (the start address counts 16-byte units from bit 0)
            int b = 0;
            uint32_t b_phase = 1;
            bool ok = true;
#pragma unroll 1
            for (int i = 0; i < iters && ok; i++) {
                const int sa = i % kA, sb = i % S::kB;
                if (!wait_or_abort(bar_a + 8 * sa, (i / kA) & 1, abort_flag) ||
                    !wait_or_abort(bar_bfull + 8 * sb, (i / S::kB) & 1, abort_flag)) {
                    ok = false;
                    break;
                }
                const uint32_t a_at = a_tmem + sa * kAColumns;
                const uint64_t b_desc = desc0 + (uint64_t)(sb * (S::kBBytes / 16));
                const int ng = min(GPS, p.Kg - (it0 + i) * GPS);
#pragma unroll 1
                for (int gi = 0; gi < ng; gi++) {
                    if (!wait_or_abort(bar_tempty + 8 * b, b_phase, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < S::kMmas; ks++) {
                        const int at = gi * S::kMmas + ks;
                        tc_mma<S::kF16>(tmem_base + b * TM, a_at + at * 8, b_desc + at * 2, idesc, ks > 0 ? 1u : 0u);
                    }
                    tc_commit(bar_tfull + 8 * b);  // the group's sums are complete in TMEM
                    if (++b == kTmemBufs) b = 0, b_phase ^= 1;
                }
                tc_commit(bar_bempty + 8 * sb);  // the stage's operands have been consumed
            }
            // the last commits' arrivals land before this CTA's shared memory can be handed on
            if (ok && iters > 0) wait_or_abort(bar_bempty + 8 * ((iters - 1) % S::kB), ((iters - 1) / S::kB) & 1, abort_flag);
        }
    } else {
        // =================== loader: packed weights, codes and scales of the rows ===================
        if (elect_one()) {
            const uint8_t* stripes = p.wq + (int64_t)n_tile * 4 * p.Kg * BS;
            const int live_stripes = min(4, p.Ng - n_tile * 4);  // (columns beyond the weights: nothing is read, nothing is stored)
            auto load_raw = [&](int i) {
                const int it = it0 + i, slot = i % S::kSlots;
                const uint32_t bytes = (uint32_t)(min(GPS, p.Kg - it * GPS) * BS), bar = bar_raw + 8 * slot;
                mbar_expect_tx(bar, bytes * live_stripes);
#pragma unroll 1
                for (int j = 0; j < live_stripes; j++)
                    bulk_g2s(smem0 + S::kSlotOff + slot * S::kSlotBytes + j * S::kRawStripe,
                             stripes + ((int64_t)j * p.Kg + (int64_t)it * GPS) * BS, bytes, bar);
            };
            auto load_scales = [&](int i) {
                const int it = it0 + i, slot = i % S::kSlots;
                const uint32_t bytes = (uint32_t)(min(GPS, p.Kg - it * GPS) * S::kSums * TM * 4), bar = bar_scales + 8 * slot;
                mbar_expect_tx(bar, bytes);
                bulk_g2s(smem0 + S::kSlotOff + slot * S::kSlotBytes + S::kRawBytes,
                         p.sc + ((int64_t)m_tile * p.Kg + (int64_t)it * GPS) * (S::kSums * TM), bytes, bar);
            };
            const int first = min(S::kSlots / 2, iters);
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
            bool ok = true;
#pragma unroll 1
            for (int i = 0; i < iters && ok; i++) {
                const int s = i % S::kB, j = i + S::kAhead;
                ok = wait_or_abort(bar_bempty + 8 * s, ((i / S::kB) & 1) ^ 1, abort_flag);
                if (!ok) break;
                mbar_expect_tx(bar_bfull + 8 * s, S::kBBytes);
                // rows and k beyond the matrix read 0
                tma_load_2d(smem0 + s * S::kBBytes, &codes_map, bar_bfull + 8 * s, (it0 + i) * kStageRow, (int)m0);
                if (i == 0) {  // (the other half of the slots; in front of the first codes it is in their way)
#pragma unroll 1
                    for (int k = first; k < min(S::kSlots, iters); k++) load_raw(k);
#pragma unroll 1
                    for (int k = 0; k < min(S::kAhead, iters); k++) load_scales(k);
                }
                if (j < iters) {
                    if (j >= S::kSlots) {
                        ok = wait_or_abort(bar_free + 8 * (j % S::kSlots), ((j / S::kSlots) & 1) ^ 1, abort_flag);
                        if (!ok) break;
                        load_raw(j);
                    }
                    load_scales(j);
                }
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
        if (warp < kEpiWarps && !*aborted) {
            // rows rank, rank + cs, ... of the tile: the partial sums of all ranks in rank order
            const float* red = reinterpret_cast<const float*>(smem);
#pragma unroll 1
            for (int m = rank + cs * warp; m < live; m += cs * kEpiWarps) {
                uint64_t sum[2] = {};  // columns lane, lane + 32 and lane + 64, lane + 96
#pragma unroll 1
                for (int q = 0; q < cs; q++) {
                    const float* src = cluster.map_shared_rank(red, q) + m * kTileN + lane;
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        const uint64_t v = pack2(src[64 * c], src[64 * c + 32]);
                        sum[c] = q ? fadd2(sum[c], v) : v;
                    }
                }
                float out[4];
                unpack2(sum[0], out[0], out[1]), unpack2(sum[1], out[2], out[3]);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int64_t n = n0 + lane + 32 * c;
                    if (n < p.N) p.y[(m0 + m) * p.ldy + n] = out[c];
                }
            }
        }
        __syncwarp();
        cluster.sync();  // nobody leaves while its partial tile is being read
    }

    // ---- teardown: everyone meets, then the allocating warp frees TMEM
    tc_fence_before();
    __syncthreads();
    if (*aborted) {
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
                     "r"(512u)
                     : "memory");
    }
}

template <int FMT, int G, bool FOLD>
int launch_variant(const PrefillParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t s) {
    using S = WideShape<FMT, G>;
    static std::atomic<bool> attr_done[64] = {};  // set once per device; a second setter repeats the same call
    int dev = 0;
    Q4FC_CUDA_OK(cudaGetDevice(&dev));
    auto* fn = fc_prefill_wide_kernel<FMT, G, FOLD>;
    if (dev >= 64 || !attr_done[dev]) {
        Q4FC_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, S::template kSmem<FOLD>));
        Q4FC_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        if (dev < 64) attr_done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = S::template kSmem<FOLD>;
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
int launch_fold(const PrefillParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t s) {
    return p.fold > 0 ? launch_variant<FMT, G, true>(p, map, grid, s) : launch_variant<FMT, G, false>(p, map, grid, s);
}

}  // namespace

int launch_prefill_wide(int fmt, int G, const PrefillParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t s) {
    if (fmt == kQ4_1) return G == 32 ? launch_fold<kQ4_1, 32>(p, map, grid, s) : launch_fold<kQ4_1, 128>(p, map, grid, s);
    if (fmt == kQ4_0) return G == 32 ? launch_fold<kQ4_0, 32>(p, map, grid, s) : launch_fold<kQ4_0, 128>(p, map, grid, s);
    return G == 32 ? launch_fold<kQ4_0Signed, 32>(p, map, grid, s) : launch_fold<kQ4_0Signed, 128>(p, map, grid, s);
}

}  // namespace q4fc
