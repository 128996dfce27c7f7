// Quantised GEMM on tcgen05 for Q8_0, Q4_0, Q5_K and Q6_K (on its row-planar copy), eight or more activation rows, and for Q4_K from 65 on:
//
//     out[n][r] = Σ_k W[r][k] · x[n][k]
//
// The sibling of the kernel in qgemm_tc.cu: the same roles, activation tiles, work items and two MMAs per product, W·x_hi and W·x_lo, because
// the W operand is an exact integer in fp16 and its scale is multiplied in after the drain, in fp32.  What differs is where the scale changes:
//
//   Q8_0, Q4_0  one d per 32 columns: q (-128 .. 127; q − 8) is the operand, and a stage of 64 columns fills two accumulators, one per block.  The d
//               of a (row, block) goes from the unpacking warps to the drain warps through shared memory.
//   Q4_K, Q5_K  sc·(q − 8), sc·(q − 16) (|.| ≤ 1008), drained with d.  What the centring and the minimum leave, c = 8·d·sc − dmin·m (16) per 32 columns,
//               meets the sub-block sums of x in one more accumulator per super-block: c is formed in fp32, scaled by a power of two that d and dmin
//               give (both sides compute it) and split into fp16 hi + lo.  (Summing q and the minimum apart, as qgemm_tc.cu does, doubles the error.)
//   Q6_K        sc·(q − 32) has up to 13 bits: hi (rounded to 11) and lo (the rest, exact), three MMAs per 16 columns, drained with d.
//
// An accumulator of Q4_K holds two stages, which halves the drains: gate / up of the 8B shape against 2047 rows 894 us in qgemm_tc.cu, 831 here (1160 TFLOP/s of MMAs; cuBLAS
// sustains 1397; both as first measured), error against 64 bits 2.8e-7 and 1.3e-7.  The others hold one: two would take 7 to 12 % less time, but the adder truncates, and at 2048
// columns the error would be 1.3e-7 where the kernel that these formats had before gave 1.25e-7.
//
// The weights arrive as tiled TMA boxes of one super-block (256 columns) of 128 rows: Q8_0 272 bytes a row, Q4_K and Q4_0 144, Q5_K 176 (odd multiples of 16: eight
// lanes cover all banks), Q6_K its ql, qh and scale planes, the first two swizzled for the same reason.  Rows past the end of the matrix arrive as zeros.
//
// Before, the formats other than Q4_K went through the dequantising kernel of qgemm_tc.cu: three MMAs per product, W as fp16 hi + lo of the dequantised value, raw bytes
// fetched by the unpacking warps themselves between two barriers of theirs.  The linears of an 8B layer against 1000 rows, ms, before and now: Q8_0 2.35, 1.20, Q4_0 2.16,
// 1.17, Q5_K 3.51, 1.02, Q6_K 2.66, 1.03 (of the tensor pipe at its measured rate 35, 36, 41 and, with three MMAs, 61 %); Q6_K 2048x5632 by 777 rows 162, 64 us.
//
// 20 warps: 0-7 drain, 8 loads x, 9 and 11 issue MMAs in turns, 10 loads W, 12-19 unpack; barriers, rings and the reasons as in qgemm_tc.cu.
// Every wait is bounded.

#include <cstring>
#include <mutex>
#include <type_traits>

#include <cuda.h>

#include "internal.h"
#include "qgemm_common.cuh"

namespace yule {
namespace {

enum Fmt { kQ8, kQ4, kQ5K, kQ6K, kQ4K };

constexpr int kProdWarps = 8;
constexpr int kLoaderWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1, kRawWarp = kEpiWarps + 2, kMmaWarp2 = kEpiWarps + 3, kFirstProdWarp = kEpiWarps + 4;
constexpr int kThreads = (kEpiWarps + 4 + kProdWarps) * 32;  // 640
constexpr int kLaunchRegs = 96;  // registers per thread that 640 threads are launched with (the build checks that the 128-row kernels get them)
// Registers move to the drain warps, which at 128 activation rows hold 64 sums beside what they read, below three sets of up to 32: together no more than the launch brought.
template <bool TWO_SETS>
struct Registers {
    static constexpr int kDrain = TWO_SETS ? 168 : 144, kControl = 32, kProd = TWO_SETS ? 56 : 80;
    static_assert(kEpiWarps * kDrain + 4 * kControl + kProdWarps * kProd <= (kEpiWarps + 4 + kProdWarps) * kLaunchRegs, "register split");
};
constexpr uint32_t kStages = 4;    // of the operand ring: W in tensor memory, x in shared memory; a stage is 64 columns
constexpr uint32_t kMaxAcc = 8, kMaxRaw = 8;
constexpr uint32_t kScaleRing = 8;  // stages whose block scales are kept for the drains (see Tile)
constexpr size_t kMaxSmem = 227 * 1024;

constexpr int kMapsPerMatrix = 3;  // Q6_K: ql, qh, scales; else one
struct IntMaps {
    CUtensorMap m[kGemmSegs][kMapsPerMatrix];
};

template <int FMT, int BN>
struct Tile {
    static constexpr bool MERGED = BN <= 64;  // hi and lo rows of x as one operand of 2·BN rows, as in the Q4_K kernel
    static constexpr bool BLOCK32 = FMT == kQ8 || FMT == kQ4, OFFSET = FMT == kQ5K || FMT == kQ4K, WLO = FMT == kQ6K;
    static constexpr uint32_t kMainCols = MERGED ? 2 * BN : BN;
    static constexpr uint32_t CW = BN / 2;                 // columns per drain warp
    static constexpr uint32_t kXHalfBytes = BN * 64 * 2;   // one fp16 term of the activation slab
    static constexpr uint32_t kBmBytes = BN * 16 * 2;      // sub-block sums of x
    static constexpr uint32_t kSuperBytes = 8 * kXHalfBytes + kBmBytes;
    static constexpr uint32_t kACols = (WLO ? 2 : 1) * 32;  // tensor-memory columns of a stage's W (hi, then lo)
    static constexpr uint32_t kAccs = BLOCK32 ? 2 : 1;      // accumulators a stage fills
    static constexpr uint32_t kAccFit = (512 - kStages * kACols) / kMainCols;
    static constexpr uint32_t NBUF = kAccFit < kMaxAcc ? kAccFit : kMaxAcc;
    // The issuing warps know an accumulator barrier's parity only (qgemm_tc.cu): the drain of the use before last has to be known to be over, which
    // takes a ring one longer than what lies between two stages of a warp.  A scale of stage j lies where that of stage j - 8 was: stage j is
    // unpacked once the MMAs of stage j - 4 are done, whose accumulators were free, so the drains are past accumulator 2 (j - 4) + 1 - NBUF.
    static_assert(NBUF >= kAccs + (OFFSET ? 2 : 1) && (!BLOCK32 || 7 + NBUF <= 2 * kScaleRing - 1), "accumulator ring");
    static constexpr uint32_t kABase = NBUF * kMainCols;
    static_assert(kABase + kStages * kACols <= 512, "tensor memory");
    static constexpr uint32_t kSpan = FMT == kQ4K ? 2 : 1;  // stages that an accumulator holds (with kSpan = 1 and BLOCK32: half of one)
    static constexpr uint32_t kStageBytes = 2 * kXHalfBytes;
    // Behind the last slot, which is where every super-block's last stage lies: the sub-block sums of x (one bulk copy brings them with that stage)
    // and the offset's operand, c_hi | c_hi | c_lo | c_lo, eight columns each.
    static constexpr uint32_t kOffSums = kStages * kStageBytes, kOffOffset = kOffSums + (OFFSET ? kBmBytes : 0u);
    static constexpr uint32_t kOffRaw = kOffOffset + (OFFSET ? kTileRows * 32 * 2 : 0u);
    static constexpr uint32_t kRawRow = FMT == kQ8 ? 272 : FMT == kQ5K ? 176 : 144;
    static constexpr uint32_t kRawBytes = FMT == kQ6K ? kTileRows * 208 : kTileRows * kRawRow;
    static constexpr uint32_t kScaleBytes = BLOCK32 ? kScaleRing * 2 * kTileRows * 4 : 0;
    static constexpr uint32_t kTailBytes = (2 * kStages + 2 * kMaxAcc + 2 * kMaxRaw) * 8 + 32;
    static constexpr uint32_t kFixed = 1024 + kOffRaw + kScaleBytes + kTailBytes;  // (1024: the swizzled planes start on such boundaries)
    static constexpr uint32_t kRawFit = (kMaxSmem - kFixed) / kRawBytes;
    static constexpr uint32_t kRaw = kRawFit < 6 ? kRawFit : 6;  // super-blocks of raw bytes in flight
    static_assert(kRaw >= 2, "shared memory");
    static constexpr size_t kSmem = kFixed + kRaw * kRawBytes;
};

// Power of two that both sides of Q5_K's offset use: |16·d·sc − dmin·m| times it stays below 2^14.
__device__ __forceinline__ uint32_t offset_exponent(float d, float dmin) {
    const float bound = fmaxf(1008.f * fabsf(d), 63.f * fabsf(dmin)) * 2.f;
    const uint32_t e = __float_as_uint(bound) >> 23;  // 2^(e - 127) ≤ bound < 2^(e - 126)
    return e < 20u ? 20u : e;                         // (no d and no dmin: anything finite)
}
__device__ __forceinline__ float offset_scale(uint32_t e) { return __uint_as_float((127u + 13u + 127u - e) << 23); }      // 2^(13 - (e - 127))
__device__ __forceinline__ float offset_unscale(uint32_t e) { return __uint_as_float((e - 13u) << 23); }

// 32-bit words of a run of N words that starts at byte AT of the 16-byte chunks `c` (AT even)
template <uint32_t AT, int N, int C>
__device__ __forceinline__ void words_in(const uint4 (&c)[C], uint32_t (&w)[N]) {
    auto word = [&](uint32_t i) {
        const uint4 &q = c[i >> 2];
        return (i & 3u) == 0 ? q.x : (i & 3u) == 1 ? q.y : (i & 3u) == 2 ? q.z : q.w;
    };
#pragma unroll
    for (int k = 0; k < N; k++) w[k] = (AT & 2u) ? __funnelshift_r(word(AT / 4 + k), word(AT / 4 + k + 1), 16) : word(AT / 4 + k);
}

template <int FMT, int BN>
__global__ void __launch_bounds__(kThreads, 1) qgemm_int_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ IntMaps w_maps) {
    using T = Tile<FMT, BN>;
    constexpr uint32_t NBUF = T::NBUF, CW = T::CW, kXHalfBytes = T::kXHalfBytes, kStageBytes = T::kStageBytes;
    extern __shared__ unsigned char smem_raw[];
    yule_pdl_launch_dependents();
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    unsigned char *smem = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);  // stages | raw boxes | scales | barriers
    unsigned char *raw = smem + T::kOffRaw;
    static_assert(T::kOffRaw % 1024 == 0 && (FMT != kQ6K || T::kRawBytes % 1024 == 0), "swizzle");
    float *scales = reinterpret_cast<float *>(raw + T::kRaw * T::kRawBytes);  // BLOCK32: [kScaleRing][2][128]
    uint64_t *bars = reinterpret_cast<uint64_t *>(reinterpret_cast<unsigned char *>(scales) + T::kScaleBytes);
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kStages;
    const uint32_t bar_acc_full = bar_empty + 8 * kStages, bar_acc_empty = bar_acc_full + 8 * kMaxAcc;
    const uint32_t bar_raw_full = bar_acc_empty + 8 * kMaxAcc, bar_raw_empty = bar_raw_full + 8 * kMaxRaw;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kStages + 2 * kMaxAcc + 2 * kMaxRaw);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; s++) {
            mbar_init(bar_full + 8 * s, kProdWarps + 1);  // one arrival per unpacking warp + the loader's expect_tx
            mbar_init(bar_empty + 8 * s, 1);              // tcgen05.commit
        }
        for (uint32_t b = 0; b < NBUF; b++) {
            // tcgen05.commit and, where the drains read scales that the unpacking warps stored, an arrival of the thread that saw those complete
            mbar_init(bar_acc_full + 8 * b, T::BLOCK32 ? 2 : 1);
            mbar_init(bar_acc_empty + 8 * b, kEpiWarps);
        }
        for (uint32_t b = 0; b < T::kRaw; b++) {
            mbar_init(bar_raw_full + 8 * b, 1);            // the loader's expect_tx
            mbar_init(bar_raw_empty + 8 * b, kProdWarps);  // every unpacking warp is done with the box
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    const uint32_t bpr = p.n_cols / 256;  // super-blocks per row

    if (warp >= kEpiWarps && warp < kFirstProdWarp) {
        move_registers<true, Registers<T::BLOCK32 && !T::MERGED>::kControl, kLaunchRegs>();
        if (warp == kLoaderWarp) {
            if (lane == 0) {
                yule_pdl_wait();  // the activation tiles come from the kernel before this one
                RingPos ring;
                bool ok = true;
                ItemWalk items(p);
                    for (Item wi; ok && items.next(p, bpr, wi);) {
                    const unsigned char *src = reinterpret_cast<const unsigned char *>(p.xb) + (size_t)wi.nt * bpr * T::kSuperBytes;
                    for (uint32_t kb = 4 * wi.sb0; kb < 4 * wi.sb1; kb++, ring.advance(kStages)) {
                        const uint32_t s = ring.s;
                        ok = mbar_wait(bar_empty + 8 * s, ring.ph ^ 1u, abort_flag, p.status);
                        if (!ok) break;
                        const uint32_t g = kb & 3u, bytes = 2 * kXHalfBytes + ((T::OFFSET && g == 3) ? T::kBmBytes : 0u);  // the sums ride with the last stage
                        mbar_arrive_expect_tx(bar_full + 8 * s, bytes);
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                         smem_u32(smem + (size_t)s * kStageBytes)),
                                     "l"(src + (size_t)(kb >> 2) * T::kSuperBytes + (size_t)g * 2 * kXHalfBytes), "r"(bytes), "r"(bar_full + 8 * s)
                                     : "memory");
                    }
                }
            }
        } else if (warp == kMmaWarp || warp == kMmaWarp2) {
            const uint32_t mine = warp == kMmaWarp ? 0u : 1u;
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);  // fp16 × fp16 → fp32, K-major, M = 128, N = BN
            [[maybe_unused]] constexpr uint32_t idesc2 = (1u << 4) | ((uint32_t)((2 * BN) >> 3) << 17) | ((uint32_t)(kTileRows >> 4) << 24);
            constexpr uint32_t x_lbo = BN * 16;  // bytes of one 8-column step of an activation slab (of its hi or lo rows)
            bool ok = true;
            RingPos ring, acc;
            ItemWalk items(p);
                for (Item wi; ok && items.next(p, bpr, wi);) {
                for (uint32_t kb = 4 * wi.sb0; kb < 4 * wi.sb1 && ok; kb += T::kSpan, ring.advance(kStages)) {
                    const bool closes = T::OFFSET && (kb & 3u) == 4u - T::kSpan;
                    if ((kb / T::kSpan & 1u) != mine) {
#pragma unroll
                        for (uint32_t i = 0; i < T::kAccs; i++) acc.advance(NBUF);
                        if (closes) acc.advance(NBUF);
                        if (T::kSpan == 2) ring.advance(kStages);
                        continue;
                    }
                    auto await = [&](uint32_t bar, uint32_t parity) { ok = ok && mbar_wait(bar, parity, abort_flag, p.status); };
                    auto all_ok = [&] {
                        ok = __all_sync(0xffffffffu, ok);
                        tc_fence_after();
                        return ok;
                    };
                    // The 16-column steps [K0, K1) of ring slot s.  The adder truncates, which costs a part of what the accumulator holds, so the
                    // products with lo terms go first (`small`), or to columns of their own.
                    auto w_at = [&](uint32_t s) { return tmem_base + T::kABase + s * T::kACols; };
                    auto x_at = [&](uint32_t s) { return smem_desc(smem_u32(smem + (size_t)s * kStageBytes), T::MERGED ? 2 * x_lbo : x_lbo, 128); };
                    auto small = [&](auto k0c, auto k1c, auto freshc, uint32_t d_main, uint32_t s) {
                        constexpr uint32_t K0 = decltype(k0c)::value, K1 = decltype(k1c)::value;
                        const uint32_t w0 = w_at(s);
                        const uint64_t db0 = x_at(s);
                        mma_steps<K0, K1>([&](auto kc) {
                            constexpr uint32_t k = decltype(kc)::value;
                            constexpr int add = k != K0 || !decltype(freshc)::value;
                            if constexpr (T::MERGED) {
                                const uint64_t db = db0 + (uint64_t)((k * 4u * x_lbo) >> 4);
                                umma_f16_ts<add>(d_main, w0 + 8 * k, db, idesc2);
                                if (T::WLO) umma_f16_ts<1>(d_main + BN, w0 + 32 + 8 * k, db, idesc);  // W_lo·x_hi beside the other small products
                            } else {
                                const uint64_t db = db0 + (uint64_t)((k * 2u * x_lbo) >> 4);
                                umma_f16_ts<add>(d_main, w0 + 8 * k, db + (uint64_t)(kXHalfBytes >> 4), idesc);
                                if (T::WLO) umma_f16_ts<1>(d_main, w0 + 32 + 8 * k, db, idesc);
                            }
                        });
                    };
                    auto large = [&](auto k0c, auto k1c, uint32_t d_main, uint32_t s) {
                        if constexpr (!T::MERGED) {
                            const uint32_t w0 = w_at(s);
                            const uint64_t db0 = x_at(s);
                            mma_steps<decltype(k0c)::value, decltype(k1c)::value>([&](auto kc) {
                                constexpr uint32_t k = decltype(kc)::value;
                                umma_f16_ts<1>(d_main, w0 + 8 * k, db0 + (uint64_t)((k * 2u * x_lbo) >> 4), idesc);
                            });
                        }
                    };
                    constexpr std::integral_constant<uint32_t, 0> k0{};
                    constexpr std::integral_constant<uint32_t, 2> k2{};
                    constexpr std::integral_constant<uint32_t, 4> k4{};
                    constexpr std::true_type fresh{};
                    if constexpr (T::kSpan == 2) {
                        const uint32_t d_main = tmem_base + acc.s * T::kMainCols, s0 = ring.s;
                        await(bar_acc_empty + 8 * acc.s, acc.ph ^ 1u);
                        await(bar_full + 8 * s0, ring.ph);
                        if (!all_ok()) break;
                        if (elect_one()) small(k0, k4, fresh, d_main, s0);
                        __syncwarp();
                        ring.advance(kStages);
                        await(bar_full + 8 * ring.s, ring.ph);
                        if (!all_ok()) break;
                        if (elect_one()) {
                            small(k0, k4, std::false_type{}, d_main, ring.s);
                            large(k0, k4, d_main, s0);
                            umma_commit(bar_empty + 8 * s0);
                            large(k0, k4, d_main, ring.s);
                            umma_commit(bar_acc_full + 8 * acc.s);
                            if (!closes) umma_commit(bar_empty + 8 * ring.s);
                        }
                        __syncwarp();
                        acc.advance(NBUF);
                    } else {
                        const uint32_t s = ring.s;
                        auto fill = [&](auto k0c, auto k1c, bool last) {
                            await(bar_acc_empty + 8 * acc.s, acc.ph ^ 1u);
                            if (decltype(k0c)::value == 0) await(bar_full + 8 * s, ring.ph);
                            if (!all_ok()) return;
                            if (elect_one()) {
                                const uint32_t d_main = tmem_base + acc.s * T::kMainCols;
                                small(k0c, k1c, fresh, d_main, s);
                                large(k0c, k1c, d_main, s);
                                umma_commit(bar_acc_full + 8 * acc.s);
                                if (last) umma_commit(bar_empty + 8 * s);
                                if (T::BLOCK32) mbar_arrive(bar_acc_full + 8 * acc.s);
                            }
                            __syncwarp();
                            acc.advance(NBUF);
                        };
                        if constexpr (T::BLOCK32) {
                            fill(k0, k2, false);
                            if (!ok) break;
                            fill(k2, k4, true);
                        } else {
                            fill(k0, k4, !closes);
                        }
                        if (!ok) break;
                    }
                    if (closes) {  // Σ_s c_s · (sum of x over sub-block s): the lo terms of c, then the hi terms, against hi and lo sums side by side
                        await(bar_acc_empty + 8 * acc.s, acc.ph ^ 1u);
                        if (!all_ok()) break;
                        if (elect_one()) {
                            const uint32_t d_off = tmem_base + acc.s * T::kMainCols, c_at = smem_u32(smem + T::kOffOffset);
                            const uint64_t sums = smem_desc(smem_u32(smem + T::kOffSums), x_lbo, 128);
                            umma_f16(d_off, smem_desc(c_at + 4096, 2048, 128), sums, idesc, 0u);
                            umma_f16(d_off, smem_desc(c_at, 2048, 128), sums, idesc, 1u);
                            umma_commit(bar_acc_full + 8 * acc.s);
                            umma_commit(bar_empty + 8 * ring.s);
                        }
                        __syncwarp();
                        acc.advance(NBUF);
                    }
                }
            }
        } else if (warp == kRawWarp) {
            if (lane == 0) {
                UnitWalk walk(p, bpr);
                for (uint32_t u = 0; walk.live; u++, walk.next(p, bpr)) {
                    const uint32_t slot = u % T::kRaw, ph = (u / T::kRaw) & 1u;
                    if (!mbar_wait(bar_raw_empty + 8 * slot, ph ^ 1u, abort_flag, p.status)) break;
                    const uint32_t dst = smem_u32(raw + (size_t)slot * T::kRawBytes), bar = bar_raw_full + 8 * slot, y = walk.it.mt * kTileRows;
                    auto box = [&](int map, uint32_t x, uint32_t to) {
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(to),
                                     "l"(reinterpret_cast<uint64_t>(&w_maps.m[walk.it.seg][map])), "r"(bar), "r"(x), "r"(y)
                                     : "memory");
                    };
                    mbar_arrive_expect_tx(bar, T::kRawBytes);
                    if constexpr (FMT == kQ6K) {
                        box(0, walk.sb * 128, dst);
                        box(1, walk.sb * 64, dst + kTileRows * 128);
                        box(2, walk.sb * 16, dst + kTileRows * 192);
                    } else {
                        box(0, walk.sb * (T::kRawRow / 8), dst);  // elements of eight bytes, an even number of them
                    }
                }
            }
        }
    } else if (warp >= kFirstProdWarp) {
        move_registers<true, Registers<T::BLOCK32 && !T::MERGED>::kProd, kLaunchRegs>();
        const uint32_t ptid = threadIdx.x - kFirstProdWarp * 32;
        const uint32_t r = ptid & 127u, hf = __shfl_sync(0xffffffffu, ptid >> 7, 0);  // row of the tile, half of the work on it
        bool ok = true;
        RingPos ring;
        uint32_t n_stage = 0;
        const uint32_t w_lanes = tmem_base + T::kABase + ((warp & 3u) << 21);  // this warp's 32 lanes
        auto open = [&]() {
            ok = mbar_wait(bar_empty + 8 * ring.s, ring.ph ^ 1u, abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok);  // (a warp stays together: its stores are the warp's)
            tc_fence_after();
            return ok;
        };
        auto close = [&]() {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_full + 8 * ring.s);
            ring.advance(kStages);
            n_stage++;
        };
        const __half2 k1024 = __half2half2(__ushort_as_half(0x6400));
        // Q8_0, Q4_0: block 2g + HF of the row, in the 16-byte chunks that hold it
        [[maybe_unused]] auto block32 = [&](auto gc, auto hfc, const unsigned char *row) {
            constexpr uint32_t g = decltype(gc)::value, HF = decltype(hfc)::value, SIZE = FMT == kQ8 ? 34 : 18, C = FMT == kQ8 ? 3 : 2;
            constexpr uint32_t at = SIZE * (2 * g + HF), first = at / 16, in = at & 15u;
            uint4 c[C];
#pragma unroll
            for (uint32_t i = 0; i < C; i++) c[i] = *reinterpret_cast<const uint4 *>(row + 16 * (first + i));
            uint32_t dw[1];
            words_in<(in & ~3u)>(c, dw);
            const float d = __half2float(__ushort_as_half((unsigned short)(dw[0] >> (8 * (in & 2u)))));
            uint32_t w[FMT == kQ8 ? 8 : 4];
            words_in<in + 2>(c, w);
            if (!open()) return;
            scales[(n_stage % kScaleRing) * 2 * kTileRows + HF * kTileRows + r] = d;
            const uint32_t to = w_lanes + ring.s * T::kACols + HF * 16;
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                uint4 v[2];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    if constexpr (FMT == kQ8) {  // byte ^ 128 = byte + 128
                        const __half2 bias = as_half2(0x64806480u);
                        const uint32_t a = w[2 * (i + j)] ^ 0x80808080u, b = w[2 * (i + j) + 1] ^ 0x80808080u;
                        auto two = [&](uint32_t x) { return as_u32(__hsub2(as_half2((x & 0x00FF00FFu) | 0x64006400u), bias)); };
                        v[j] = make_uint4(two(a), two(a >> 8), two(b), two(b >> 8));
                    } else {  // byte k of eight columns: columns 2k (low nibble) and 2k + 1
                        const __half2 bias = as_half2(0x64086408u);
                        const uint32_t lo = w[i + j] & 0x0F0F0F0Fu, hi = (w[i + j] >> 4) & 0x0F0F0F0Fu;
                        v[j] = make_uint4(as_u32(__hsub2(as_half2(biased_pair(lo, 0x4140u)), bias)), as_u32(__hsub2(as_half2(biased_pair(hi, 0x4140u)), bias)),
                                          as_u32(__hsub2(as_half2(biased_pair(lo, 0x4342u)), bias)), as_u32(__hsub2(as_half2(biased_pair(hi, 0x4342u)), bias)));
                    }
                }
                tmem_st8(to + 4 * i, v[0], v[1]);
            }
            close();
        };
        // Q4_K, Q5_K: sixteen bytes of the quants of a 64-column group give sixteen columns of its first and of its second sub-block
        [[maybe_unused]] auto group_q45 = [&](auto gc, const unsigned char *row, const uint4 &hdr, const ScalesMins &sm, const uint4 &qh) {
            constexpr uint32_t g = decltype(gc)::value, j0 = (2 * g) & 3u;
            constexpr float middle = FMT == kQ5K ? 16.f : 8.f;
            const uint32_t scw = g < 2 ? sm.sc_lo : sm.sc_hi;
            const __half2 sc0 = __hsub2(as_half2(biased_pair(scw, 0x4040u + j0 * 0x0101u)), k1024);
            const __half2 sc1 = __hsub2(as_half2(biased_pair(scw, 0x4040u + (j0 + 1) * 0x0101u)), k1024);
            // (1024 + 16·q)·(sc / 16) − (64 + middle)·sc = (q − middle)·sc, exact: 80·sc ≤ 5040 = 16·315, 72·sc ≤ 4536 = 8·567
            const __half2 k16th = __float2half2_rn(0.0625f), kbias = __float2half2_rn(-64.f - middle);
            const __half2 a0 = __hmul2(sc0, k16th), b0 = __hmul2(sc0, kbias), a1 = __hmul2(sc1, k16th), b1 = __hmul2(sc1, kbias);
            const uint4 ql = *reinterpret_cast<const uint4 *>(row + (FMT == kQ5K ? 48 : 16) + 32 * g + 16 * hf);
            if (!open()) return;
            const uint32_t q[4] = {ql.x, ql.y, ql.z, ql.w}, h[4] = {qh.x, qh.y, qh.z, qh.w};
            const uint32_t to = w_lanes + ring.s * T::kACols + hf * 8;
            // bytes (0, 2) and (1, 3) of a word: nibble to bits 4-7, fifth bit (bit J of its byte) to bit 8 of each half
            auto five = [&](uint32_t nib, uint32_t bit, const __half2 &a, const __half2 &b) {
                return as_u32(__hfma2(as_half2((nib & 0x00F000F0u) | (FMT == kQ5K ? bit & 0x01000100u : 0u) | 0x64006400u), a, b));
            };
            uint4 lo[2], hi[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                auto low = [&](uint32_t w, uint32_t x, bool odd) { return five(odd ? w >> 4 : w << 4, odd ? x >> (2 * g) : x << (8 - 2 * g), a0, b0); };
                auto high = [&](uint32_t w, uint32_t x, bool odd) { return five(odd ? w >> 8 : w, odd ? x >> (2 * g + 1) : x << (7 - 2 * g), a1, b1); };
                lo[e] = make_uint4(low(q[2 * e], h[2 * e], false), low(q[2 * e], h[2 * e], true), low(q[2 * e + 1], h[2 * e + 1], false), low(q[2 * e + 1], h[2 * e + 1], true));
                hi[e] = make_uint4(high(q[2 * e], h[2 * e], false), high(q[2 * e], h[2 * e], true), high(q[2 * e + 1], h[2 * e + 1], false), high(q[2 * e + 1], h[2 * e + 1], true));
            }
            tmem_st8(to, lo[0], lo[1]);
            tmem_st8(to + 16, hi[0], hi[1]);
            if constexpr (g == 3) {
                const float2 dd = __half22float2(as_half2(hdr.x));
                const float scale = offset_scale(offset_exponent(dd.x, dd.y));
                const float ds = middle * dd.x;
                uint32_t c[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    float v[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const uint32_t i = 2 * k + e, sh = 8 * (i & 3u);
                        const float sc = (float)(((i < 4 ? sm.sc_lo : sm.sc_hi) >> sh) & 63u), mn = (float)(((i < 4 ? sm.m_lo : sm.m_hi) >> sh) & 63u);
                        v[e] = (ds * sc - dd.y * mn) * scale;
                    }
                    const __half2 top = __floats2half2_rn(v[0], v[1]);
                    if (hf == 0) {
                        c[k] = as_u32(top);
                    } else {
                        const float2 back = __half22float2(top);
                        c[k] = as_u32(__floats2half2_rn(v[0] - back.x, v[1] - back.y));
                    }
                }
                unsigned char *slab = smem + T::kOffOffset + hf * 4096 + (r >> 3) * 128 + (r & 7u) * 16;
                *reinterpret_cast<uint4 *>(slab) = make_uint4(c[0], c[1], c[2], c[3]);
                *reinterpret_cast<uint4 *>(slab + 2048) = make_uint4(c[0], c[1], c[2], c[3]);
                fence_async_smem();  // generic-proxy stores → visible to the tensor core's reads
            }
            close();
        };
        // Q6_K: 32 columns of a stage from 32 bytes of nibbles (low ones in the first stage of a half super-block, high ones in the second)
        [[maybe_unused]] auto group_q6 = [&](auto gc, const uint4 (&ql)[2], const uint4 (&qh)[2], uint32_t scw) {
            constexpr uint32_t g = decltype(gc)::value;
            const uint32_t l[8] = {ql[0].x, ql[0].y, ql[0].z, ql[0].w, ql[1].x, ql[1].y, ql[1].z, ql[1].w};
            const uint32_t h[8] = {qh[0].x, qh[0].y, qh[0].z, qh[0].w, qh[1].x, qh[1].y, qh[1].z, qh[1].w};
            const uint32_t sh = 4 * (g & 1u) + 2 * hf;  // the bit pair's place
            if (!open()) return;
            const uint32_t to = w_lanes + ring.s * T::kACols + hf * 16;
#pragma unroll
            for (int e = 0; e < 2; e++) {  // sixteen columns with one scale
                const __half2 sc = __half2half2(__short2half_rn((short)(signed char)(scw >> (8 * e))));
                uint4 hi[2], lo[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int k = 4 * e + 2 * i;
                    auto two = [&](uint32_t q6, uint32_t &top, uint32_t &rest) {
                        const __half2 q = __hsub2(as_half2((q6 & 0x00FF00FFu) | 0x64006400u), as_half2(0x64206420u));  // 1056
                        const __half2 t = __hmul2(sc, q);
                        top = as_u32(t);
                        rest = as_u32(__hfma2(sc, q, __hneg2(t)));
                    };
                    const uint32_t v = ((l[k] >> (4 * (g & 1u))) & 0x0F0F0F0Fu) | (((h[k] >> sh) << 4) & 0x30303030u);
                    const uint32_t u = ((l[k + 1] >> (4 * (g & 1u))) & 0x0F0F0F0Fu) | (((h[k + 1] >> sh) << 4) & 0x30303030u);
                    two(v, hi[i].x, lo[i].x);
                    two(v >> 8, hi[i].y, lo[i].y);
                    two(u, hi[i].z, lo[i].z);
                    two(u >> 8, hi[i].w, lo[i].w);
                }
                tmem_st8(to + 8 * e, hi[0], hi[1]);
                tmem_st8(to + 32 + 8 * e, lo[0], lo[1]);
            }
            close();
        };
        UnitWalk walk(p, bpr);
        for (uint32_t u = 0; walk.live && ok; u++, walk.next(p, bpr)) {
            const uint32_t slot = u % T::kRaw, ph = (u / T::kRaw) & 1u;
            ok = mbar_wait(bar_raw_full + 8 * slot, ph, abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const unsigned char *box = raw + (size_t)slot * T::kRawBytes;
            if constexpr (T::BLOCK32) {
                const unsigned char *row = box + r * T::kRawRow;
                auto all = [&](auto hfc) {
                    mma_steps<0, 4>([&](auto gc) {
                        if (ok) block32(gc, hfc, row);
                    });
                };
                if (hf == 0) all(std::integral_constant<uint32_t, 0>{});
                else all(std::integral_constant<uint32_t, 1>{});
            } else if constexpr (T::OFFSET) {
                const unsigned char *row = box + r * T::kRawRow;
                const uint4 hdr = *reinterpret_cast<const uint4 *>(row), qh = FMT == kQ5K ? *reinterpret_cast<const uint4 *>(row + 16 + 16 * hf) : hdr;
                const ScalesMins sm = q4k_scales_mins(hdr.y, hdr.z, hdr.w);
                mma_steps<0, 4>([&](auto gc) {
                    if (ok) group_q45(gc, row, hdr, sm, qh);
                });
            } else {
                // ql: chunk c of row r lies at c ^ (r mod 8), qh: at c ^ (r / 2 mod 4); the scales of a row are sixteen bytes
                const unsigned char *qlp = box + r * 128, *qhp = box + kTileRows * 128 + r * 64, *scp = box + kTileRows * 192 + r * 16;
                mma_steps<0, 2>([&](auto hc) {
                    constexpr uint32_t half = decltype(hc)::value;  // 128 columns
                    uint4 ql[2], qh[2];
#pragma unroll
                    for (uint32_t i = 0; i < 2; i++) {
                        ql[i] = *reinterpret_cast<const uint4 *>(qlp + 16 * ((4 * half + 2 * hf + i) ^ (r & 7u)));
                        qh[i] = *reinterpret_cast<const uint4 *>(qhp + 16 * ((2 * half + i) ^ ((r >> 1) & 3u)));
                    }
                    const uint2 sc = *reinterpret_cast<const uint2 *>(scp + 8 * half);  // two scales per 32 columns
                    const uint32_t s0 = sc.x >> (16 * hf), s1 = sc.y >> (16 * hf);
                    if (ok) group_q6(std::integral_constant<uint32_t, 2 * half>{}, ql, qh, s0);
                    if (ok) group_q6(std::integral_constant<uint32_t, 2 * half + 1>{}, ql, qh, s1);
                });
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_raw_empty + 8 * slot);  // this warp is done with the box
        }
    } else {
        move_registers<true, Registers<T::BLOCK32 && !T::MERGED>::kDrain, kLaunchRegs>();
        // drain warp: TMEM lanes [32·(warp % 4), +32) = rows of the tile, columns [CW·(warp / 4), +CW)
        yule_pdl_wait();
        const uint32_t lane_base = (warp & 3u) * 32u, col_base = (warp >> 2) * CW;
        RingPos ring;
        bool ok = true;
        [[maybe_unused]] uint32_t n_stage = 0;
        ItemWalk items(p);
            for (Item wi; ok && items.next(p, bpr, wi);) {
            const uint32_t row = wi.mt * kTileRows + lane_base + lane;
            const uint8_t *rowp = p.w[wi.seg] + (size_t)(row < p.n_rows[wi.seg] ? row : p.n_rows[wi.seg] - 1) * p.w_row_bytes;
            // the scales of a super-block: Q4_K, Q5_K (d, dmin) at its start, Q6_K d in the last plane of the row
            auto scale_at = [&](uint32_t sb) -> uint32_t {
                if constexpr (T::OFFSET) return __ldg(reinterpret_cast<const uint32_t *>(rowp + (size_t)sb * T::kRawRow));
                else if constexpr (FMT == kQ6K) return __ldg(reinterpret_cast<const unsigned short *>(rowp + (size_t)bpr * 208) + sb);
                else return 0;
            };
            // Sums in fp32, pairs of columns 2j, 2j + 1.  What rounds is the addition to a long sum, so sums are kept in levels: up to 64 activation
            // rows, where registers allow it, a super-block, five of those, and all; at 128 rows sixteen super-blocks, which are then
            // added to the CTA's block of the work area (64 KB) in L2, without waiting for it.  (Loaded, added and stored here they cost 4 % in time spent on the loop alone, 7 %
            // with the waiting: 28672x4096 by 2048 rows 1036 -> 988 us, 8192x8192 by 2016 631 -> 604, under the power cap.)  A chain over all of 14336 columns has an
            // error of 3.6e-7 with an addition per 32 columns and 2.9e-7 with one per 64.
            constexpr uint32_t kLevel = T::MERGED ? 5 : 16;
            uint64_t sums[T::MERGED ? 3 : T::BLOCK32 ? 2 : 1][CW / 2];
            auto clear = [&](int k) {
#pragma unroll
                for (uint32_t j = 0; j < CW / 2; j++) sums[k][j] = 0;
            };
            [[maybe_unused]] auto add_up = [&](int to, int from) {
#pragma unroll
                for (uint32_t j = 0; j < CW / 2; j++) sums[to][j] = add2(sums[to][j], sums[from][j]);
            };
            // (this CTA's block of the work area, four columns of a row together)
            [[maybe_unused]] auto kept = [&] { return reinterpret_cast<float4 *>(part_block(p, 2 * kGemmMaxCtas + blockIdx.x, BN)) + (size_t)warp * (CW / 4) * 32 + lane; };
            [[maybe_unused]] auto add_kept = [&] {
                const float4 *from = kept();
#pragma unroll
                for (uint32_t j = 0; j < CW / 2; j += 2) {
                    const float4 v = __ldcg(from + j / 2 * 32);
                    sums[0][j] = add2(sums[0][j], pair(v.x, v.y));
                    sums[0][j + 1] = add2(sums[0][j + 1], pair(v.z, v.w));
                }
            };
            clear(0);
            uint32_t dd_cur = 0, dd_next = scale_at(wi.sb0);
            // The accumulator at the head of the ring: wait for it, read it, give it back; what(j, two of its sums, factor twice) for its columns.
            // hi | lo products lie side by side up to 64 rows, except in the offset.
            auto drain = [&](auto sidesc, auto chunkc, auto factor, auto what) {
                constexpr bool sides = T::MERGED && decltype(sidesc)::value;
                constexpr uint32_t CH = decltype(chunkc)::value;
                ok = mbar_wait(bar_acc_full + 8 * ring.s, ring.ph, abort_flag, p.status);
                ok = __all_sync(0xffffffffu, ok);  // (a warp stays together: its loads are the warp's)
                if (!ok) return;
                tc_fence_after();
                const uint32_t at = tmem_base + (lane_base << 16) + ring.s * T::kMainCols + col_base;
                const float f = factor();  // (where it comes from shared memory: there since the accumulator is full, until that is given back)
                const uint64_t f2 = pair(f, f);
#pragma unroll
                for (uint32_t c0 = 0; c0 < CW; c0 += CH) {
                    uint32_t v[CH], vl[sides ? CH : 1];
                    if constexpr (CH >= 32) {
#pragma unroll
                        for (uint32_t c1 = 0; c1 < CH; c1 += 32) tmem_ld32_issue(at + c0 + c1, v + c1);
                    } else {
                        tmem_ld16_issue(at + c0, v);
                    }
                    if constexpr (sides) tmem_ld16_issue(at + BN + c0, vl);
                    tmem_ld_wait();
                    if (c0 + CH == CW) {  // the accumulator goes back before the arithmetic on what was read last
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_acc_empty + 8 * ring.s);
                        ring.advance(NBUF);
                    }
#pragma unroll
                    for (uint32_t j = 0; j < CH; j += 2) {
                        uint64_t t = pair_bits(v[j], v[j + 1]);
                        if constexpr (sides) t = add2(t, pair_bits(vl[j], vl[j + 1]));
                        what((c0 + j) / 2, t, f2);
                    }
                }
            };
            constexpr std::true_type sides{};
            constexpr std::integral_constant<uint32_t, T::MERGED ? 16 : 32> chunk{};
            constexpr int in = T::MERGED ? 2 : 0;
            auto into = [&](uint32_t j, uint64_t t, uint64_t f2) { sums[in][j] = fma2(f2, t, sums[in][j]); };
            for (uint32_t sb = wi.sb0; sb < wi.sb1 && ok; sb++) {
                const uint32_t nth = (sb - wi.sb0) % kLevel;
                if constexpr (T::MERGED) {
                    clear(2);
                    if (nth == 0) clear(1);
                } else if (nth == 0 && sb != wi.sb0) {
                    float4 *to = kept();
                    const bool first = sb == wi.sb0 + kLevel;
#pragma unroll
                    for (uint32_t j = 0; j < CW / 2; j += 2) {
                        const float2 a = unpair(sums[0][j]), b = unpair(sums[0][j + 1]);
                        if (first) __stcg(to + j / 2 * 32, make_float4(a.x, a.y, b.x, b.y));
                        else asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to + j / 2 * 32), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y) : "memory");
                    }
                    clear(0);
                }
                if constexpr (T::BLOCK32) {
#pragma unroll 1
                    for (uint32_t g = 0; g < 4 && ok; g++, n_stage++) {
                        const float *sc = scales + (n_stage % kScaleRing) * 2 * kTileRows + lane_base + lane;
                        if constexpr (T::MERGED) {
                            drain(sides, chunk, [&] { return sc[0]; }, into);
                            if (ok) drain(sides, chunk, [&] { return sc[kTileRows]; }, into);
                        } else {
                            constexpr std::integral_constant<uint32_t, CW> whole{};
                            drain(sides, whole, [&] { return sc[0]; }, [&](uint32_t j, uint64_t t, uint64_t f2) { sums[1][j] = mul2(f2, t); });
                            if (ok) drain(sides, chunk, [&] { return sc[kTileRows]; }, [&](uint32_t j, uint64_t t, uint64_t f2) { sums[0][j] = add2(sums[0][j], fma2(f2, t, sums[1][j])); });
                        }
                    }
                } else {
                    dd_cur = dd_next;  // take the super-block's scales, ask for the next one's
                    if (sb + 1 < wi.sb1) dd_next = scale_at(sb + 1);
                    const float2 dd = __half22float2(as_half2(dd_cur));
#pragma unroll 1
                    for (uint32_t g = 0; g < 4 / T::kSpan && ok; g++) drain(sides, chunk, [&] { return dd.x; }, into);
                    if (T::OFFSET && ok) drain(std::false_type{}, chunk, [&] { return offset_unscale(offset_exponent(dd.x, dd.y)) * (1.0f / kSumScale); }, into);
                }
                if constexpr (T::MERGED) {
                    add_up(1, 2);
                    if (nth == kLevel - 1 || sb + 1 == wi.sb1) add_up(0, 1);
                }
            }
            if (!T::MERGED && ok && wi.sb1 - wi.sb0 > kLevel) add_kept();
            if (!ok) break;
            float acc[CW];
#pragma unroll
            for (uint32_t j = 0; j < CW; j += 2) {
                const float2 a = unpair(sums[0][j / 2]);
                acc[j] = a.x;
                acc[j + 1] = a.y;
            }
            finish_item<BN, CW>(p, wi, bpr, warp, lane, lane_base, col_base, acc);
        }
    }

    // common exit: nothing of this CTA may still be in flight when its TMEM and shared memory go
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (*abort_flag) {
        // gave up: let copies and MMAs that were already issued drain before the resources are freed
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int FMT, int BN>
cudaError_t launch_int(const GemmParams &p, const IntMaps &maps, uint32_t grid, bool pdl, cudaStream_t s) {
    auto kern = qgemm_int_kernel<FMT, BN>;
    static bool attr_done[64] = {};  // the opt-in for large dynamic shared memory belongs to the device
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !attr_done[dev]) {
            cudaFuncAttributes fa;  // the split of the registers counts on what the launch brings: a library that was not built by build.py must not hang
            e = cudaFuncGetAttributes(&fa, kern);
            if (e == cudaSuccess && fa.numRegs < kLaunchRegs) e = cudaErrorInvalidValue;
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    return launch_kernel(kern, dim3(grid), dim3(kThreads), Tile<FMT, BN>::kSmem, s, pdl, p, maps);
}

template <int FMT>
cudaError_t launch_bn(const GemmParams &p, const IntMaps &maps, uint32_t grid, bool pdl, cudaStream_t s) {
    return p.bn == 32 ? launch_int<FMT, 32>(p, maps, grid, pdl, s) : p.bn == 64 ? launch_int<FMT, 64>(p, maps, grid, pdl, s) : launch_int<FMT, 128>(p, maps, grid, pdl, s);
}

}  // namespace

// Every matrix of the launch: Q8_0, Q4_0, Q5_K and Q4_K rows on 16-byte boundaries (their super-blocks are multiples of 16 bytes), Q6_K with its planar copy.  Up to
// 64 activation rows Q4_K stays in qgemm_tc.cu, whose stages of two column groups at 32 rows have fewer hand-offs (8192x28672 by 32 rows 71 us).
bool qgemm_int_supported(const QGemm &g) {
    if (g.type == YULE_DTYPE_Q6_K) {
        if (!g.planar) return false;
        for (uint32_t i = 0; i < g.n_more; i++)
            if (!g.planar_more[i]) return false;
        return true;
    }
    if (g.type != YULE_DTYPE_Q8_0 && g.type != YULE_DTYPE_Q4_0 && g.type != YULE_DTYPE_Q5_K && (g.type != YULE_DTYPE_Q4_K || g.n_tokens <= 64)) return false;
    uintptr_t all = reinterpret_cast<uintptr_t>(g.w);
    for (uint32_t i = 0; i < g.n_more; i++) all |= reinterpret_cast<uintptr_t>(g.w_more[i]);
    return (all & 15) == 0;
}

// `p` as launch_qgemm_mm (qgemm_tc.cu) has filled it in for any format
cudaError_t launch_qgemm_int(const QGemm &g, const void *params, uint32_t grid, cudaStream_t s) {
    GemmParams p = *static_cast<const GemmParams *>(params);
    IntMaps maps;
    memset(&maps, 0, sizeof(maps));
    const uint32_t bpr = g.n_cols / 256;
    for (uint32_t i = 0; i < p.n_seg; i++) {
        cudaError_t e;
        if (g.type == YULE_DTYPE_Q6_K) {
            const uint8_t *w = p.w[i] = i ? g.planar_more[i - 1] : g.planar;
            p.w_row_bytes = q6k_planar_row_bytes(g.n_cols);
            e = cached_tensor_map_2d(w, 1, (uint64_t)bpr * 128, p.n_rows[i], p.w_row_bytes, 128, kTileRows, &maps.m[i][0], 128);
            if (e == cudaSuccess) e = cached_tensor_map_2d(w + (size_t)bpr * 128, 1, (uint64_t)bpr * 64, p.n_rows[i], p.w_row_bytes, 64, kTileRows, &maps.m[i][1], 64);
            if (e == cudaSuccess) e = cached_tensor_map_2d(w + (size_t)bpr * 192, 1, (uint64_t)bpr * 16, p.n_rows[i], p.w_row_bytes, 16, kTileRows, &maps.m[i][2]);
        } else {
            const uint32_t unit = g.type == YULE_DTYPE_Q8_0 ? 272 : g.type == YULE_DTYPE_Q5_K ? 176 : 144;
            e = cached_tensor_map_2d(p.w[i], 8, (uint64_t)bpr * unit / 8, p.n_rows[i], (uint64_t)bpr * unit, unit / 8, kTileRows, &maps.m[i][0]);
        }
        if (e != cudaSuccess) return e;
    }
    // What the adder's truncation takes of a result on average, measured on products of either sign (bias against 64 bits); two additions a drain
    // cost less than four, and beside hi | lo as one operand less still.
    const bool merged = p.bn <= 64;
    p.truncation = g.type == YULE_DTYPE_Q6_K ? 0.82e-7f : g.type == YULE_DTYPE_Q4_K ? 0.8e-7f : g.type == YULE_DTYPE_Q5_K ? 0.56e-7f : merged ? 0.15e-7f : 0.45e-7f;
    switch (g.type) {
        case YULE_DTYPE_Q8_0: return launch_bn<kQ8>(p, maps, grid, g.pdl, s);
        case YULE_DTYPE_Q4_0: return launch_bn<kQ4>(p, maps, grid, g.pdl, s);
        case YULE_DTYPE_Q5_K: return launch_bn<kQ5K>(p, maps, grid, g.pdl, s);
        case YULE_DTYPE_Q4_K: return launch_int<kQ4K, 128>(p, maps, grid, g.pdl, s);
        default: return launch_bn<kQ6K>(p, maps, grid, g.pdl, s);
    }
}

}  // namespace yule
