// What the quantised GEMM kernels on tcgen05 (qgemm_tc.cu, qgemm_int.cu) have in common: barriers, tensor-memory and MMA instructions, the
// numbering of work items and the end of an item.
#pragma once

#include <type_traits>

#include <cuda_fp16.h>

#include "internal.h"

namespace yule {
namespace {

constexpr int kTileRows = 128;  // rows of W per tile = TMEM lanes
constexpr int kEpiWarps = 8;    // drain warps
constexpr float kSumScale = 1.0f / 32.0f;     // the sub-block sums of x are stored divided by 32
constexpr long long kWaitCycles = 2000000000LL;  // ~1 s: far beyond any real stall

constexpr int kGemmSegs = 3;  // matrices that share their activation tiles (Q/K/V; gate/up) in one launch
struct GemmParams {
    const uint8_t *w[kGemmSegs];  // blocks, row-major, per matrix
    const __half *xb;      // activation tiles written by gemm_xprep_kernel
    const float *oscale;   // per (padded) activation row: 1 / row scale
    float *out[kGemmSegs]; // [n_tokens][out_stride] per matrix
    const float *residual; // added to the results of matrix 0 (same layout; single-matrix launches only) or null
    uint32_t n_rows[kGemmSegs], out_stride[kGemmSegs];
    uint32_t mt0[kGemmSegs + 1];  // first row tile of each matrix in the launch's numbering; [n_seg] = n_mtiles
    uint32_t n_seg;
    uint32_t n_cols, n_tokens;
    uint32_t bn;           // activation rows per tile: 32, 64 or 128
    uint32_t n_mtiles, n_ntiles;
    // The first split_tiles tiles are dealt by super-blocks: their split_units = split_tiles · n_cols / 256 in equal runs to split_ctas CTAs; whole
    // tiles follow, one per CTA and round.
    uint32_t split_tiles, split_ctas, split_units;
    uint64_t by_ctas, by_units, by_bpr, by_ntiles;  // what divides by split_ctas, split_units, n_cols / 256 and n_ntiles (see quotient)
    float *split_part;        // blocks of [bn][128] partial results: two per CTA (its runs touch at most two tiles), then one per CTA
    uint32_t *split_tickets;  // per (split tile, drain warp) the number of its parts that are stored; left at zero
    uint32_t type;         // GGUF type id of the weights (generic kernel)
    uint64_t w_row_bytes;  // bytes of one row of the weight tensor
    uint32_t unit_bytes;   // generic kernel: bytes of 256 columns of one row
    uint32_t raw_stride;   // generic kernel: shared-memory row stride of the raw copy (an odd multiple of 16 bytes)
    uint32_t raw_chunks;   // generic kernel: 16-byte chunks copied per row and unit
    uint32_t raw_ring_bytes;  // generic kernel: two slots of 128 rows
    float truncation;      // what the adder of the tensor core takes of a result on average, as a fraction: given back at the end
    float out_scale;       // a power of two: 1; generic kernel: 1 / kGenericWScale
    int *status;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
constexpr uint32_t kSuspendNs = 20000;  // a waiting warp sleeps up to this long instead of spending issue slots on polls
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "n"(kSuspendNs)
        : "memory");
    return ok != 0;
}
// Bounded wait.  False: the CTA is giving up (this thread ran out of time, or another did).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 1;; it++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 255u) == 0u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > kWaitCycles) {
                *abort_flag = 1;
                atomicExch(status, kStatusGemmTimeout);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory operand descriptor, K-major, no swizzle: lbo = bytes between the two core
// matrices of a 16-column step, sbo = bytes between 8-row groups.  Bit 46 is the descriptor
// version of this architecture.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

// True in one lane of the warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(one)::"memory");
    return one != 0;
}

// D[tmem] (+)= A[smem] · B[smem], fp16 operands, fp32 accumulate, one CTA.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Both from shared memory, descriptors as their words (the upper one is the same for all steps of an operand), the accumulate flag known at compile time.
template <int ACC>
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "n"(ACC)
        : "memory");
}
// A from tensor memory (lane = row, a column two fp16 values), the accumulate flag known at compile time.
template <int ACC>
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "n"(ACC)
        : "memory");
}
// 4 or 8 words per lane into as many columns of the warp's 32 lanes; in tensor memory after tmem_st_wait().
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint4 &v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4 &a, const uint4 &b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The mbarrier gets one arrival when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// The same load without the wait: the registers hold the values only after tmem_ld_wait().
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Two fp32 operations per instruction, each rounded as the single one is.  The drain's arithmetic and the unpacking share the issue
// slots of an SM with everything else; a stage has to get by with fewer of them than its MMAs take clocks.
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t pair_bits(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The eight 6-bit scales and mins of a super-block from its 12 packed bytes
// (yule-core/src/dequant.rs:165-176), four per word, one byte each.
struct ScalesMins {
    uint32_t sc_lo, sc_hi, m_lo, m_hi;  // sub-blocks 0-3 and 4-7
};
__device__ __forceinline__ ScalesMins q4k_scales_mins(uint32_t s0, uint32_t s1, uint32_t s2) {
    ScalesMins r;
    r.sc_lo = s0 & 0x3F3F3F3Fu;
    r.m_lo = s1 & 0x3F3F3F3Fu;
    r.sc_hi = (s2 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u);
    r.m_hi = ((s2 >> 4) & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u);
    return r;
}
// fp16 pair (1024 + a, 1024 + b) from two bytes: 0x6400 | v is the half 1024 + v for v < 1024
__device__ __forceinline__ uint32_t biased_pair(uint32_t word, uint32_t selector) { return __byte_perm(word, 0x64646464u, selector); }
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }

// f(integral_constant<uint32_t, K>) for K in [K0, K1)
template <uint32_t K0, uint32_t K1, class F>
__device__ __forceinline__ void mma_steps(F f) {
    if constexpr (K0 < K1) {
        f(std::integral_constant<uint32_t, K0>{});
        mma_steps<K0 + 1, K1>(f);
    }
}

// Registers move between the warpgroups of a CTA whose launch brought LAUNCH per thread.  Called by every warp of a warpgroup.
template <bool ON, int REGS, int LAUNCH>
__device__ __forceinline__ void move_registers() {
    if constexpr (ON) {
        if constexpr (REGS > LAUNCH) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS));
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS));
    }
}

// Position in the stage ring without a runtime division (an integer division runs on the same
// slow pipe as the half conversions): slot and phase parity, advanced once per stage.
struct RingPos {
    uint32_t s = 0, ph = 0;
    __device__ __forceinline__ void advance(uint32_t stages) {
        if (++s == stages) {
            s = 0;
            ph ^= 1u;
        }
    }
};

// n / d for any 32-bit n, with by = divide_by(d): ceil(2^64 / d), which is too large by less than 2^-32 of it, so that what n times it has too much never reaches
// the next whole number; 0 stands for d = 1.  (A division by a number that is not known takes some hundred clocks, and an item has seven, some of them one after the other and
// between its last sums and their stores: 1024x4096 by 65 rows 16.5 us with multiplications, 17.1 with divisions.)
inline uint64_t divide_by(uint32_t d) { return d > 1 ? ~0ull / d + 1 : 0ull; }
__device__ __forceinline__ uint32_t quotient(uint32_t n, uint64_t by) { return by ? (uint32_t)__umul64hi(by, n) : n; }

// A work item: tile (row tile x activation tile) and the range of super-blocks [sb0, sb1) of its columns.
struct Item {
    uint32_t tile, mt, nt, sb0, sb1, seg;  // mt: row tile inside matrix `seg`
    uint32_t part;                         // which of this CTA's runs, where the tile is split
};
// This CTA's work items, in the order in which every role goes through them: its run of the split tiles' super-blocks, which covers a part of one
// tile or of two, then whole tiles.  (Dealing whole tiles alone leaves the last round as empty as it comes: 448 tiles of a 70B gate / up
// on 148 SMs are four rounds for 3.03 of work, 112 tiles of a 1.1B down projection one for 0.76.  The parts first, so that adding them up
// runs under the tiles that follow.)
// (Selects instead of branches, and nothing that hides from the compiler that all threads have the same item: ring positions and tensor-memory addresses
// depend on how often loops run, and have to be uniform registers; and with branches the callers' loops came out three times over. Either
// made the GEMM a tenth to a quarter slower.)
struct ItemWalk {
    uint32_t step;
    __device__ __forceinline__ explicit ItemWalk(const GemmParams &p) : step((uint32_t)(blockIdx.x >= p.split_ctas) << 1) {}
    __device__ __forceinline__ bool next(const GemmParams &p, uint32_t bpr, Item &r) {
        const uint32_t lo = quotient(blockIdx.x * p.split_units, p.by_ctas), hi = quotient((blockIdx.x + 1) * p.split_units, p.by_ctas);  // this CTA's run
        const uint32_t first = quotient(lo, p.by_bpr), mid = (first + 1) * bpr;                                                       // and where its first tile ends
        const bool run = step < 2, second = step == 1;
        r.tile = run ? first + step : p.split_tiles + (step - 2) * gridDim.x + blockIdx.x;
        r.sb0 = run && !second ? lo + bpr - mid : 0;
        r.sb1 = !run ? bpr : second ? hi - mid : (hi < mid ? hi : mid) + bpr - mid;
        r.part = run ? step : 0;
        step = run && hi <= mid ? 2 : step + 1;
        r.mt = quotient(r.tile, p.by_ntiles);
        r.nt = r.tile - r.mt * p.n_ntiles;
        r.seg = 0;
        while (r.seg + 1 < p.n_seg && r.mt >= p.mt0[r.seg + 1]) r.seg++;
        r.mt -= p.mt0[r.seg];
        return r.tile < p.n_mtiles * p.n_ntiles;
    }
};
// The (work item, super-block) pairs of this CTA in the order every role goes through them.
struct UnitWalk {
    ItemWalk items;
    Item it;
    uint32_t sb;
    bool live;
    __device__ __forceinline__ UnitWalk(const GemmParams &p, uint32_t bpr) : items(p) { load(p, bpr); }
    __device__ __forceinline__ void load(const GemmParams &p, uint32_t bpr) {
        live = items.next(p, bpr, it);
        sb = it.sb0;
    }
    __device__ __forceinline__ void next(const GemmParams &p, uint32_t bpr) {
        if (++sb == it.sb1) load(p, bpr);
    }
};
// The block of the work area for an item's partial sums, and one that is no other item's while a whole tile is at work.
__device__ __forceinline__ float *part_block(const GemmParams &p, uint32_t index, uint32_t bn) { return p.split_part + (size_t)index * (bn * kTileRows); }
__device__ __forceinline__ uint32_t own_part(const Item &wi) { return 2 * blockIdx.x + wi.part; }

// The end of a work item for one drain warp: its scaled sums to the output, or, where the columns of a tile are split, to the work area.
// acc[j] is row lane_base + lane, column col_base + j of the tile.
template <int BN, uint32_t CW>
__device__ __forceinline__ void finish_item(const GemmParams &p, const Item &wi, uint32_t bpr, uint32_t warp, uint32_t lane, uint32_t lane_base, uint32_t col_base,
                                            float (&acc)[CW]) {
    const uint32_t row = wi.mt * kTileRows + lane_base + lane;
    const uint32_t n0 = wi.nt * BN + col_base;
    // Four residuals are asked for before the first of their stores (which may be to the same matrix, so nothing but
    // this order lets them overlap): one by one they took 24 us per tile, so they take 7.
    auto store = [&](auto scaledc) {
        constexpr bool scaled = decltype(scaledc)::value;
#pragma unroll
        for (uint32_t c0 = 0; c0 < CW; c0 += 16) {
            const float osc = !scaled && lane < 16 ? p.oscale[n0 + c0 + lane] : 0.f;  // padded to whole tiles
            if constexpr (!scaled) {  // (not one by one between the stores, each of which is conditional: 1024x1024 by 65 rows 12.2 us, 13.9 so)
#pragma unroll
                for (uint32_t j = 0; j < 16; j++) acc[c0 + j] = fmaf(acc[c0 + j], p.truncation, acc[c0 + j]) * __shfl_sync(0xffffffffu, osc, j) * p.out_scale;
            }
#pragma unroll
            for (uint32_t j0 = 0; j0 < 16; j0 += 4) {
                const size_t o0 = (size_t)(n0 + c0 + j0) * p.out_stride[wi.seg] + row;
                const uint32_t live = row < p.n_rows[wi.seg] && n0 + c0 + j0 < p.n_tokens ? p.n_tokens - (n0 + c0 + j0) : 0u;
                float res[4];
                if (p.residual) {
#pragma unroll
                    for (uint32_t j = 0; j < 4; j++) res[j] = j < live ? p.residual[o0 + j * p.out_stride[wi.seg]] : 0.f;
                }
#pragma unroll
                for (uint32_t j = 0; j < 4; j++)
                    if (j < live) p.out[wi.seg][o0 + j * p.out_stride[wi.seg]] = p.residual ? acc[c0 + j0 + j] + res[j] : acc[c0 + j0 + j];
            }
        }
    };
    if (wi.sb1 - wi.sb0 < bpr) {
        // This item covers a part of the columns.  Every drain warp stores its block of scaled partial sums, then
        // takes a ticket of its (tile, warp); the warp that finds all the other parts stored adds them in the
        // order of the parts (its own included, so the sum does not depend on who came last) and writes the result.
        const size_t in_block = (size_t)col_base * kTileRows + lane_base + lane;
        float *mine = part_block(p, own_part(wi), BN) + in_block;
#pragma unroll
        for (uint32_t c0 = 0; c0 < CW; c0 += 16) {
            const float osc = lane < 16 ? p.oscale[n0 + c0 + lane] : 0.f;
#pragma unroll
            for (uint32_t j = 0; j < 16; j++)
                __stcg(mine + (size_t)(c0 + j) * kTileRows, fmaf(acc[c0 + j], p.truncation, acc[c0 + j]) * __shfl_sync(0xffffffffu, osc, j) * p.out_scale);
        }
        __syncwarp();
        // the CTAs whose runs hold the tile's first and its last super-block; the first of them may have begun with the tile before
        const uint32_t u0 = wi.tile * bpr;
        const uint32_t cta0 = quotient((u0 + 1) * p.split_ctas - 1, p.by_units), n_parts = quotient((u0 + bpr) * p.split_ctas - 1, p.by_units) - cta0 + 1;
        uint32_t ticket = 0;
        uint32_t *tk = p.split_tickets + (size_t)wi.tile * kEpiWarps + warp;
        if (lane == 0) {
            // (release: the stores of the warp, which it has met; acquire: those of the warps that took theirs before)
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(ticket) : "l"(tk) : "memory");
            if (ticket == n_parts - 1) *tk = 0;  // left at zero for the next launch
        }
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket != n_parts - 1) return;
        __syncwarp();
        const uint32_t first = 2 * cta0 + (quotient(cta0 * p.split_units, p.by_ctas) < u0 ? 1u : 0u);
#pragma unroll
        for (uint32_t j = 0; j < CW; j++) acc[j] = 0.f;
        // the loads of up to KS parts are in flight together; the additions keep the order of the parts
        constexpr uint32_t KS = CW <= 16 ? 4 : (CW <= 32 ? 2 : 1);
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < n_parts; k0 += KS) {
            float v[KS][CW];
#pragma unroll
            for (uint32_t q = 0; q < KS; q++) {
                const uint32_t k = k0 + q;
                const float *from = part_block(p, k == 0 ? first : 2 * (cta0 + k), BN) + in_block;
#pragma unroll
                for (uint32_t j = 0; j < CW; j++) v[q][j] = k < n_parts ? __ldcg(from + (size_t)j * kTileRows) : 0.f;
            }
#pragma unroll
            for (uint32_t q = 0; q < KS; q++)
#pragma unroll
                for (uint32_t j = 0; j < CW; j++) acc[j] += v[q][j];
        }
        store(std::true_type{});  // the parts were scaled
        return;
    }
    store(std::false_type{});
}

}  // namespace
}  // namespace yule
