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
    uint32_t ksplit, sb_per;  // split of the columns: `ksplit` work items per tile, `sb_per` super-blocks each (the last may be shorter)
    float *split_part;        // ksplit > 1: per work item a [bn][128] block of partial results
    uint32_t *split_tickets;  // ksplit > 1: per (tile, drain warp) the number of items that have stored theirs; left at zero
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

// A work item: tile (row tile x activation tile) and the range of super-blocks [sb0, sb1) of its columns.
struct Item {
    uint32_t tile, ks, mt, nt, sb0, sb1, seg;  // mt: row tile inside matrix `seg`
};
__device__ __forceinline__ Item decode_item(const GemmParams &p, uint32_t item, uint32_t bpr) {
    Item r;
    r.tile = item / p.ksplit;
    r.ks = item - r.tile * p.ksplit;
    r.mt = r.tile / p.n_ntiles;
    r.nt = r.tile - r.mt * p.n_ntiles;
    r.seg = 0;
    while (r.seg + 1 < p.n_seg && r.mt >= p.mt0[r.seg + 1]) r.seg++;
    r.mt -= p.mt0[r.seg];
    r.sb0 = r.ks * p.sb_per;
    r.sb1 = r.sb0 + p.sb_per < bpr ? r.sb0 + p.sb_per : bpr;
    return r;
}
// The (work item, super-block) pairs of this CTA in the order every role goes through them.
struct UnitWalk {
    uint32_t item, sb, sb1, mt, seg;
    bool live;
    __device__ __forceinline__ void load(const GemmParams &p, uint32_t n_items, uint32_t bpr) {
        live = item < n_items;
        if (live) {
            const Item it = decode_item(p, item, bpr);
            sb = it.sb0;
            sb1 = it.sb1;
            mt = it.mt;
            seg = it.seg;
        }
    }
    __device__ __forceinline__ void start(const GemmParams &p, uint32_t n_items, uint32_t bpr) {
        item = blockIdx.x;
        load(p, n_items, bpr);
    }
    __device__ __forceinline__ void next(const GemmParams &p, uint32_t n_items, uint32_t bpr) {
        if (++sb == sb1) {
            item += gridDim.x;
            load(p, n_items, bpr);
        }
    }
};

// The end of a work item for one drain warp: its scaled sums to the output, or, where the columns of a tile are split, to the work area.
// acc[j] is row lane_base + lane, column col_base + j of the tile.
template <int BN, uint32_t CW>
__device__ __forceinline__ void finish_item(const GemmParams &p, const Item &wi, uint32_t item, uint32_t warp, uint32_t lane, uint32_t lane_base, uint32_t col_base,
                                            float (&acc)[CW]) {
    const uint32_t row = wi.mt * kTileRows + lane_base + lane;
    const uint32_t n0 = wi.nt * BN + col_base;
    if (p.ksplit > 1) {
        // This item covers a part of the columns.  Every drain warp stores its block of scaled partial sums, then
        // takes a ticket of its (tile, warp); the warp that finds all the other parts stored adds them in the
        // order of the parts (its own included, so the sum does not depend on who came last) and writes the result.
        float *mine = p.split_part + (size_t)item * (BN * kTileRows) + lane_base + lane;
#pragma unroll
        for (uint32_t c0 = 0; c0 < CW; c0 += 16) {
            const float osc = lane < 16 ? p.oscale[n0 + c0 + lane] : 0.f;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float sc = __shfl_sync(0xffffffffu, osc, j);
                __stcg(mine + (size_t)(col_base + c0 + j) * kTileRows, fmaf(acc[c0 + j], p.truncation, acc[c0 + j]) * sc * p.out_scale);
            }
        }
        __threadfence();
        __syncwarp();
        uint32_t ticket = 0;
        uint32_t *tk = p.split_tickets + (size_t)wi.tile * kEpiWarps + warp;
        if (lane == 0) {
            ticket = atomicAdd(tk, 1u);
            if (ticket == p.ksplit - 1) *tk = 0;  // left at zero for the next launch
        }
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket != p.ksplit - 1) return;
        __threadfence();
        const float *parts = p.split_part + (size_t)(wi.tile * p.ksplit) * (BN * kTileRows) + (size_t)col_base * kTileRows + lane_base + lane;
#pragma unroll
        for (uint32_t j = 0; j < CW; j++) acc[j] = 0.f;
        // the loads of up to KS parts are in flight together; the additions keep the order of the parts
        constexpr uint32_t KS = CW <= 16 ? 4 : (CW <= 32 ? 2 : 1);
#pragma unroll 1
        for (uint32_t ks0 = 0; ks0 < p.ksplit; ks0 += KS, parts += KS * BN * kTileRows) {
            float v[KS][CW];
#pragma unroll
            for (uint32_t q = 0; q < KS; q++)
#pragma unroll
                for (uint32_t j = 0; j < CW; j++)
                    v[q][j] = ks0 + q < p.ksplit ? __ldcg(parts + (size_t)q * (BN * kTileRows) + (size_t)j * kTileRows) : 0.f;
#pragma unroll
            for (uint32_t q = 0; q < KS; q++)
#pragma unroll
                for (uint32_t j = 0; j < CW; j++) acc[j] += v[q][j];
        }
#pragma unroll
        for (uint32_t c0 = 0; c0 < CW; c0 += 4) {
            const size_t o0 = (size_t)(n0 + c0) * p.out_stride[wi.seg] + row;
            const uint32_t live = row < p.n_rows[wi.seg] && n0 + c0 < p.n_tokens ? p.n_tokens - (n0 + c0) : 0u;
            float res[4];
            if (p.residual) {
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) res[j] = j < live ? p.residual[o0 + j * p.out_stride[wi.seg]] : 0.f;
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; j++)
                if (j < live) p.out[wi.seg][o0 + j * p.out_stride[wi.seg]] = p.residual ? acc[c0 + j] + res[j] : acc[c0 + j];
        }
        return;
    }
#pragma unroll
    for (uint32_t c0 = 0; c0 < CW; c0 += 16) {
        const float osc = lane < 16 ? p.oscale[n0 + c0 + lane] : 0.f;  // padded to whole tiles
        // Four residuals are asked for before the first of their stores (which may be to the same matrix, so nothing but
        // this order lets them overlap): one by one they took 24 us per tile, so they take 7.
#pragma unroll
        for (int j0 = 0; j0 < 16; j0 += 4) {
            const size_t o0 = (size_t)(n0 + c0 + j0) * p.out_stride[wi.seg] + row;
            const uint32_t live = row < p.n_rows[wi.seg] && n0 + c0 + j0 < p.n_tokens ? p.n_tokens - (n0 + c0 + j0) : 0u;
            float res[4];
            if (p.residual) {
#pragma unroll
                for (uint32_t j = 0; j < 4; j++) res[j] = j < live ? p.residual[o0 + j * p.out_stride[wi.seg]] : 0.f;
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                const float val = fmaf(acc[c0 + j0 + j], p.truncation, acc[c0 + j0 + j]) * __shfl_sync(0xffffffffu, osc, j0 + j) * p.out_scale;
                if (j < live) p.out[wi.seg][o0 + j * p.out_stride[wi.seg]] = p.residual ? val + res[j] : val;
            }
        }
    }
}

}  // namespace
}  // namespace yule
