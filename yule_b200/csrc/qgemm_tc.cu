// Quantised GEMM on the 5th-generation tensor cores (tcgen05, accumulators in TMEM):
//
//     out[n][r] = Σ_k W[r][k] · x[n][k]        W: Q4_K blocks, x: 8 to 64 fp32 activation rows
//
// (With more rows Q4_K goes through qgemm_int.cu, and so do Q8_0, Q4_0, Q5_K and Q6_K at any number; the generic form of this kernel takes the other formats and what those kernels refuse.)
//
// This is the prefill / batched-decode counterpart of the matvec kernels: the weights cross HBM
// once per pass over up to 64 (generic: 128) activation rows instead of once per four.  The reference runs
// prefill as one matvec chain per token (yule-infer/src/gpu_runner.rs:146-160); the arithmetic
// contract is the same fp32 dot product.
//
// Operands.  A Q4_K weight is d·sc·q − dmin·m with a 4-bit q, 6-bit sc and m per 32 columns and
// fp16 d, dmin per 256.  The tensor core multiplies the exact integers: the W operand of a stage is
// sc·q (≤ 945, exact in fp16), the 64-column partial sums are drained from TMEM after every stage
// and multiplied by that row's d in fp32 on the way into register accumulators.  The min term is one
// more MMA per super-block, (m of the 8 sub-blocks) × (per-sub-block sums of x), drained with −dmin.
// Activations are fp32, which tcgen05 cannot take: each row is scaled by a power of two that puts
// its largest element in [2¹³, 2¹⁴) and split into fp16 hi + lo (22 significant bits); two MMAs per
// 16 columns, W·x_hi and W·x_lo (up to 64 activation rows one MMA against both terms side by side as
// one operand of twice the rows).  The tensor core adds into its fp32 accumulator with truncation, a
// bias that grows with the chain length; draining after every stage, and the small products before the
// large ones, keep a chain of large ones at 4 MMAs (8 at 32 rows) and leave the long sum to ordinary
// round-to-nearest fp32; the mean of the bias is given back at the end.  Error against 64 bits (2-norm),
// 2048 to 28672 columns: Q4_K by 24 rows 2.6e-7 to 3.2e-7, by 48 rows 2.3e-7 to 2.5e-7.
//
// Work items: (row tile, activation tile) pairs; those that do not fill a round of CTAs (all of them in small matrices, tensor-parallel
// shards, with few activation rows) are dealt by super-blocks (each in equal parts, or all in equal runs that may end inside a tile), ahead of the whole tiles, and the
// last drain warp of a (tile, warp) to finish adds up the scaled partial sums in the order of the parts.
//
// One CTA per SM, 20 warps, persistent over the work items:
//   warps 0-7   drain warps: tcgen05.ld of their 32 TMEM lanes × half of the columns after every
//               stage, FMA by d (and −dmin) into registers, two columns per instruction; at the end of a tile
//               scale, residual, store
//   warp  8     one thread: bulk copies (TMA engine) of the pre-arranged activation tiles
//   warps 9, 11 tcgen05.mma issue, even stages from one, odd stages from the other; warp 9 also owns
//               the TMEM allocation
//   warp  10    one thread: tiled TMA loads (cp.async.bulk.tensor.2d) of the raw Q4_K bytes, one
//               128-row × 144-byte box per super-block, six boxes in flight; rows past the end of the matrix arrive as zeros
//   warps 12-19 unpack Q4_K from that shared-memory copy → fp16 sc·q in tensor memory, where the MMA takes its
//               W operand from: a row is a lane, a column two weights, and 64 weights of a row are 32 columns
// A stage is a 128-row × 64-column slab of W plus the matching hi and lo slabs of x in shared memory; the last
// stage of a super-block also carries the 4 KB m slab (shared memory) and the sub-block sums of x.  At 32 activation rows
// a stage is two such column groups (a chain of eight MMAs and half the hand-offs per column).  Tensor memory holds
// four stages of W and behind them a ring of accumulators, three of 128 columns (four of 64 at 32 rows), in which the min term of a
// super-block takes its turn like a stage.
// One launch can run over up to three matrices that read the same activations (Q/K/V; gate/up): their row
// tiles are numbered one after the other.
// The activation operand is the no-swizzle K-major core-matrix layout: 8 rows × 16 bytes per core matrix,
// core matrices of one 8-column step contiguous along the rows.  Of eight columns the order is
// 0,2,1,3,4,6,5,7 (the order in which nibble pairs fall out of a 32-bit word) in both operands, so the products pair up correctly.
//
// What bounds it: the hand-offs of a stage between the roles, and issue slots; no role's work alone (measured with one taken out at a time).  32 rows, W in
// shared memory and in tensor memory: 8192x8192 32.6, 26.4 us (re-layout included); tiles that did not fill a round dealt by super-blocks: gate / up of the 70B shape 121, 103.
//
// Every wait is bounded: a pipeline that stops making progress sets the context's status word,
// raises the CTA's abort flag, lets all roles fall through to the common exit and frees its TMEM.

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <type_traits>
#include <unordered_map>

#include <cuda.h>
#include <cuda_fp16.h>

#include "dequant_device.cuh"
#include "internal.h"
#include "qgemm_common.cuh"

namespace yule {
namespace {

constexpr int kBM = 128;  // rows of W per tile = TMEM lanes
constexpr int kBK = 64;   // columns per stage (a quarter of a super-block)
constexpr int kProdWarps = 8;
constexpr int kLoaderWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1, kRawWarp = kEpiWarps + 2, kMmaWarp2 = kEpiWarps + 3,
              kFirstProdWarp = kEpiWarps + 4;
constexpr int kGemmThreads = (kEpiWarps + 4 + kProdWarps) * 32;  // 640
constexpr int kLaunchRegs = 96;  // registers per thread that 640 threads are launched with (the build checks that the 128-row kernels get them)
constexpr int kDrainRegs = 144, kControlRegs = 32, kProdRegs = 80;
static_assert(kEpiWarps * kDrainRegs + 4 * kControlRegs + kProdWarps * kProdRegs <= (kEpiWarps + 4 + kProdWarps) * kLaunchRegs, "register split");
constexpr uint32_t kStages = 4;  // of the operand ring: W in tensor memory, x in shared memory
// Super-blocks of raw Q4_K bytes in flight per CTA: what the activation stages leave room for.  (At 128 rows only the dequantising variant is built, whose ring
// is sized at launch and does not count in these.)
constexpr uint32_t kRawSlots = 6;
__host__ __device__ constexpr uint32_t raw_slots_for(uint32_t bn) { return bn >= 128 ? 3u : kRawSlots; }
// 64-column groups of W per stage.  The exact kernel at 32 activation rows takes two: its MMAs are narrow and its
// drains short, so the waits, fences and barrier arrivals of a stage, not its work, set the pace, and a stage of
// twice the columns halves them.  A chain is then eight MMAs (one per 16 columns against hi | lo), the same length as
// at 128 rows.
__host__ __device__ constexpr uint32_t groups_per_stage(uint32_t bn, bool generic) {
    return (!generic && bn <= 32) ? 2u : 1u;
}
constexpr uint32_t kRawBytes = kBM * 144;          // one super-block of 128 rows: 18 KB
// 2^-23: what truncation takes of a stage's sum on average (measured 0.9e-7 of the result, exact kernel 0.7e-7, at 32 rows
// 1.2e-7) is given back.
constexpr float kTruncation = 0.00000011920929f;
constexpr float kGenericWScale = 1024.f;      // generic kernel: weights are scaled by 2^10 before the fp16 hi/lo split
constexpr uint32_t kAmBytes = kBM * 16 * 2;  // the m slab of a super-block: 128 rows × 16 columns, 4 KB

struct GemmMaps {
    CUtensorMap m[kGemmSegs];  // exact kernel: tiled view of each weight matrix
};

// Eight consecutive weights (columns col0 .. col0+7 of a 256-column unit, col0 a multiple of 8) from a
// 2-byte-aligned copy of the unit's blocks, with the arithmetic of the per-element routines
// (dequant_device.cuh): one header decode per call instead of one per weight.
__device__ __forceinline__ void dequant8_unit(const unsigned char *unit, uint32_t type, uint32_t col0, float (&v)[8]) {
    auto u16_at = [&](uint32_t byte_off) { return (uint32_t) * reinterpret_cast<const unsigned short *>(unit + byte_off); };
    if (type == YULE_DTYPE_Q8_0) {
        const uint32_t b = (col0 >> 5) * 34, i0 = col0 & 31u;
        const float d = f16_bits_to_f32(u16_at(b));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t w = u16_at(b + 2 + i0 + 2 * k);
            v[2 * k] = __fmul_rn((float)(int)(signed char)(w & 0xFFu), d);
            v[2 * k + 1] = __fmul_rn((float)(int)(signed char)(w >> 8), d);
        }
    } else if (type == YULE_DTYPE_Q4_0) {
        const uint32_t b = (col0 >> 5) * 18, i0 = col0 & 31u;
        const float d = f16_bits_to_f32(u16_at(b));
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const uint32_t w = u16_at(b + 2 + i0 / 2 + 2 * k);  // two bytes = four weights: low nibble first
#pragma unroll
            for (int q = 0; q < 4; q++) v[4 * k + q] = __fmul_rn(__fsub_rn((float)((w >> (4 * q)) & 0xFu), 8.0f), d);
        }
    } else if (type == YULE_DTYPE_Q6_K) {
        const uint32_t h = col0 >> 7, r = col0 & 127u, g = r >> 5, l0 = r & 31u;
        const float d = f16_bits_to_f32(u16_at(208));
        const uint32_t scw = u16_at(192 + 8 * h + 2 * g);  // the two scales of this 32-column group
        const float ds = __fmul_rn(d, (float)(int)(signed char)((l0 >> 4) ? (scw >> 8) : (scw & 0xFFu)));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t ql = u16_at(64 * h + 32 * (g & 1u) + l0 + 2 * k) >> (4 * (g >> 1));
            const uint32_t qh = u16_at(128 + 32 * h + l0 + 2 * k) >> (2 * g);
            const int q0 = (int)((ql & 0xFu) | ((qh & 3u) << 4)) - 32;
            const int q1 = (int)(((ql >> 8) & 0xFu) | (((qh >> 8) & 3u) << 4)) - 32;
            v[2 * k] = __fmul_rn(ds, (float)q0);
            v[2 * k + 1] = __fmul_rn(ds, (float)q1);
        }
    } else if (type == YULE_DTYPE_Q5_K) {
        // dequant.rs:297-338: eight columns of sub-block s; nibbles of group s/2, fifth bits in bit s of qh
        const uint32_t s = col0 >> 5, l0 = col0 & 31u;
        uint32_t sc, mn;
        if (s < 4) {
            sc = unit[4 + s] & 63u;
            mn = unit[8 + s] & 63u;
        } else {
            sc = (unit[8 + s] & 0xFu) | ((unit[s] >> 6) << 4);
            mn = (unit[8 + s] >> 4) | ((unit[4 + s] >> 6) << 4);
        }
        const float ds = __fmul_rn(f16_bits_to_f32(u16_at(0)), (float)sc);
        const float dm = __fmul_rn(f16_bits_to_f32(u16_at(2)), (float)mn);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t ql = u16_at(48 + 32 * (s >> 1) + l0 + 2 * k) >> (4 * (s & 1u));
            const uint32_t qh = u16_at(16 + l0 + 2 * k) >> s;
            const uint32_t q0 = (ql & 0xFu) | ((qh & 1u) << 4), q1 = ((ql >> 8) & 0xFu) | (((qh >> 8) & 1u) << 4);
            v[2 * k] = __fsub_rn(__fmul_rn((float)q0, ds), dm);
            v[2 * k + 1] = __fsub_rn(__fmul_rn((float)q1, ds), dm);
        }
    } else if (type == YULE_DTYPE_Q2_K) {
        // dequant.rs:196-214: (d*scale)*q - dmin*min, sub-blocks of 16
        const uint32_t sm = unit[col0 >> 4];
        const float ds = __fmul_rn(f16_bits_to_f32(u16_at(80)), (float)(sm & 0xFu));
        const float dm = __fmul_rn(f16_bits_to_f32(u16_at(82)), (float)(sm >> 4));
        const uint32_t qs = u16_at(16 + (col0 >> 2));
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = __fsub_rn(__fmul_rn(ds, (float)((qs >> (2 * k)) & 3u)), dm);
    } else if (type == YULE_DTYPE_Q3_K) {
        // dequant.rs:219-251: 6-bit scale centred at 32, 3-bit weight centred at 4
        const uint32_t j = col0 >> 4;
        const uint32_t lo4 = j < 8 ? (unit[96 + j] & 0xFu) : (unit[88 + j] >> 4);
        const uint32_t hi2 = (unit[104 + (j >> 2)] >> (2 * (j & 3u))) & 3u;
        const float ds = __fmul_rn(f16_bits_to_f32(u16_at(108)), (float)((int)(lo4 | (hi2 << 4)) - 32));
        const uint32_t qs = u16_at(32 + (col0 >> 2)), hm = unit[col0 >> 3];
#pragma unroll
        for (int k = 0; k < 8; k++)
            v[k] = __fmul_rn(ds, (float)((int)(((qs >> (2 * k)) & 3u) | (((hm >> k) & 1u) << 2)) - 4));
    } else if (type == YULE_DTYPE_Q8_1) {
        const uint32_t b = (col0 >> 5) * 36, i0 = col0 & 31u;
        const float d = f16_bits_to_f32(u16_at(b));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t w = u16_at(b + 4 + i0 + 2 * k);
            v[2 * k] = __fmul_rn((float)(int)(signed char)(w & 0xFFu), d);
            v[2 * k + 1] = __fmul_rn((float)(int)(signed char)(w >> 8), d);
        }
    } else if (type == YULE_DTYPE_Q4_1 || type == YULE_DTYPE_Q5_0 || type == YULE_DTYPE_Q5_1) {
        // dequant.rs:91-138: optional minimum m after d, optional 32 fifth bits before the nibbles
        const bool has_m = type != YULE_DTYPE_Q5_0, has_qh = type != YULE_DTYPE_Q4_1;
        const uint32_t bb = type == YULE_DTYPE_Q4_1 ? 20u : type == YULE_DTYPE_Q5_0 ? 22u : 24u;
        const uint32_t b = (col0 >> 5) * bb, i0 = col0 & 31u;
        const uint32_t qh_off = has_m ? 4u : 2u, qs_off = qh_off + (has_qh ? 4u : 0u);
        const float d = f16_bits_to_f32(u16_at(b));
        const float m = has_m ? f16_bits_to_f32(u16_at(b + 2)) : 0.f;
        const uint32_t qh = has_qh ? unit[b + qh_off + (i0 >> 3)] : 0u;
        const uint32_t qs = u16_at(b + qs_off + (i0 >> 1)) | (u16_at(b + qs_off + (i0 >> 1) + 2) << 16);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float q = (float)(((qs >> (4 * k)) & 0xFu) | (((qh >> k) & 1u) << 4));
            v[k] = has_m ? __fadd_rn(__fmul_rn(q, d), m) : __fmul_rn(__fsub_rn(q, 16.0f), d);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = dequant_elem(unit, type, col0 + i);
    }
}

// Words of four bytes from a 2-byte-aligned shared-memory address (one word more is read than returned).
template <int N>
__device__ __forceinline__ void words_at(const unsigned char *p, uint32_t (&w)[N]) {
    const uint32_t mis = smem_u32(p) & 2u;
    const uint32_t *a = reinterpret_cast<const uint32_t *>(p - mis);
    uint32_t prev = a[0];
#pragma unroll
    for (int k = 0; k < N; k++) {
        const uint32_t next = a[k + 1];
        w[k] = __funnelshift_r(prev, next, 8 * mis);
        prev = next;
    }
}
// 32 consecutive weights of Q6_K (columns col0 .. col0 + 31 of a super-block) times 2^10 as fp16 hi + lo, eight columns at a time to
// put(i, hi, lo) in the order 0,2,1,3,4,6,5,7.  The same values as dequant8_unit and its split give, without conversion
// instructions: a quant is a half after one OR and one subtraction, 2^10·d·sc a pair of halves.  False: a scale that is not finite or too large;
// nothing was written.  2048x5632 against 777 rows: 275 us with dequant8_unit, 185 with this.  (A tensor with a row-planar copy goes to qgemm_int.cu.)
template <class Put>
__device__ __forceinline__ bool unpack32_q6k(const unsigned char *unit, uint32_t col0, bool live, Put put) {
    auto finite = [](__half2 d) { return __hle(__habs(__low2half(d)), __ushort_as_half(0x7BFF)); };  // false for infinities and NaN
    auto u16_at = [&](uint32_t off) { return *reinterpret_cast<const unsigned short *>(unit + off); };
    const uint32_t h = col0 >> 7, g = (col0 >> 5) & 3u;
    const float d = live ? f16_bits_to_f32(u16_at(208)) * kGenericWScale : 0.f;
    const uint32_t scw = u16_at(192 + 8 * h + 2 * g);  // the scales of the first and the last sixteen columns
    __half2 dh[2], dl[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float ds = d * (float)(int)(signed char)(scw >> (8 * k));
        dh[k] = __float2half2_rn(ds);
        dl[k] = __float2half2_rn(ds - __low2float(dh[k]));
    }
    if (!finite(dh[0]) || !finite(dh[1])) return false;
    uint32_t ql[8], qh[8];
    words_at(unit + 64 * h + 32 * (g & 1u), ql);
    words_at(unit + 128 + 32 * h, qh);
    const uint32_t sl = 4 * (g >> 1), sh = 2 * g;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        auto split = [&](uint32_t q6, uint32_t &hi, uint32_t &lo) {
            const __half2 q = __hsub2(as_half2((q6 & 0x00FF00FFu) | 0x64006400u), as_half2(0x64206420u));  // 1056
            const __half2 a = dh[i >> 1], b = dl[i >> 1], x = __hfma2(a, q, __hmul2(b, q));
            hi = as_u32(x);
            lo = as_u32(__hfma2(b, q, __hfma2(a, q, __hneg2(x))));
        };
        const uint32_t v = ((ql[2 * i] >> sl) & 0x0F0F0F0Fu) | (((qh[2 * i] >> sh) & 0x03030303u) << 4);
        const uint32_t u = ((ql[2 * i + 1] >> sl) & 0x0F0F0F0Fu) | (((qh[2 * i + 1] >> sh) & 0x03030303u) << 4);
        uint4 hv, lv;
        split(v, hv.x, lv.x);
        split(v >> 8, hv.y, lv.y);
        split(u, hv.z, lv.z);
        split(u >> 8, hv.w, lv.w);
        put(i, hv, lv);
    }
    return true;
}

// At 128 activation rows the drain warps hold 64 sums and 32 fresh accumulators each: registers move to them from the others.  Called
// by every warp of a warpgroup.
template <int BN, int REGS>
__device__ __forceinline__ void split_registers() {
    move_registers<BN == 128, REGS, kLaunchRegs>();
}

// One row's share of a super-block: the 16-byte header (d, dmin, packed scales) and this thread's
// 16 of the 32 quant bytes of each of the four 64-column groups.
struct RowBlock {
    uint4 hdr;
    uint4 q[4];
};

// GENERIC = false: the Q4_K kernel with exact integer operands.  GENERIC = true: any block format;
// the producers dequantise to fp32 exactly as the CPU code does and split the value, scaled by 2^10,
// into fp16 hi + lo; three MMAs per 16 columns (W_hi·x_hi, W_hi·x_lo, W_lo·x_hi); no raw-block ring.
template <int BN, bool GENERIC>
struct Tile {
    // Up to 64 activation rows the hi and lo terms of the activations sit side by side as one operand of 2·BN rows:
    // one MMA per 16 columns instead of two, the two products land in neighbouring accumulator columns and the drain adds them.
    static constexpr bool MERGED = BN <= 64;
    // Tensor memory: accumulators in a ring, behind them the W operand of every stage.  The min term of a super-block (exact kernel)
    // takes a place in the ring of accumulators like a stage does.
    static constexpr uint32_t kMainCols = MERGED ? 2 * BN : BN;
    static constexpr uint32_t CW = BN / 2;                   // columns per drain warp
    static constexpr uint32_t kXHalfBytes = BN * kBK * 2;    // one fp16 term of the activation slab
    static constexpr uint32_t kBmBytes = BN * 16 * 2;        // sub-block sums of x: BN rows × (8 hi + 8 lo)
    static constexpr uint32_t KG = groups_per_stage(BN, GENERIC);  // 64-column groups per stage
    static constexpr uint32_t SPB = 4 / KG;                        // stages per super-block
    static constexpr uint32_t kACols = (GENERIC ? 2 : 1) * KG * kBK / 2;  // tensor-memory columns of a stage's W (generic: hi, then lo)
    static constexpr uint32_t NBUF = (512 - kStages * kACols) / kMainCols;
    static constexpr uint32_t kABase = NBUF * kMainCols;
    static_assert(NBUF >= (GENERIC ? 2 : 3) && kABase + kStages * kACols <= 512, "tensor memory");
    // stage (exact):   m | KG × (x_hi | x_lo) | sums   (everything after m arrives in one bulk copy)
    // stage (generic): x_hi | x_lo
    static constexpr uint32_t kOffX = GENERIC ? 0u : kAmBytes;
    static constexpr uint32_t kOffSums = kOffX + KG * 2 * kXHalfBytes;
    static constexpr uint32_t kStageBytes = kOffSums + (GENERIC ? 0u : kBmBytes);
    static constexpr uint32_t kRaw = raw_slots_for(BN);
    static constexpr uint32_t kRawRingBytes = GENERIC ? 0u : kRaw * kRawBytes;  // generic: sized at launch
    // activation tiles in global memory, per (activation tile, super-block): four (hi, lo) slabs, then the sums
    static constexpr uint32_t kSuperBytes = 8 * kXHalfBytes + kBmBytes;
};

template <int BN, bool GENERIC>
__global__ void __launch_bounds__(kGemmThreads, 1) qgemm_tc_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ GemmMaps w_maps) {
    using T = Tile<BN, GENERIC>;
    constexpr uint32_t NBUF = T::NBUF, CW = T::CW, kXHalfBytes = T::kXHalfBytes, kStageBytes = T::kStageBytes;
    extern __shared__ __align__(128) unsigned char smem[];
    yule_pdl_launch_dependents();
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (the shuffles tell the compiler what is the same in a warp)
    unsigned char *raw = smem + (size_t)kStages * kStageBytes;  // boxes of raw Q4_K bytes
    uint64_t *bars = reinterpret_cast<uint64_t *>(raw + (GENERIC ? p.raw_ring_bytes : T::kRawRingBytes));  // full[4] empty[4] acc_full[4] acc_empty[4] raw_full[6] raw_empty[6]
    const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kStages;
    const uint32_t bar_acc_full = bar_empty + 8 * kStages, bar_acc_empty = bar_acc_full + 32;
    const uint32_t bar_raw_full = bar_acc_empty + 32, bar_raw_empty = bar_raw_full + 8 * kRawSlots;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kStages + 8 + 2 * kRawSlots);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; s++) {
            mbar_init(bar_full + 8 * s, kProdWarps + 1);  // one arrival per producer warp + the loader's expect_tx
            mbar_init(bar_empty + 8 * s, 1);              // tcgen05.commit
        }
        for (uint32_t b = 0; b < NBUF; b++) {
            mbar_init(bar_acc_full + 8 * b, 1);
            mbar_init(bar_acc_empty + 8 * b, kEpiWarps);
        }
        for (uint32_t b = 0; b < T::kRaw; b++) {
            mbar_init(bar_raw_full + 8 * b, 1);            // the loader's expect_tx
            mbar_init(bar_raw_empty + 8 * b, kProdWarps);  // every producer warp is done with the box
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    const uint32_t bpr = p.n_cols / 256;  // super-blocks per row

    if (warp >= kEpiWarps && warp < kFirstProdWarp) {
        split_registers<BN, kControlRegs>();  // (one instruction for the warpgroup)
        if (warp == kLoaderWarp) {
            if (lane == 0) {
                yule_pdl_wait();  // the activation tiles come from the kernel before this one
                RingPos ring;
                bool ok = true;
                ItemWalk items(p);
                    for (Item wi; ok && items.next(p, bpr, wi);) {
                    const unsigned char *src = reinterpret_cast<const unsigned char *>(p.xb) + (size_t)wi.nt * bpr * T::kSuperBytes;
                    for (uint32_t kb = T::SPB * wi.sb0; kb < T::SPB * wi.sb1; kb++, ring.advance(kStages)) {
                        const uint32_t s = ring.s, ph = ring.ph;
                        if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, p.status)) {
                            ok = false;
                            break;
                        }
                        const uint32_t g = kb % T::SPB;
                        const uint32_t bytes = T::KG * 2 * kXHalfBytes + ((!GENERIC && g == T::SPB - 1) ? T::kBmBytes : 0u);  // the sums ride with the last stage
                        const uint32_t dst = smem_u32(smem + (size_t)s * kStageBytes + T::kOffX);
                        mbar_arrive_expect_tx(bar_full + 8 * s, bytes);
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                                     "l"(src + (size_t)(kb / T::SPB) * T::kSuperBytes + (size_t)g * T::KG * 2 * kXHalfBytes), "r"(bytes),
                                     "r"(bar_full + 8 * s)
                                     : "memory");
                    }
                }
            }
        } else if (warp == kMmaWarp || warp == kMmaWarp2) {
            // The whole warp goes through the loop, so that addresses and descriptors are uniform registers, and one lane issues: with the loop
            // in one lane every MMA moved its operands there first, which took the issuing thread 47 clocks an MMA alone and 140 beside the
            // other roles.  The warps alternate stages, so that one waits, fences and commits while the other's MMAs run.
            //   A parity wait cannot tell a phase from the one two before it, and need not: a stage slot always belongs to the same warp (an
            // even number of slots), and of an accumulator slot's uses a warp skips so few that the drain of the use before the one it asks
            // for is known to be over: drains end in order, and it has waited for one that is at most NBUF + 3 uses back (NBUF >= 3), or
            // NBUF + 2 where no min term sits between the stages (NBUF >= 2).
            const uint32_t mine = warp == kMmaWarp ? 0u : 1u;
            // fp16 × fp16 → fp32, both operands K-major, M = 128, N = BN
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
            [[maybe_unused]] constexpr uint32_t idesc2 = (1u << 4) | ((uint32_t)((2 * BN) >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);  // N = 2·BN
            constexpr uint32_t x_lbo = BN * 16;  // bytes of one 8-column step of an activation slab (of its hi or lo rows)
            bool ok = true;
            RingPos ring, acc;
            ItemWalk items(p);
                for (Item wi; ok && items.next(p, bpr, wi);) {
                for (uint32_t kb = T::SPB * wi.sb0; kb < T::SPB * wi.sb1; kb++, ring.advance(kStages)) {
                    const uint32_t s = ring.s;
                    if ((kb & 1u) != mine) {  // (a super-block has an even number of stages)
                        acc.advance(NBUF);
                        if (!GENERIC && kb % T::SPB == T::SPB - 1) acc.advance(NBUF);
                        continue;
                    }
                    ok = mbar_wait(bar_acc_empty + 8 * acc.s, acc.ph ^ 1u, abort_flag, p.status) && mbar_wait(bar_full + 8 * s, ring.ph, abort_flag, p.status);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t d_main = tmem_base + acc.s * T::kMainCols;
                    const uint32_t stage = smem_u32(smem + (size_t)s * kStageBytes);
                    const uint32_t x_hi = stage + T::kOffX, w0 = tmem_base + T::kABase + s * T::kACols;
                    // One descriptor per stage; the 16-column steps are constants added to its address field (the
                    // issuing thread's own instruction stream, not the tensor pipe, can bound the MMA rate).
                    const uint64_t db0 = T::MERGED ? smem_desc(x_hi, 2 * x_lbo, 128) : smem_desc(x_hi, x_lbo, 128);
                    // The tensor core truncates when it adds to an accumulator, which costs a part of what the accumulator holds.  So
                    // the products with lo terms go first, or to the columns of their own: the hi·hi sums see four additions (eight at two
                    // column groups per stage), not eight or twelve.
                    auto steps = [&](auto f) {
                        f(std::integral_constant<uint32_t, 0>{});
                        f(std::integral_constant<uint32_t, 1>{});
                        f(std::integral_constant<uint32_t, 2>{});
                        f(std::integral_constant<uint32_t, 3>{});
                        if constexpr (T::KG == 2) {  // the second group's slabs follow the first's in both operands
                            f(std::integral_constant<uint32_t, 4>{});
                            f(std::integral_constant<uint32_t, 5>{});
                            f(std::integral_constant<uint32_t, 6>{});
                            f(std::integral_constant<uint32_t, 7>{});
                        }
                    };
                    constexpr uint32_t w_lo = T::kACols / 2;  // generic: the columns of the weights' lo terms
                    if (elect_one()) {
                        if constexpr (T::MERGED) {
                            steps([&](auto k16c) {
                                constexpr uint32_t k16 = decltype(k16c)::value;
                                // rows [0, BN) of an 8-column step are the hi terms, rows [BN, 2·BN) the lo terms
                                const uint64_t db = db0 + (uint64_t)((k16 * 4u * x_lbo) >> 4);
                                umma_f16_ts<(k16 != 0)>(d_main, w0 + 8 * k16, db, idesc2);  // every stage starts a fresh accumulator
                                if (GENERIC)  // the lo term of the weights against the hi term of the activations: beside the other small products
                                    umma_f16_ts<1>(d_main + BN, w0 + w_lo + 8 * k16, db, idesc);
                            });
                        } else {
                            steps([&](auto k16c) {
                                constexpr uint32_t k16 = decltype(k16c)::value;
                                const uint64_t dbh = db0 + (uint64_t)((k16 * 2u * x_lbo) >> 4);
                                umma_f16_ts<(k16 != 0)>(d_main, w0 + 8 * k16, dbh + (uint64_t)(kXHalfBytes >> 4), idesc);  // every stage starts a fresh accumulator
                                if (GENERIC)  // the lo term of the weights against the hi term of the activations
                                    umma_f16_ts<1>(d_main, w0 + w_lo + 8 * k16, dbh, idesc);
                            });
                            steps([&](auto k16c) {
                                constexpr uint32_t k16 = decltype(k16c)::value;
                                umma_f16_ts<1>(d_main, w0 + 8 * k16, db0 + (uint64_t)((k16 * 2u * x_lbo) >> 4), idesc);
                            });
                        }
                        umma_commit(bar_acc_full + 8 * acc.s);  // the accumulators may be drained once these MMAs are done
                        if (GENERIC || kb % T::SPB != T::SPB - 1) umma_commit(bar_empty + 8 * s);  // and the operands overwritten
                    }
                    __syncwarp();
                    acc.advance(NBUF);
                    if (!GENERIC && kb % T::SPB == T::SPB - 1) {  // Σ_s m_s · (sum of x over sub-block s), hi and lo sums side by side
                        ok = mbar_wait(bar_acc_empty + 8 * acc.s, acc.ph ^ 1u, abort_flag, p.status);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
                        if (elect_one()) {
                            umma_f16(tmem_base + acc.s * T::kMainCols, smem_desc(stage, 2048, 128), smem_desc(stage + T::kOffSums, x_lbo, 128), idesc, 0u);
                            umma_commit(bar_acc_full + 8 * acc.s);
                            umma_commit(bar_empty + 8 * s);
                        }
                        __syncwarp();
                        acc.advance(NBUF);
                    }
                }
            }
        } else if (warp == kRawWarp) {
            if (!GENERIC && lane == 0) {
                UnitWalk walk(p, bpr);
                for (uint32_t u = 0; walk.live; u++, walk.next(p, bpr)) {
                    const uint32_t slot = u % T::kRaw, ph = (u / T::kRaw) & 1u;
                    if (!mbar_wait(bar_raw_empty + 8 * slot, ph ^ 1u, abort_flag, p.status)) break;
                    const uint32_t x = walk.sb * 144u, y = walk.it.mt * kBM;  // byte column (a multiple of 16), first row
                    mbar_arrive_expect_tx(bar_raw_full + 8 * slot, kRawBytes);
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                            smem_u32(raw + (size_t)slot * kRawBytes)),
                        "l"(reinterpret_cast<uint64_t>(&w_maps.m[walk.it.seg])), "r"(bar_raw_full + 8 * slot), "r"(x), "r"(y)
                        : "memory");
                }
            }
        }
    } else if (warp >= kFirstProdWarp) {
        split_registers<BN, kProdRegs>();
        const uint32_t ptid = threadIdx.x - kFirstProdWarp * 32;  // 0..255
        const uint32_t r = ptid & 127u, hf = ptid >> 7;           // row of the tile, which 16 bytes of the 32
        if (GENERIC) {
            // Any block format.  The eight producer warps copy a 256-column unit of the raw bytes of the tile's 128
            // rows into one of two shared-memory slots with 16-byte cp.async from the aligned address at or below
            // each row's unit start (the blocks themselves are only 2-byte aligned), always one unit ahead of the
            // one being unpacked; thread (r, hf) then dequantises columns [32·hf, 32·hf + 32) of every stage for
            // row r from that copy with the arithmetic of the bit-exact per-element routines, scales by 2^10 and
            // splits into fp16 hi + lo.
            const uint32_t w_at = tmem_base + T::kABase + ((warp & 3u) << 21) + hf * 16;  // this warp's lanes, this thread's columns of a stage
            const uint32_t ub = p.unit_bytes, rstride = p.raw_stride, c16 = p.raw_chunks;
            const uint32_t slot_bytes = kBM * rstride;
            auto unit_start = [&](const UnitWalk &w, uint32_t tile_row) {  // address of row `tile_row`'s bytes of the unit
                uint32_t grow = w.it.mt * kBM + tile_row;
                grow = grow < p.n_rows[w.it.seg] ? grow : p.n_rows[w.it.seg] - 1;
                return reinterpret_cast<uintptr_t>(p.w[w.it.seg]) + (size_t)grow * p.w_row_bytes + (size_t)w.sb * ub;
            };
            auto copy_unit = [&](const UnitWalk &w, uint32_t u) {
                if (w.live) {
                    const uint32_t dst0 = smem_u32(raw + (size_t)(u & 1u) * slot_bytes);
                    uint32_t row = 0, c = ptid;
                    while (c >= c16) {
                        c -= c16;
                        row++;
                    }
                    for (uint32_t e = ptid; e < kBM * c16; e += 256) {
                        const uintptr_t src = (unit_start(w, row) & ~(uintptr_t)15) + (size_t)c * 16;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + row * rstride + c * 16), "l"(src) : "memory");
                        c += 256;
                        while (c >= c16) {
                            c -= c16;
                            row++;
                        }
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");  // one group per unit, empty past the end
            };
            RingPos ring;
            bool ok = true;
            UnitWalk cur(p, bpr), ahead = cur;  // the unit being unpacked and the one being copied
            copy_unit(ahead, 0);
            // A warp that has given up goes on through its units, without copying or unpacking: the barriers below count all eight warps and have no
            // bound, so one that left would keep those that passed its last wait just before it ran out.
            for (uint32_t u = 0; cur.live; u++, cur = ahead) {
                ahead.next(p, bpr);
                if (ok) copy_unit(ahead, u + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");   // this thread's copies of unit u have landed
                asm volatile("bar.sync 2, 256;" ::: "memory");         // and everyone else's
                const bool live = cur.it.mt * kBM + r < p.n_rows[cur.it.seg];
                const unsigned char *rawrow = raw + (size_t)(u & 1u) * slot_bytes + (size_t)r * rstride + (unit_start(cur, r) & 15u);
                for (uint32_t g = 0; g < 4 && ok; g++, ring.advance(kStages)) {
                    ok = mbar_wait(bar_empty + 8 * ring.s, ring.ph ^ 1u, abort_flag, p.status);
                    ok = __all_sync(0xffffffffu, ok);  // (a warp stays together: its stores are the warp's)
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t w_hi = w_at + ring.s * T::kACols, w_lo = w_hi + T::kACols / 2;
                    uint4 hi[4], lo[4];
                    const bool done = p.type == YULE_DTYPE_Q6_K && unpack32_q6k(rawrow, g * kBK + hf * 32, live, [&](uint32_t c8, const uint4 &h, const uint4 &l) { hi[c8] = h, lo[c8] = l; });
                    if (__all_sync(0xffffffffu, done)) {
#pragma unroll
                        for (uint32_t c8 = 0; c8 < 4; c8 += 2) {
                            tmem_st8(w_hi + 4 * c8, hi[c8], hi[c8 + 1]);
                            tmem_st8(w_lo + 4 * c8, lo[c8], lo[c8 + 1]);
                        }
                    } else {
#pragma unroll 1
                        for (uint32_t c8 = 0; c8 < 4; c8++) {
                            const uint32_t col0 = g * kBK + hf * 32 + c8 * 8;  // column inside the unit
                            float v[8];
                            dequant8_unit(rawrow, p.type, col0, v);
#pragma unroll
                            for (int i = 0; i < 8; i++) v[i] = live ? v[i] * kGenericWScale : 0.f;
                            // positions 0..7 of the 16 bytes hold columns 0,2,1,3,4,6,5,7 (the order of the activation tiles)
                            const float o[8] = {v[0], v[2], v[1], v[3], v[4], v[6], v[5], v[7]};
                            uint32_t h[4], l[4];
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const __half2 hh = __floats2half2_rn(o[2 * i], o[2 * i + 1]);
                                const float2 back = __half22float2(hh);
                                h[i] = as_u32(hh);
                                l[i] = as_u32(__floats2half2_rn(o[2 * i] - back.x, o[2 * i + 1] - back.y));
                            }
                            __syncwarp();
                            tmem_st4(w_hi + 4 * c8, make_uint4(h[0], h[1], h[2], h[3]));
                            tmem_st4(w_lo + 4 * c8, make_uint4(l[0], l[1], l[2], l[3]));
                        }
                    }
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_full + 8 * ring.s);
                }
                asm volatile("bar.sync 2, 256;" ::: "memory");  // the slot may be overwritten by unit u + 2
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        } else {
            bool ok = true;
            const uint32_t in_core = (r >> 3) * 128 + (r & 7u) * 16;  // place of this row in the m slab
            const uint32_t w_at = tmem_base + T::kABase + ((warp & 3u) << 21) + hf * 8;  // this warp's lanes, this thread's columns of a stage
            const __half2 k1024 = __half2half2(__ushort_as_half(0x6400)), kneg1024 = __half2half2(__ushort_as_half(0xE400));
            const __half2 kneg64 = __half2half2(__ushort_as_half(0xD400)), k16th = __half2half2(__ushort_as_half(0x2C00));
            RingPos ring;
            // the four stages of one super-block
            auto unpack_block = [&](const RowBlock &cur) {
                const ScalesMins sm = q4k_scales_mins(cur.hdr.y, cur.hdr.z, cur.hdr.w);
    #pragma unroll
                for (uint32_t g = 0; g < 4; g++) {
                    const uint32_t s = ring.s;
                    const bool opens = g % T::KG == 0, closes = g % T::KG == T::KG - 1;  // first / last group of its stage
                    // scales of sub-blocks 2g (low nibbles) and 2g + 1 (high nibbles) as fp16 pairs (sc, sc)
                    const uint32_t scw = g < 2 ? sm.sc_lo : sm.sc_hi, j0 = (2 * g) & 3u;
                    const __half2 sc0 = __hsub2(as_half2(biased_pair(scw, 0x4040u + j0 * 0x0101u)), k1024);
                    const __half2 sc1 = __hsub2(as_half2(biased_pair(scw, 0x4040u + (j0 + 1) * 0x0101u)), k1024);
                    // low nibbles: (1024 + q)·sc − 1024·sc, high nibbles where they lie: (1024 + 16·q)·(sc / 16) − 64·sc; both q·sc, exact
                    const __half2 nb0 = __hmul2(sc0, kneg1024), nb1 = __hmul2(sc1, kneg64), sc1_16 = __hmul2(sc1, k16th);  // −1024·sc ≥ −64512
                    if (opens) {
                        ok = mbar_wait(bar_empty + 8 * s, ring.ph ^ 1u, abort_flag, p.status);
                        ok = __all_sync(0xffffffffu, ok);  // (a warp stays together: its stores are the warp's)
                        if (!ok) return;
                        tc_fence_after();
                    }
                    // byte b of the 32 holds column b (low nibble, sub-block 2g) and column 32 + b (high nibble)
                    const uint32_t qw[4] = {cur.q[g].x, cur.q[g].y, cur.q[g].z, cur.q[g].w};
                    uint4 lo[2], hi[2];
    #pragma unroll
                    for (int half8 = 0; half8 < 2; half8++) {
                        const uint32_t w0 = qw[2 * half8], w1 = qw[2 * half8 + 1], w0s = w0 >> 8, w1s = w1 >> 8;
                        // pairs are bytes (0, 2) and (1, 3) of a word
                        auto low = [&](uint32_t w) { return as_u32(__hfma2(as_half2((w & 0x000F000Fu) | 0x64006400u), sc0, nb0)); };
                        auto high = [&](uint32_t w) { return as_u32(__hfma2(as_half2((w & 0x00F000F0u) | 0x64006400u), sc1_16, nb1)); };
                        lo[half8] = make_uint4(low(w0), low(w0s), low(w1), low(w1s));
                        hi[half8] = make_uint4(high(w0), high(w0s), high(w1), high(w1s));
                    }
                    // eight columns are four words of tensor memory: 16·hf of the first 32, 16·hf of the last
                    const uint32_t w = w_at + s * T::kACols + (g % T::KG) * 32;
                    tmem_st8(w, lo[0], lo[1]);
                    tmem_st8(w + 16, hi[0], hi[1]);
                    if (g == 3) {
                        // the eight mins of the super-block, twice: columns 0-7 meet the hi sums, 8-15 the lo sums
                        uint4 m;
                        m.x = as_u32(__hsub2(as_half2(biased_pair(sm.m_lo, 0x5140u)), k1024));
                        m.y = as_u32(__hsub2(as_half2(biased_pair(sm.m_lo, 0x5342u)), k1024));
                        m.z = as_u32(__hsub2(as_half2(biased_pair(sm.m_hi, 0x5140u)), k1024));
                        m.w = as_u32(__hsub2(as_half2(biased_pair(sm.m_hi, 0x5342u)), k1024));
                        *reinterpret_cast<uint4 *>(smem + (size_t)s * kStageBytes + hf * 2048 + in_core) = m;
                        fence_async_smem();  // generic-proxy stores → visible to the tensor core's reads
                    }
                    if (closes) {
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_full + 8 * s);
                        ring.advance(kStages);
                    }
                }
            };
            UnitWalk walk(p, bpr);
            for (uint32_t u = 0; walk.live && ok; u++, walk.next(p, bpr)) {
                const uint32_t slot = u % T::kRaw, ph = (u / T::kRaw) & 1u;
                ok = mbar_wait(bar_raw_full + 8 * slot, ph, abort_flag, p.status);
                if (!__all_sync(0xffffffffu, ok)) break;
                // row r of the box: 144 bytes; rows are 36 words apart, so eight lanes cover all 32 banks
                const unsigned char *bp = raw + (size_t)slot * kRawBytes + r * 144u;
                RowBlock cur;
                cur.hdr = *reinterpret_cast<const uint4 *>(bp);
    #pragma unroll
                for (int g = 0; g < 4; g++) cur.q[g] = *reinterpret_cast<const uint4 *>(bp + 16 + g * 32 + hf * 16);
                unpack_block(cur);
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_raw_empty + 8 * slot);  // this warp is done with the box
            }
        }  // exact Q4_K producer
    } else {
        split_registers<BN, kDrainRegs>();
        // drain warp: TMEM lanes [32·(warp % 4), +32) = rows of the tile, columns [CW·(warp / 4), +CW)
        yule_pdl_wait();
        const uint32_t lane_base = (warp & 3u) * 32u, col_base = (warp >> 2) * CW;
        RingPos ring;
        bool ok = true;
        ItemWalk items(p);
        for (Item wi; ok && items.next(p, bpr, wi);) {
            const uint32_t mt = wi.mt;
            const uint32_t row = mt * kBM + lane_base + lane;
            const uint8_t *rowp = p.w[wi.seg] + (size_t)(row < p.n_rows[wi.seg] ? row : p.n_rows[wi.seg] - 1) * bpr * 144;
            uint64_t acc2[CW / 2];  // pairs of sums: columns 2j, 2j + 1
#pragma unroll
            for (uint32_t j = 0; j < CW / 2; j++) acc2[j] = 0;
            uint32_t dd_cur = 0, dd_next = GENERIC ? 0u : __ldg(reinterpret_cast<const uint32_t *>(rowp + (size_t)wi.sb0 * 144));  // (d, dmin) of the first super-block
            // the accumulator at the head of the ring: wait for it, and give it back
            auto await = [&]() {
                const bool full = mbar_wait(bar_acc_full + 8 * ring.s, ring.ph, abort_flag, p.status);
                ok = __all_sync(0xffffffffu, full);  // (a warp stays together: its loads are the warp's)
                tc_fence_after();
                return tmem_base + (lane_base << 16) + ring.s * T::kMainCols + col_base;
            };
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_empty + 8 * ring.s);
                ring.advance(NBUF);
            };
            for (uint32_t sb = wi.sb0; sb < wi.sb1 && ok; sb++) {
                if (!GENERIC) {  // new super-block: take its (d, dmin), ask for the next one's
                    dd_cur = dd_next;
                    if (sb + 1 < wi.sb1) dd_next = __ldg(reinterpret_cast<const uint32_t *>(rowp + (size_t)(sb + 1) * 144));
                }
                const float2 dd = GENERIC ? make_float2(1.f, 0.f) : __half22float2(as_half2(dd_cur));
                const uint64_t d2 = pair(dd.x, dd.x);
#pragma unroll
                for (uint32_t g = 0; g < T::SPB; g++) {
                    uint32_t at = await();
                    if (!ok) break;
                    // the accumulators go back before the arithmetic on what was read last
                    if constexpr (T::MERGED) {
                        uint32_t v[CW], vl[CW];
#pragma unroll
                        for (uint32_t c0 = 0; c0 < CW; c0 += 16) {
                            tmem_ld16_issue(at + c0, v + c0);
                            tmem_ld16_issue(at + BN + c0, vl + c0);  // the products with the lo terms
                        }
                        tmem_ld_wait();
                        release();
#pragma unroll
                        for (uint32_t j = 0; j < CW; j += 2) acc2[j / 2] = fma2(d2, add2(pair_bits(v[j], v[j + 1]), pair_bits(vl[j], vl[j + 1])), acc2[j / 2]);
                    } else {
                        uint32_t v[32];
                        tmem_ld32_issue(at, v);
                        tmem_ld_wait();
#pragma unroll
                        for (uint32_t j = 0; j < 32; j += 2) acc2[j / 2] = fma2(d2, pair_bits(v[j], v[j + 1]), acc2[j / 2]);
                        tmem_ld32_issue(at + 32, v);
                        tmem_ld_wait();
                        release();
#pragma unroll
                        for (uint32_t j = 0; j < 32; j += 2) acc2[16 + j / 2] = fma2(d2, pair_bits(v[j], v[j + 1]), acc2[16 + j / 2]);
                    }
                }
                if (!GENERIC && ok) {  // the stage that ends a super-block is followed by the min term
                    const uint32_t at = await();
                    if (!ok) break;
                    constexpr uint32_t R = CW < 32 ? CW : 32;
                    const float minus_dmin = -dd.y * (1.0f / kSumScale);
                    const uint64_t m2 = pair(minus_dmin, minus_dmin);
#pragma unroll
                    for (uint32_t c0 = 0; c0 < CW; c0 += R) {
                        uint32_t v[R];
#pragma unroll
                        for (uint32_t c1 = 0; c1 < R; c1 += 16) tmem_ld16_issue(at + c0 + c1, v + c1);
                        tmem_ld_wait();
                        if (c0 + R == CW) release();
#pragma unroll
                        for (uint32_t j = 0; j < R; j += 2) acc2[(c0 + j) / 2] = fma2(m2, pair_bits(v[j], v[j + 1]), acc2[(c0 + j) / 2]);
                    }
                }
            }
            if (!ok) break;
            float acc[CW];
#pragma unroll
            for (uint32_t j = 0; j < CW; j += 2) {
                const float2 a = unpair(acc2[j / 2]);
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

// Activation rows → the GEMM's operand tiles, one CTA per (padded) row: power-of-two row scale,
// fp16 hi/lo split, the column order of the W operand inside every group of eight, and the
// per-32-column sums for the min term.  Optional prologues: RMSNorm (out = x · inv · w as in
// yule-infer/src/model_runner.rs:254-263) or SwiGLU (silu(gate) · x, kernels/cuda/silu_mul.cu:3-14).
struct XprepParams {
    const float *x;
    const float *gate;    // when set: y = silu(gate) · x
    const float *norm_w;  // when set: y = x · inv_rms · norm_w
    float eps;
    uint32_t x_stride, n_tokens, n_cols, bn;
    unsigned char *xb;
    float *oscale;
};

__device__ __forceinline__ void load8(const float *from, float (&to)[8]) {  // (the host has checked the alignment)
    const float4 a = *reinterpret_cast<const float4 *>(from), b = *reinterpret_cast<const float4 *>(from + 4);
    to[0] = a.x, to[1] = a.y, to[2] = a.z, to[3] = a.w, to[4] = b.x, to[5] = b.y, to[6] = b.z, to[7] = b.w;
}
// Power of two that puts a row's largest element in [2^13, 2^14) (a rounding above at the most).
__device__ __forceinline__ float row_scale(float amax) {
    float scale = 1.f;
    if (amax > 1e-30f && amax < 1e30f) {
        int ex;
        frexpf(amax, &ex);  // amax = m · 2^ex, m in [0.5, 1)
        scale = ldexpf(1.f, 14 - ex);
    }
    return scale;
}
// Eight columns from k0 on of (padded) activation row n, scaled, to the operand tiles; the four threads of a 32-column sub-block, `step` lanes apart, add up its
// sum, which `first` of them stores.
__device__ __forceinline__ void put_columns(const XprepParams &p, uint32_t n, uint32_t k0, float (&v)[8], float scale, uint32_t step, bool first) {
    const uint32_t nt = n / p.bn, r = n % p.bn;
    const uint32_t bpr = p.n_cols / 256;
    const uint32_t x_half_bytes = p.bn * kBK * 2, bm_bytes = p.bn * 32, super_bytes = 8 * x_half_bytes + bm_bytes;
    const uint32_t core = ((r >> 3) * 64 + (r & 7u) * 8) * 2;  // byte offset of this row inside an 8-column step
    // 16 bytes of columns [k0, k0 + 8): term 0 = hi, 1 = lo
    auto slab16 = [&](uint32_t k0, uint32_t term) {
        const uint32_t sb = k0 >> 8, g = (k0 >> 6) & 3u, kc = (k0 >> 3) & 7u;
        if (p.bn <= 64)  // hi and lo rows of an 8-column step side by side (one operand of 2·bn rows)
            return p.xb + ((size_t)nt * bpr + sb) * super_bytes + (size_t)(2 * g) * x_half_bytes + (2 * kc + term) * (p.bn * 16) + core;
        return p.xb + ((size_t)nt * bpr + sb) * super_bytes + (size_t)(2 * g + term) * x_half_bytes + kc * (p.bn * 16) + core;
    };
    // the two bytes of sub-block s (of super-block sb) in the sums slab: column s (hi) or 8 + s (lo)
    auto sum_slot = [&](uint32_t sb, uint32_t s, uint32_t term) {
        return reinterpret_cast<__half *>(p.xb + ((size_t)nt * bpr + sb) * super_bytes + 8 * (size_t)x_half_bytes +
                                          term * (p.bn * 16) + core) + s;
    };
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        v[i] *= scale;
        sum += v[i];
    }
    // positions 0..7 of the 16 bytes hold columns 0,2,1,3,4,6,5,7
    const float o[8] = {v[0], v[2], v[1], v[3], v[4], v[6], v[5], v[7]};
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __half2 hh = __floats2half2_rn(o[2 * i], o[2 * i + 1]);
        const float2 back = __half22float2(hh);
        h[i] = as_u32(hh);
        l[i] = as_u32(__floats2half2_rn(o[2 * i] - back.x, o[2 * i + 1] - back.y));
    }
    *reinterpret_cast<uint4 *>(slab16(k0, 0)) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(slab16(k0, 1)) = make_uint4(l[0], l[1], l[2], l[3]);
    // four consecutive threads of a row cover one 32-column sub-block
    sum += __shfl_xor_sync(0xffffffffu, sum, step);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2 * step);
    if (first) {
        sum *= kSumScale;  // 32 elements of up to 2^14 each: keep the sum inside fp16's range
        const __half sh = __float2half_rn(sum);
        *sum_slot(k0 >> 8, (k0 >> 5) & 7u, 0) = sh;
        *sum_slot(k0 >> 8, (k0 >> 5) & 7u, 1) = __float2half_rn(sum - __half2float(sh));
    }
}

// ROWS rows per CTA, as many threads (up to 1024) as have columns to work on; a thread keeps its 8·CHUNKS columns of a row in registers from
// the single read to the stores, so rows of up to 8192·CHUNKS / ROWS columns cost one round trip to memory and two block reductions
// whatever their length.  A thread's 16 bytes of a term lie alone in their 8-column step, the next row's 16 bytes behind them: with two rows in
// neighbouring lanes a warp writes whole 32-byte sectors, with one it writes halves.  2048 rows of 14336 columns with SwiGLU 137 -> 102 us,
// of 4096 columns with RMSNorm 29 -> 24.  Where there are not rows enough to give every SM
// two, one per CTA keeps more SMs at work.
constexpr int kXprepThreads = 1024;
constexpr uint32_t kXprepMaxRanks = 4;  // CTAs that share a row
template <int CHUNKS, int ROWS>
__global__ void __launch_bounds__(kXprepThreads) gemm_xprep_kernel(const XprepParams p) {
    yule_pdl_launch_dependents();
    yule_pdl_wait();
    __shared__ float red[32 * ROWS];
    const uint32_t lane_row = threadIdx.x % ROWS, tc = threadIdx.x / ROWS, row_threads = blockDim.x / ROWS;
    const uint32_t n = blockIdx.x * ROWS + lane_row;
    const bool live = n < p.n_tokens;  // else a padding row of the last tile: all zeros
    const float *x = p.x + (size_t)n * p.x_stride;
    const float *gate = p.gate ? p.gate + (size_t)n * p.x_stride : nullptr;
    // over the threads of a row, which are every ROWS-th lane
    auto row_reduce = [&](float v, bool is_max) {
        auto both = [&](float a, float b) { return is_max ? fmaxf(a, b) : a + b; };
        for (int o = 16; o >= ROWS; o >>= 1) v = both(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();
        if ((threadIdx.x & 31u) < ROWS) red[(threadIdx.x >> 5) * ROWS + lane_row] = v;
        __syncthreads();
        const uint32_t n_warps = blockDim.x >> 5, first = (threadIdx.x & 31u) / ROWS;
        v = 0.f;  // (sums of squares, magnitudes: nothing is below zero)
        for (uint32_t w = first; w < n_warps; w += 32 / ROWS) v = both(v, red[w * ROWS + lane_row]);
        for (int o = 16; o >= ROWS; o >>= 1) v = both(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    };
    float v[CHUNKS][8];
#pragma unroll
    for (int c = 0; c < CHUNKS; c++) {
        const uint32_t k0 = ((uint32_t)c * row_threads + tc) * 8;
        if (live && k0 < p.n_cols) {
            load8(x + k0, v[c]);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[c][i] = 0.f;
        }
    }
    if (p.norm_w) {
        float ss = 0.f;
#pragma unroll
        for (int c = 0; c < CHUNKS; c++)
#pragma unroll
            for (int i = 0; i < 8; i++) ss = fmaf(v[c][i], v[c][i], ss);
        ss = row_reduce(ss, false);
        const float inv = 1.0f / sqrtf(ss / (float)p.n_cols + p.eps);
#pragma unroll
        for (int c = 0; c < CHUNKS; c++) {
            const uint32_t k0 = ((uint32_t)c * row_threads + tc) * 8;
            if (live && k0 < p.n_cols) {
                float w[8];
                load8(p.norm_w + k0, w);
#pragma unroll
                for (int i = 0; i < 8; i++) v[c][i] = v[c][i] * inv * w[i];
            }
        }
    }
    if (gate) {
#pragma unroll
        for (int c = 0; c < CHUNKS; c++) {
            const uint32_t k0 = ((uint32_t)c * row_threads + tc) * 8;
            if (live && k0 < p.n_cols) {
                float gt[8];
                load8(gate + k0, gt);
#pragma unroll
                for (int i = 0; i < 8; i++) v[c][i] = (gt[i] / (1.0f + expf(-gt[i]))) * v[c][i];
            }
        }
    }
    float amax = 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; c++)
#pragma unroll
        for (int i = 0; i < 8; i++) amax = fmaxf(amax, fabsf(v[c][i]));
    amax = row_reduce(amax, true);
    const float scale = row_scale(amax);
    if (tc == 0) p.oscale[n] = live ? 1.0f / scale : 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; c++) {
        const uint32_t k0 = ((uint32_t)c * row_threads + tc) * 8;
        if (k0 >= p.n_cols) break;  // whole warps leave together (256 columns are 32 threads of a row)
        put_columns(p, n, k0, v[c], scale, ROWS, (tc & 3u) == 0);
    }
}

// The same for few rows: a cluster of CTAs has each row (or pair of rows), a CTA an equal share of the 256-column blocks, a thread eight columns.  What bounds one
// CTA per row is the one SM behind it: a row of 28672 columns with SwiGLU is 230 KB to read and 115 KB to write.  Sum of squares and largest element
// meet in every CTA's shared memory behind one cluster barrier: under a norm the largest is that of x · w, times the norm's factor (its roundings may
// put the scaled row's largest element at 2^14 itself, far inside the operands' range).  32 rows, us between the launches around it, one CTA per row and
// this: 4096 columns with RMSNorm 5.2 -> 3.6, 8192 6.6 -> 4.1; with SwiGLU 14336 columns 8.1 -> 5.3, 28672 15.6 -> 6.5.  128 rows of 4096
// columns 7.7 -> 5.0, 256 7.5 -> 4.8.
template <int ROWS>
__global__ void __launch_bounds__(kXprepThreads) gemm_xprep_cluster_kernel(const XprepParams p) {
    yule_pdl_launch_dependents();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (every CTA of the cluster runs before another stores to it)
    __shared__ float2 red[32 * ROWS], shares[kXprepMaxRanks * ROWS];  // (sum of squares, largest)
    uint32_t rank, ranks;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(ranks));
    const uint32_t lane_row = threadIdx.x % ROWS, tc = threadIdx.x / ROWS, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t n = blockIdx.x / ranks * ROWS + lane_row, blocks = p.n_cols / 256, b0 = blocks * rank / ranks, b1 = blocks * (rank + 1) / ranks;
    const uint32_t k0 = b0 * 256 + tc * 8;
    const bool live = n < p.n_tokens, mine = k0 < b1 * 256;  // (`mine`: whole warps)
    float v[8] = {}, w[8] = {}, ss = 0.f, most = 0.f;
    auto reduce = [&]() {  // over the lanes of a row
#pragma unroll
        for (int o = 16; o >= ROWS; o >>= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
        }
    };
    if (live && mine && p.norm_w) load8(p.norm_w + k0, w);  // (weights: nothing before this launch writes them)
    yule_pdl_wait();
    if (live && mine) {
        load8(p.x + (size_t)n * p.x_stride + k0, v);
        if (p.gate) {
            float gt[8];
            load8(p.gate + (size_t)n * p.x_stride + k0, gt);
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = (gt[i] / (1.0f + expf(-gt[i]))) * v[i];
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            ss = fmaf(v[i], v[i], ss);
            most = fmaxf(most, fabsf(p.norm_w ? v[i] * w[i] : v[i]));
        }
    }
    reduce();
    if (lane < ROWS) red[warp * ROWS + lane] = make_float2(ss, most);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        ss = 0.f, most = 0.f;
        for (uint32_t i = lane / ROWS; i < (blockDim.x >> 5); i += 32 / ROWS) {
            const float2 r = red[i * ROWS + lane_row];
            ss += r.x, most = fmaxf(most, r.y);
        }
        reduce();
        for (uint32_t to_rank = lane / ROWS; to_rank < ranks; to_rank += 32 / ROWS) {  // this CTA's share to slot `rank` of every CTA
            uint32_t to;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(smem_u32(&shares[rank * ROWS + lane_row])), "r"(to_rank));
            asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(ss), "f"(most) : "memory");
        }
        __syncwarp();
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    ss = 0.f, most = 0.f;
    for (uint32_t i = 0; i < ranks; i++) {
        const float2 r = shares[i * ROWS + lane_row];
        ss += r.x, most = fmaxf(most, r.y);
    }
    if (p.norm_w) {
        const float inv = 1.0f / sqrtf(ss / (float)p.n_cols + p.eps);
        most *= inv;
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = v[i] * inv * w[i];
    }
    const float scale = row_scale(most);
    if (rank == 0 && tc == 0) p.oscale[n] = live ? 1.0f / scale : 0.f;
    if (mine) put_columns(p, n, k0, v, scale, ROWS, (tc & 3u) == 0);
}

// 2-D view of a Q4_K matrix for the TMA engine: bytes along a row, rows; box = one super-block
// (144 bytes) of 128 rows.  Rows past the end read as zeros (a block of zeros dequantises to 0).
cudaError_t encode_weight_map(const uint8_t *w, uint32_t n_rows, uint32_t n_cols, CUtensorMap *out) {
    const uint64_t row_bytes = (uint64_t)(n_cols / 256) * 144;
    return cached_tensor_map_2d(w, 1, row_bytes, n_rows, row_bytes, 144, kBM, out);  // one driver call per (tensor, shape), not per launch
}

template <int BN, bool GENERIC>
cudaError_t launch_gemm(const GemmParams &p, const GemmMaps &w_maps, uint32_t grid, size_t smem, bool pdl, cudaStream_t s) {
    auto kern = qgemm_tc_kernel<BN, GENERIC>;
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
            if (e == cudaSuccess && BN == 128 && fa.numRegs < kLaunchRegs) e = cudaErrorInvalidValue;
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    return launch_kernel(kern, dim3(grid), dim3(kGemmThreads), smem, s, pdl, p, w_maps);
}

// Which tiles are dealt by super-blocks: those that do not fill a round of CTAs, a tile to sixteen CTAs at the most (its parts have to be added up), at least
// four super-blocks to a CTA.  A part costs its stores, a ticket and its share of the sum, some 3 to 5 us that the tensor pipe waits in part, against
// super-blocks of 1.8 us at 128 activation rows and 1.1 at 32.  So not where that would shorten the round by fewer than three super-blocks, and runs that
// end inside a tile, with two parts for most CTAs, only where they shorten it by four more (128 rows) or eight (32 rows: 64 tiles of 32 super-blocks in halves
// 21 us, in 148 equal runs 23.5; 80 tiles 31 us whole, 25 in equal runs; 448 tiles 119.5 us as four rounds, 104 as three and the rest in parts).
// Nor runs in place of a round of whole tiles of which they spare no more than an eighth: their CTAs are at different columns, and share nothing in the caches that they
// do not hold whole (8192x28672 by 2016 rows, 136 tiles beyond six rounds: 2291 us whole, 2354 in 148 runs; 128 tiles of 32 super-blocks 75.2, 76.3; 120 of 56 127.9, 120.6).
void split_tiles(GemmParams &p, uint32_t tiles, uint32_t bpr, uint32_t ctas) {
    p.split_tiles = p.split_ctas = p.split_units = 0;
    const uint32_t rest = tiles % ctas, units = rest * bpr;
    if (rest == 0) return;
    uint32_t most = 16, run = 4;
    if (const char *k = knob("YULE_GEMM_KSPLIT"))
        if (atoi(k) > 0) most = (uint32_t)atoi(k), run = 1;
    auto least = [](uint32_t a, uint32_t b, uint32_t c) { return a < b ? (a < c ? a : c) : (b < c ? b : c); };
    const uint32_t parts = least(ctas / rest, most, bpr / run), even = parts > 1 ? rest * parts : rest;  // every tile in equal parts
    const uint32_t equal = least(ctas, rest * most, units / run);                                         // runs that may end inside a tile
    auto longest = [&](uint32_t to) { return (units + to - 1) / to; };
    uint32_t to = even;
    if (equal > even && longest(even) >= longest(equal) + (p.bn >= 128 ? 4u : 8u) && (even > rest || longest(even) > longest(equal) + bpr / 8)) to = equal;
    if (to <= rest || (run > 1 && bpr < longest(to) + 3)) return;
    p.split_tiles = rest;
    p.split_ctas = to;
    p.split_units = units;
}

uint32_t pick_bn(uint32_t n_tokens) { return n_tokens <= 32 ? 32 : (n_tokens <= 64 ? 64 : 128); }

}  // namespace

// The same through a per-process cache: a map depends on the address and the shape only, and encoding one costs a
// driver call, which the matvec entry points would otherwise pay on every launch.
cudaError_t cached_tensor_map_2d(const void *base, uint32_t elem_bytes, uint64_t inner, uint64_t n_rows, uint64_t row_stride_bytes,
                                 uint32_t box_inner, uint32_t box_rows, void *out, uint32_t swizzle) {
    struct Key {
        const void *base;
        uint64_t inner, n_rows, stride;
        uint32_t elem, box_inner, box_rows, swizzle;
        bool operator==(const Key &o) const {
            return base == o.base && inner == o.inner && n_rows == o.n_rows && stride == o.stride && elem == o.elem &&
                   box_inner == o.box_inner && box_rows == o.box_rows && swizzle == o.swizzle;
        }
    };
    struct Hash {
        size_t operator()(const Key &k) const {
            size_t h = std::hash<const void *>()(k.base);
            for (uint64_t v : {k.inner, k.n_rows, k.stride, (uint64_t)k.elem, (uint64_t)k.box_inner, (uint64_t)k.box_rows, (uint64_t)k.swizzle})
                h = h * 0x9E3779B97F4A7C15ull + std::hash<uint64_t>()(v);
            return h;
        }
    };
    static std::unordered_map<Key, CUtensorMap, Hash> cache;
    static std::mutex mu;
    const Key key{base, inner, n_rows, row_stride_bytes, elem_bytes, box_inner, box_rows, swizzle};
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it == cache.end()) {
        CUtensorMap m;
        cudaError_t e = encode_tensor_map_2d(base, elem_bytes, inner, n_rows, row_stride_bytes, box_inner, box_rows, &m, swizzle);
        if (e != cudaSuccess) return e;
        if (cache.size() >= 16384) cache.clear();
        it = cache.emplace(key, m).first;
    }
    memcpy(out, &it->second, sizeof(CUtensorMap));
    return cudaSuccess;
}

// Tiled 2-D tensor map over rows of `elem_bytes`-sized elements (1 or 8): `inner` elements per row, `n_rows` rows
// `row_stride_bytes` apart (a multiple of 16; base 16-byte aligned), box of box_inner x box_rows elements, swizzled
// within 0 (not at all), 64 or 128 bytes, out-of-range elements read as zeros.  `out` is a CUtensorMap.
cudaError_t encode_tensor_map_2d(const void *base, uint32_t elem_bytes, uint64_t inner, uint64_t n_rows, uint64_t row_stride_bytes,
                                 uint32_t box_inner, uint32_t box_rows, void *out, uint32_t swizzle) {
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    static std::mutex mu;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!encode) {
            void *fn = nullptr;
            cudaDriverEntryPointQueryResult qres;
            cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
            if (e != cudaSuccess) return e;
            if (qres != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
            encode = reinterpret_cast<EncodeFn>(fn);
        }
    }
    if (elem_bytes != 1 && elem_bytes != 8) return cudaErrorInvalidValue;
    const cuuint64_t dims[2] = {inner, n_rows};
    const cuuint64_t strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = encode(static_cast<CUtensorMap *>(out), elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT64, 2,
                        const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        swizzle == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : swizzle == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Q4_K runs on the exact-integer kernel here up to 64 activation rows, beyond and for Q8_0, Q4_0, Q5_K and Q6_K on that of qgemm_int.cu, the others on the generic one (YULE_GEMM_GENERIC=1
// sends all of them there, for comparison).  The activation tiles are laid out per 256 columns.
bool qgemm_supported(uint32_t type, uint32_t n_cols, uint32_t n_tokens) {
    return is_quantized(type) && n_cols % 256 == 0 && n_cols > 0 && n_cols <= 65536 && n_tokens >= 1;
}

size_t qgemm_scratch_bytes(uint32_t n_tokens, uint32_t n_cols) {
    const uint32_t bn = pick_bn(n_tokens);
    const size_t padded = (size_t)((n_tokens + bn - 1) / bn) * bn;
    return kGemmSplitBytes + padded * n_cols * 4 + padded * (n_cols / 256) * 32 + padded * sizeof(float) + 512;
}

cudaError_t launch_qgemm_xprep(const QGemm &g, int sm_count, cudaStream_t s, uint64_t *launches) {
    if (!qgemm_supported(g.type, g.n_cols, g.n_tokens)) return cudaErrorInvalidValue;
    // rows are read 16 bytes at a time: buffers start on 256-byte boundaries, and the entry points take strides of whole float4s only
    if (((reinterpret_cast<uintptr_t>(g.x) | reinterpret_cast<uintptr_t>(g.gate) | reinterpret_cast<uintptr_t>(g.norm_w)) & 15) || g.x_stride % 4) return cudaErrorInvalidValue;
    const uint32_t bn = pick_bn(g.n_tokens);
    const uint32_t n_ntiles = (g.n_tokens + bn - 1) / bn, padded = n_ntiles * bn;
    unsigned char *xb = reinterpret_cast<unsigned char *>(g.scratch) + kGemmSplitBytes;
    const size_t tiles_bytes = (size_t)padded * g.n_cols * 4 + (size_t)padded * (g.n_cols / 256) * 32;
    float *oscale = reinterpret_cast<float *>(xb + ((tiles_bytes + 255) & ~(size_t)255));

    XprepParams xp = {};
    xp.x = g.x;
    xp.gate = g.gate;
    xp.norm_w = g.norm_w;
    xp.eps = g.eps;
    xp.x_stride = g.x_stride;
    xp.n_tokens = g.n_tokens;
    xp.n_cols = g.n_cols;
    xp.bn = bn;
    xp.xb = xb;
    xp.oscale = oscale;
    cudaError_t e;
    auto launch = [&](auto kern, uint32_t chunks, uint32_t rows) {
        return launch_kernel(kern, dim3(padded / rows), dim3(rows * (((g.n_cols / 8 + chunks - 1) / chunks + 31) / 32 * 32)), 0, s, g.pdl, xp);
    };
    // A row on a cluster where it is read at once: all rows together are a CTA of 1024 threads per SM at the most (beyond: 128 rows of 14336 columns 8.7 us with one
    // CTA per row, 9.8 on clusters of four; 28672: 16.9 and 22.9), and there are not rows enough for two per SM.  Clusters of four up to 64 rows, two beyond (8192
    // columns: 32 rows 4.5 us with two, 4.1 with four, 4.2 with eight; 128 rows 5.4 and 5.3 with two and four); two rows per CTA where they fit.
    // Not rows that are only laid out, on clusters of two, by a launch that nothing hides: its start costs more than a half row saves (a call of 128 rows and 128 rows of W,
    // re-layout and GEMM: 1024 columns 22.3 us, 21.4 with one CTA per row, 2048 25.3, 23.5, 4096 27.1, 25.8; in a prompt's chain of launches the same or 1 % for the clusters).
    const uint32_t blocks = g.n_cols / 256, ranks = 2 * padded <= (uint32_t)sm_count ? 4 : 2, share = (blocks + ranks - 1) / ranks, most_warps = kXprepThreads / 32;
    const bool plain = !g.gate && !g.norm_w && !g.pdl && ranks == 2;
    if (!plain && padded < 2 * (uint32_t)sm_count && (uint64_t)padded * g.n_cols <= (uint64_t)kXprepThreads * 8 * sm_count && blocks >= ranks && share <= most_warps && !(g.gate && g.norm_w)) {
        const uint32_t rows = 2 * share <= most_warps ? 2 : 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(padded / rows * ranks);
        cfg.blockDim = dim3(share * 32 * rows);
        cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ranks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = g.pdl ? 2 : 1;
        e = rows == 2 ? launch_config<XprepParams>(cfg, gemm_xprep_cluster_kernel<2>, xp) : launch_config<XprepParams>(cfg, gemm_xprep_cluster_kernel<1>, xp);
    } else if (padded >= 2 * (uint32_t)sm_count && g.n_cols <= 16384)  // (padded is a multiple of 32)
        e = g.n_cols <= 4096 ? launch(gemm_xprep_kernel<1, 2>, 1, 2) : (g.n_cols <= 8192 ? launch(gemm_xprep_kernel<2, 2>, 2, 2) : launch(gemm_xprep_kernel<4, 2>, 4, 2));
    else if (g.n_cols <= 8192)
        e = launch(gemm_xprep_kernel<1, 1>, 1, 1);
    else if (g.n_cols <= 16384)
        e = launch(gemm_xprep_kernel<2, 1>, 2, 1);
    else if (g.n_cols <= 32768)
        e = launch(gemm_xprep_kernel<4, 1>, 4, 1);
    else if (g.n_cols <= 65536)
        e = launch(gemm_xprep_kernel<8, 1>, 8, 1);
    else
        return cudaErrorInvalidValue;
    if (e != cudaSuccess) return e;
    *launches += 1;
    return cudaSuccess;
}

cudaError_t launch_qgemm_mm(const QGemm &g, int sm_count, cudaStream_t s, uint64_t *launches) {
    if (!qgemm_supported(g.type, g.n_cols, g.n_tokens) || g.n_rows == 0) return cudaErrorInvalidValue;
    if (g.n_more > (uint32_t)kGemmSegs - 1 || (g.n_more && g.residual)) return cudaErrorInvalidValue;
    const uint32_t bn = pick_bn(g.n_tokens);
    const uint32_t n_ntiles = (g.n_tokens + bn - 1) / bn, padded = n_ntiles * bn;
    unsigned char *xb = reinterpret_cast<unsigned char *>(g.scratch) + kGemmSplitBytes;
    const size_t tiles_bytes = (size_t)padded * g.n_cols * 4 + (size_t)padded * (g.n_cols / 256) * 32;
    float *oscale = reinterpret_cast<float *>(xb + ((tiles_bytes + 255) & ~(size_t)255));
    cudaError_t e;
    GemmParams p = {};
    p.xb = reinterpret_cast<const __half *>(xb);
    p.oscale = oscale;
    p.residual = g.residual;
    p.n_cols = g.n_cols;
    p.n_tokens = g.n_tokens;
    p.bn = bn;
    p.n_seg = 1 + g.n_more;
    for (uint32_t i = 0; i < p.n_seg; i++) {
        p.w[i] = i ? g.w_more[i - 1] : g.w;
        p.out[i] = i ? g.out_more[i - 1] : g.out;
        p.n_rows[i] = i ? g.n_rows_more[i - 1] : g.n_rows;
        p.out_stride[i] = i ? g.out_stride_more[i - 1] : g.out_stride;
        if (!p.w[i] || !p.out[i] || p.n_rows[i] == 0) return cudaErrorInvalidValue;
        p.mt0[i + 1] = p.mt0[i] + (p.n_rows[i] + kBM - 1) / kBM;
    }
    for (uint32_t i = p.n_seg; i < (uint32_t)kGemmSegs; i++) p.mt0[i + 1] = p.mt0[p.n_seg];
    p.n_mtiles = p.mt0[p.n_seg];
    p.n_ntiles = n_ntiles;
    const uint32_t ctas = (uint32_t)sm_count < kGemmMaxCtas ? (uint32_t)sm_count : kGemmMaxCtas, tiles = p.n_mtiles * p.n_ntiles;
    split_tiles(p, tiles, g.n_cols / 256, ctas);
    p.by_ctas = divide_by(p.split_ctas);
    p.by_units = divide_by(p.split_units);
    p.by_bpr = divide_by(g.n_cols / 256);
    p.by_ntiles = divide_by(n_ntiles);
    p.split_tickets = reinterpret_cast<uint32_t *>(g.scratch);
    p.split_part = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(g.scratch) + kGemmTicketBytes);
    p.status = g.status;
    p.truncation = kTruncation;
    p.out_scale = 1.0f;
    const uint32_t grid = tiles > p.split_tiles ? (tiles < ctas ? tiles : ctas) : p.split_ctas;
    p.w_row_bytes = (uint64_t)(g.n_cols / block_size(g.type)) * block_bytes(g.type);
    const bool forced = knob("YULE_GEMM_GENERIC") && atoi(knob("YULE_GEMM_GENERIC"));
    if (!forced && qgemm_int_supported(g)) {
        e = launch_qgemm_int(g, &p, grid, s);
        if (e != cudaSuccess) return e;
        *launches += 1;
        return cudaSuccess;
    }
    const bool generic = forced || g.type != YULE_DTYPE_Q4_K;
    const uint32_t kg = groups_per_stage(bn, generic);
    const uint32_t stage_bytes = kg * 2 * bn * kBK * 2 + (generic ? 0u : kAmBytes + bn * 32);
    p.unit_bytes = 256 / block_size(g.type) * block_bytes(g.type);
    p.raw_chunks = (p.unit_bytes + 14 + 15) / 16;      // covers the unit from any 2-byte-aligned start
    p.raw_stride = (p.raw_chunks | 1u) * 16;            // an odd multiple of 16 bytes
    p.raw_ring_bytes = (2 * kBM * p.raw_stride + 127u) & ~127u;
    const size_t raw_ring = generic ? p.raw_ring_bytes : (size_t)raw_slots_for(bn) * kRawBytes;
    p.type = g.type;
    if (generic) p.out_scale /= kGenericWScale;
    const size_t tail_bytes = raw_ring + (2 * kStages + 8 + 2 * kRawSlots) * 8 + 32;
    const size_t smem = kStages * stage_bytes + tail_bytes;
    GemmMaps w_maps;
    memset(&w_maps, 0, sizeof(w_maps));
    if (!generic) {
        for (uint32_t i = 0; i < p.n_seg; i++) {
            e = encode_weight_map(p.w[i], p.n_rows[i], g.n_cols, &w_maps.m[i]);
            if (e != cudaSuccess) return e;
        }
    }
    if (generic)
        e = bn == 32 ? launch_gemm<32, true>(p, w_maps, grid, smem, g.pdl, s) : (bn == 64 ? launch_gemm<64, true>(p, w_maps, grid, smem, g.pdl, s) : launch_gemm<128, true>(p, w_maps, grid, smem, g.pdl, s));
    else
        e = bn == 32 ? launch_gemm<32, false>(p, w_maps, grid, smem, g.pdl, s) : launch_gemm<64, false>(p, w_maps, grid, smem, g.pdl, s);
    if (e != cudaSuccess) return e;
    *launches += 1;
    return cudaSuccess;
}

cudaError_t launch_qgemm(const QGemm &g, int sm_count, cudaStream_t s, uint64_t *launches) {
    if (g.n_rows == 0) return cudaErrorInvalidValue;
    cudaError_t e = launch_qgemm_xprep(g, sm_count, s, launches);
    if (e != cudaSuccess) return e;
    QGemm mm = g;
    mm.pdl = true;  // behind the re-layout of its own activations: only the weight copies run ahead of it
    return launch_qgemm_mm(mm, sm_count, s, launches);
}

}  // namespace yule
