// qmv_digits.cu — fused dequantise + matvec for one activation vector, every tuned block format (Q4_K, Q5_K, Q6_K on
// its row-planar copy, Q8_0, Q4_0), on the integer pipe of `mma.sync`, with the neighbouring ops of a decode step folded in.
//
// Contract: yule-core/src/dequant.rs:902-1009 (and :297-338 for Q5_K) — per row the sum over scale groups of
// d·sc·Σ q·x minus the offset or min term.
//
// Arithmetic.  The quants go into m16n8k32 u8 (Q8_0: s8) operands as they are: one AND per four 4-bit weights, nothing
// for a byte.  The activations of 128 columns become 31-bit integers times a power of two of their own, M = round(x·2^e)
// with |M| < 2^30 — exact for every element within 2^-6 of the largest of the 128, off by at most 2^-30 of that one
// otherwise (a 24-bit float split into fp16 hi + lo keeps 22 bits) — and M's four signed base-256 digits are four B columns:
// D[row][digit] = Σ q·digit is an exact 32-bit integer.  A k32 MMA takes 16 columns of one scale group (k 0-15, B columns
// 0-3) and 16 of the next (k 16-31, B columns 4-7; the other half of each B column is zero), so lane t of a quad
// receives two digits of ONE group and applies that group's scale only.  The accumulator starts at the bits of 1.5·2^23
// and is read back as a float: no conversion instruction.  Scales, 2^-e and the sub-block sums of x (min and offset
// terms) are fp32.  Everything after the rounding of x is exact or fp32 in another order than the CPU's.
//   Why integers: measured here, mma.sync m16n8k32 on 8-bit integers issues every 8.0 clocks per SM sub-partition, the
//   same as m16n8k16 f16 with half the weights (fp8 operands are turned into f16 ones), and logic ops run at half rate, so
//   fewer MMAs (8 instead of 32 per 4096 Q4_K weights) and fewer unpacking ops (3 instead of 5 per word) both count:
//   the fp16 formulation this replaced was bound by the two at 0.64 of the copy bandwidth on a 128256x4096 matrix.
//
// Schedule.  16 warps that multiply and one that copies (8 and one for independent calls, see launch_sized); one CTA per SM, whose shared memory holds the digits of x and a ring
// of weight stages (tiled TMA copies, the first ones issued before `griddepcontrol.wait`).  A stage is two boxes of 16
// rows x 2048 columns, one 256-column block per warp: two neighbouring column ranges of one 16-row tile, or the same
// columns of two tiles (of gate and up for a pair), whichever leaves fewer warps idle.  Units of one or two tiles are
// dealt round-robin.  Row sums meet in shared memory; the warps take turns finishing units (one named barrier per unit in
// flight, only the finishing warp waits on it, and a warp whose copy never came).  Rows longer than the image of x may be are several launches over a
// part of the columns each, every one adding to the result of the one before.
//   In a chain of dependent launches two CTAs of 16 warps to an SM (half the shared memory each) were tried: the hardware puts two
// CTAs of one launch on an SM as soon as there is room, 148 CTAs landed on 74 to 97 SMs, and the chain took 1.3 times as long.
//
// Folded in: RMSNorm of x (the 1/rms factor multiplies the finished rows), up to three matrices that share x, SiLU(gate)·up
// of a pair, the residual, and under tensor parallelism the (value, epoch) pairs of the exchange.

#include <cuda.h>
#include <cuda_fp16.h>

#include <mutex>

#include "internal.h"

namespace yule {

namespace {

#include "ring_common.cuh"
#include "tp_pairs.cuh"

// Warps that multiply, W: 16, or 8 in CTAs of half the size; and one that issues the copies.
__host__ __device__ constexpr int mul_threads(int w) { return w * 32; }
__host__ __device__ constexpr int cta_threads(int w) { return w * 32 + 32; }
// CTAs that registers leave room for on an SM
__host__ __device__ constexpr int ctas_per_sm(int w) { return w == 8 ? 3 : 1; }
constexpr int kTileRows = 16;
constexpr uint32_t kMaxSlots = 8;        // ring slots
constexpr uint32_t kMaxFinish = 8;       // tiles whose sums may be waiting for their finishing warp
// Shared memory of a CTA where `share` of them are to fit on an SM (one: leaves room for a CTA of the small kernels of a chain)
__host__ __device__ constexpr size_t max_smem(uint32_t share) { return (share == 3 ? 72 : share == 2 ? 110 : 200) * (size_t)1024; }

enum : int { kQ4K, kQ5K, kQ6K, kQ8, kQ4 };

// Shared-memory stage of a format.  Row pitches are ≡ 32 or 96 (mod 128) where lanes read 8 bytes, ≡ 16 where they read
// 4, so that the rows of a fragment fall into distinct banks.
template <int F>
struct Fmt {
    static constexpr uint32_t kBoxBlocks = 8;             // 256-column blocks per row in a box
    static constexpr uint32_t kCopies = F == kQ8 ? 2 : 1;  // a Q8_0 row of eight blocks is longer than a tiled copy may be
    static constexpr uint32_t kBlockBytes = F == kQ4K ? 144 : F == kQ5K ? 176 : F == kQ8 ? 272 : F == kQ4 ? 144 : 0;
    static constexpr int kPlanes = F == kQ6K ? 4 : 1;
    static constexpr uint32_t kPitch = F == kQ6K ? 0 : kBoxBlocks / kCopies * kBlockBytes + (F == kQ4 ? 16 : 32);
    // Q6_K planes: low nibbles, high bit pairs, scales, d
    static constexpr uint32_t kQlPitch = 1024 + 16, kQhPitch = 512 + 16, kScPitch = 128 + 16, kDPitch = 16;
    static constexpr uint32_t kQhOff = kTileRows * kQlPitch, kScOff = kQhOff + kTileRows * kQhPitch, kDOff = kScOff + kTileRows * kScPitch;
    static constexpr uint32_t kBoxBytes = F == kQ6K ? kDOff + kTileRows * kDPitch : kCopies * kTileRows * kPitch;
    static_assert(kBoxBytes % 128 == 0, "boxes stay 128-byte aligned");
    static constexpr uint32_t kGroupCols = F == kQ6K ? 16 : 32;           // columns that share a scale
};

template <int F>
struct DigitsParams {
    CUtensorMap map[3 * Fmt<F>::kPlanes];
    float *out[3];
    uint32_t seg_rows[3], seg_tiles[3];
    uint32_t n_seg, n_tiles, n_units, pair, two_tiles;  // two_tiles: a unit is two tiles (pair: one of gate, one of up)
    uint32_t n_cols, col0, full_cols;  // columns of this launch, the first of them, columns of a row
    const float *x, *norm_w;
    float eps;
    const float *residual;             // segment 0
    uint32_t slots, finish;
    uint32_t late_wait, accumulate;
    int *status;
    long long wait_cycles;
    TpFuse tp;
};

struct Smem {
    unsigned char *ring;
    unsigned char *img;   // digits of x: 4 bytes per column
    float *f, *sx;        // 2^-e per 128 columns; (offset constant ·) Σx per scale group
    float *red;           // sums of squares per warp
    float *inv;           // 1/rms
    float *part;          // [finish][matrix of a pair whose tiles go one by one][warp][row]
    uint64_t *bars;       // full[kMaxSlots], empty[kMaxSlots]
};
__host__ __device__ inline size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }
template <int F, int W>
constexpr uint32_t kStageBytes = W / 8 * Fmt<F>::kBoxBytes;
template <int F, int W>
__host__ __device__ inline size_t fixed_bytes(uint32_t n_cols, uint32_t finish, uint32_t nq) {
    return (size_t)n_cols * 4 + align16((size_t)(n_cols / 128) * 4) + align16((size_t)(n_cols / Fmt<F>::kGroupCols) * 4) + 64 + 16 +
           (size_t)finish * nq * W * kTileRows * 4 + 2 * kMaxSlots * 8;
}
template <int F, int W>
__device__ __forceinline__ Smem carve(unsigned char *base, uint32_t n_cols, uint32_t slots, uint32_t finish, uint32_t nq) {
    Smem s;
    s.ring = base;
    size_t off = (size_t)slots * kStageBytes<F, W>;
    s.img = base + off;
    off += (size_t)n_cols * 4;
    s.f = reinterpret_cast<float *>(base + off);
    off += align16((size_t)(n_cols / 128) * 4);
    s.sx = reinterpret_cast<float *>(base + off);
    off += align16((size_t)(n_cols / Fmt<F>::kGroupCols) * 4);
    s.red = reinterpret_cast<float *>(base + off);
    off += 64;
    s.inv = reinterpret_cast<float *>(base + off);
    off += 16;
    s.part = reinterpret_cast<float *>(base + off);
    off += (size_t)finish * nq * W * kTileRows * 4;
    s.bars = reinterpret_cast<uint64_t *>(base + off);
    return s;
}

// D = A·B + (the bits of 1.5·2^23): as a float, 1.5·2^23 + the integer sum (|sum| < 2^22)
constexpr uint32_t kIntBase = 0x4B400000u;
constexpr float kFloatBase = 12582912.f;
template <bool SIGNED>
__device__ __forceinline__ void mma_first(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (SIGNED)
        asm volatile(
            "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(kIntBase));
    else
        asm volatile(
            "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(kIntBase));
}
template <bool SIGNED>
__device__ __forceinline__ void mma_next(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (SIGNED)
        asm volatile(
            "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile(
            "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the lane's two digits of a row as one number (the upper pair's 2^16 is applied at the end)
__device__ __forceinline__ float two_digits(uint32_t lo, uint32_t hi) {
    return fmaf(__uint_as_float(hi) - kFloatBase, 256.f, __uint_as_float(lo) - kFloatBase);
}
__device__ __forceinline__ float half_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
__device__ __forceinline__ float half_at(const unsigned char *p) { return half_bits(*reinterpret_cast<const unsigned short *>(p)); }
constexpr float kMagic = 8388608.f;
// 2^23 + byte `i` of w (i < 4), as a float
__device__ __forceinline__ float magic_byte(uint32_t w, uint32_t i) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + i)); }
__device__ __forceinline__ uint32_t lds32(const unsigned char *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ uint2 lds64(const unsigned char *p) { return *reinterpret_cast<const uint2 *>(p); }
__device__ __forceinline__ uint4 lds128(const unsigned char *p) { return *reinterpret_cast<const uint4 *>(p); }

constexpr uint32_t kNib = 0x0F0F0F0Fu;
constexpr uint32_t kImgHalf = 512;  // bytes of 128 columns in the image: 8 B columns x 4 lanes x 16 bytes

// B operands of a lane: k 0-15 (live in the lanes of columns 0-3, zero in the others) and k 16-31 (the other way round).
// The dead half is set to zero once and never loaded.
struct BRegs {
    uint32_t lo[4] = {0u, 0u, 0u, 0u}, hi[4] = {0u, 0u, 0u, 0u};
    __device__ __forceinline__ void load(uint32_t addr, uint32_t is_lo) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %9, 0;\n\t"
            "@p ld.shared.v4.u32 {%0,%1,%2,%3}, [%8];\n\t"
            "@!p ld.shared.v4.u32 {%4,%5,%6,%7}, [%8];\n\t}"
            : "+r"(lo[0]), "+r"(lo[1]), "+r"(lo[2]), "+r"(lo[3]), "+r"(hi[0]), "+r"(hi[1]), "+r"(hi[2]), "+r"(hi[3])
            : "r"(addr), "r"(is_lo)
            : "memory");
    }
};
// What stays the same for a lane: its place in the image, which k half of its B column is live, the group it scales.
struct LaneView {
    uint32_t img;    // shared-memory address
    uint32_t is_lo;
    uint32_t sub;    // t >> 1
};
// Running sums of one lane: rows g and g + 8, its pair of digits (a) and the terms that are charged once (m).
struct Acc {
    float a0 = 0.f, a1 = 0.f, m0 = 0.f, m1 = 0.f;
};

// Each of the consume routines multiplies one block (256 columns) of rows g and g + 8.  `blk` is its index in the image;
// `r0` the bytes of row g's block in the stage.
template <bool Q5>
__device__ __forceinline__ void consume_q4k(const unsigned char *r0, uint32_t blk, int t, const LaneView &lv, const Smem &sm, BRegs &b, Acc &acc) {
    using S = Fmt<Q5 ? kQ5K : kQ4K>;
    const unsigned char *r1 = r0 + 8 * S::kPitch;
    const uint4 h0 = lds128(r0), h1 = lds128(r1);
    uint2 e0 = {}, e1 = {};
    if (Q5) e0 = lds64(r0 + 16 + 8 * t), e1 = lds64(r1 + 16 + 8 * t);  // fifth bits: bit s of byte l belongs to sub-block s, column l
    const float d0 = half_bits(h0.x), d1 = half_bits(h1.x);
    float m_0 = 0.f, m_1 = 0.f;
#pragma unroll
    for (int u = 0; u < 2; u++) {  // halves of 128 columns
        b.load(lv.img + (blk * 2 + u) * kImgHalf, lv.is_lo);
        const float f = sm.f[blk * 2 + u], sx = sm.sx[blk * 8 + 4 * u + t];
        uint32_t sc0, mn0, sc1, mn1;  // four 6-bit scales and mins each (dequant.rs:176-190)
        if (u == 0) {
            sc0 = h0.y & 0x3F3F3F3Fu, mn0 = h0.z & 0x3F3F3F3Fu;
            sc1 = h1.y & 0x3F3F3F3Fu, mn1 = h1.z & 0x3F3F3F3Fu;
        } else {
            sc0 = (h0.w & kNib) | ((h0.y >> 2) & 0x30303030u), mn0 = ((h0.w >> 4) & kNib) | ((h0.z >> 2) & 0x30303030u);
            sc1 = (h1.w & kNib) | ((h1.y >> 2) & 0x30303030u), mn1 = ((h1.w >> 4) & kNib) | ((h1.z >> 2) & 0x30303030u);
        }
        float s_0 = 0.f, s_1 = 0.f;
#pragma unroll
        for (int pp = 0; pp < 2; pp++) {  // sub-blocks s = 4u + 2pp (low nibbles) and s + 1 (high nibbles)
            const int s = 4 * u + 2 * pp;
            const uint32_t qo = (Q5 ? 48 : 16) + 16 * s + 8 * t;
            const uint2 w0 = lds64(r0 + qo), w1 = lds64(r1 + qo);
            uint32_t d[4];
            // Q4_K's high nibbles stay where they are (16·q: the lanes that scale them have the 1/16 in their final weight)
            auto lo = [&](uint32_t w, uint32_t e) { return Q5 ? (w & kNib) | ((s <= 4 ? e << (4 - s) : e >> (s - 4)) & 0x10101010u) : w & kNib; };
            auto hi = [&](uint32_t w, uint32_t e) {
                return Q5 ? ((w >> 4) & kNib) | ((s + 1 <= 4 ? e << (3 - s) : e >> (s - 3)) & 0x10101010u) : w & ~kNib;
            };
            mma_first<false>(d, lo(w0.x, e0.x), lo(w1.x, e1.x), hi(w0.x, e0.x), hi(w1.x, e1.x), b.lo[2 * pp], b.hi[2 * pp]);
            mma_next<false>(d, lo(w0.y, e0.y), lo(w1.y, e1.y), hi(w0.y, e0.y), hi(w1.y, e1.y), b.lo[2 * pp + 1], b.hi[2 * pp + 1]);
            s_0 = fmaf(magic_byte(sc0, 2 * pp + lv.sub) - kMagic, two_digits(d[0], d[1]), s_0);
            s_1 = fmaf(magic_byte(sc1, 2 * pp + lv.sub) - kMagic, two_digits(d[2], d[3]), s_1);
        }
        acc.a0 = fmaf(d0 * f, s_0, acc.a0);
        acc.a1 = fmaf(d1 * f, s_1, acc.a1);
        // mins: lane t charges sub-block t of the half
        m_0 = fmaf(magic_byte(mn0, t) - kMagic, sx, m_0);
        m_1 = fmaf(magic_byte(mn1, t) - kMagic, sx, m_1);
    }
    acc.m0 = fmaf(-half_bits(h0.x >> 16), m_0, acc.m0);
    acc.m1 = fmaf(-half_bits(h1.x >> 16), m_1, acc.m1);
}

__device__ __forceinline__ void consume_q6k(const unsigned char *box, uint32_t local, uint32_t blk, int g, int t, const LaneView &lv,
                                            const Smem &sm, BRegs &b, Acc &acc) {
    using S = Fmt<kQ6K>;
    const unsigned char *ql = box + g * S::kQlPitch + local * 128 + 4 * t;
    const unsigned char *qh = box + S::kQhOff + g * S::kQhPitch + local * 64 + 4 * t;
    const unsigned char *scp = box + S::kScOff + g * S::kScPitch + local * 16;
    const unsigned char *dp = box + S::kDOff + g * S::kDPitch + local * 2;
    const float d0 = half_at(dp), d1 = half_at(dp + 8 * S::kDPitch);
    constexpr float kM = kMagic + 128.f;
    float m_0 = 0.f, m_1 = 0.f;
#pragma unroll
    for (int u = 0; u < 2; u++) {
        b.load(lv.img + (blk * 2 + u) * kImgHalf, lv.is_lo);
        const float f = sm.f[blk * 2 + u];
        const uint2 sc0 = lds64(scp + 8 * u), sc1 = lds64(scp + 8 * u + 8 * S::kScPitch);
        // signed scales as unsigned ones: byte + 128
        const uint32_t c00 = sc0.x ^ 0x80808080u, c01 = sc0.y ^ 0x80808080u, c10 = sc1.x ^ 0x80808080u, c11 = sc1.y ^ 0x80808080u;
        const unsigned char *hp = qh + 32 * u;
        const uint32_t h00 = lds32(hp), h01 = lds32(hp + 16), h10 = lds32(hp + 8 * S::kQhPitch), h11 = lds32(hp + 8 * S::kQhPitch + 16);
        float s_0 = 0.f, s_1 = 0.f;
#pragma unroll
        for (int jb = 0; jb < 2; jb++) {  // columns 32·jb (low nibbles) and 32·jb + 64 (high nibbles), 16 from each of two groups
            const unsigned char *lp = ql + 64 * u + 32 * jb;
            const uint32_t w00 = lds32(lp), w01 = lds32(lp + 16), w10 = lds32(lp + 8 * S::kQlPitch), w11 = lds32(lp + 16 + 8 * S::kQlPitch);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int j = jb + 2 * c;
                auto six = [&](uint32_t w, uint32_t h) {
                    const uint32_t hb = j == 0 ? h << 4 : j == 1 ? h << 2 : j == 2 ? h : h >> 2;
                    return ((c ? w >> 4 : w) & kNib) | (hb & 0x30303030u);
                };
                uint32_t d[4];
                mma_first<false>(d, six(w00, h00), six(w10, h10), six(w01, h01), six(w11, h11), b.lo[j], b.hi[j]);
                const uint32_t n = 2 * (j & 1) + lv.sub;  // group within its four
                s_0 = fmaf(magic_byte(c ? c01 : c00, n) - kM, two_digits(d[0], d[1]), s_0);
                s_1 = fmaf(magic_byte(c ? c11 : c10, n) - kM, two_digits(d[2], d[3]), s_1);
            }
        }
        acc.a0 = fmaf(d0 * f, s_0, acc.a0);
        acc.a1 = fmaf(d1 * f, s_1, acc.a1);
        // −32 offset: lane t charges groups t and t + 4
        const float xa = sm.sx[(blk * 2 + u) * 8 + t], xb = sm.sx[(blk * 2 + u) * 8 + 4 + t];
        m_0 = fmaf(magic_byte(c00, t) - kM, xa, fmaf(magic_byte(c01, t) - kM, xb, m_0));
        m_1 = fmaf(magic_byte(c10, t) - kM, xa, fmaf(magic_byte(c11, t) - kM, xb, m_1));
    }
    acc.m0 = fmaf(d0, m_0, acc.m0);
    acc.m1 = fmaf(d1, m_1, acc.m1);
}

// Q8_0 and Q4_0: blocks of 32 weights start at even bytes; within 128 columns the alignment of their quants alternates
// (2, 0, 2, 0 mod 4).
template <bool Q8>
__device__ __forceinline__ void consume_q32(const unsigned char *r0, uint32_t blk, int t, const LaneView &lv, const Smem &sm, BRegs &b, Acc &acc) {
    using S = Fmt<Q8 ? kQ8 : kQ4>;
    constexpr uint32_t kB = Q8 ? 34 : 18;
#pragma unroll
    for (int u = 0; u < 2; u++, r0 += 4 * kB) {
        const unsigned char *r1 = r0 + 8 * S::kPitch;
        b.load(lv.img + (blk * 2 + u) * kImgHalf, lv.is_lo);
        const float f = sm.f[blk * 2 + u];
        float s_0 = 0.f, s_1 = 0.f;
#pragma unroll
        for (int pp = 0; pp < 2; pp++) {  // 32-weight blocks 2pp and 2pp + 1
            uint32_t d[4];
            if (Q8) {
                const unsigned char *p0 = r0 + 2 * kB * pp + 8 * t, *p1 = r1 + 2 * kB * pp + 8 * t;  // even one: quants at + 2
                const uint32_t x0 = lds32(p0), x1 = lds32(p0 + 4), x2 = lds32(p0 + 8), y0 = lds32(p1), y1 = lds32(p1 + 4), y2 = lds32(p1 + 8);
                const uint32_t z0 = lds32(p0 + kB + 2), z1 = lds32(p0 + kB + 6), w0 = lds32(p1 + kB + 2), w1 = lds32(p1 + kB + 6);
                mma_first<true>(d, __byte_perm(x0, x1, 0x5432), __byte_perm(y0, y1, 0x5432), z0, w0, b.lo[2 * pp], b.hi[2 * pp]);
                mma_next<true>(d, __byte_perm(x1, x2, 0x5432), __byte_perm(y1, y2, 0x5432), z1, w1, b.lo[2 * pp + 1], b.hi[2 * pp + 1]);
            } else {
                const unsigned char *p0 = r0 + 2 * kB * pp + 4 * t, *p1 = r1 + 2 * kB * pp + 4 * t;
                const uint32_t x = __byte_perm(lds32(p0), lds32(p0 + 4), 0x5432), y = __byte_perm(lds32(p1), lds32(p1 + 4), 0x5432);
                const uint32_t z = lds32(p0 + kB + 2), w = lds32(p1 + kB + 2);
                mma_first<false>(d, x & kNib, y & kNib, z & kNib, w & kNib, b.lo[2 * pp], b.hi[2 * pp]);
                mma_next<false>(d, (x >> 4) & kNib, (y >> 4) & kNib, (z >> 4) & kNib, (w >> 4) & kNib, b.lo[2 * pp + 1], b.hi[2 * pp + 1]);
            }
            const uint32_t s = 2 * pp + lv.sub;
            s_0 = fmaf(half_at(r0 + kB * s), two_digits(d[0], d[1]), s_0);
            s_1 = fmaf(half_at(r1 + kB * s), two_digits(d[2], d[3]), s_1);
        }
        acc.a0 = fmaf(f, s_0, acc.a0);
        acc.a1 = fmaf(f, s_1, acc.a1);
        if (!Q8) {  // −8 offset: lane t charges 32-weight block t
            const float sx = sm.sx[(blk * 2 + u) * 4 + t];
            acc.m0 = fmaf(half_at(r0 + kB * t), sx, acc.m0);
            acc.m1 = fmaf(half_at(r1 + kB * t), sx, acc.m1);
        }
    }
}

// Writes eight consecutive activations (columns c .. c + 7, already multiplied by the norm weights) into the image.
// Called by whole warps.
template <int F>
__device__ __forceinline__ void put8(const Smem &sm, uint32_t c, const float (&a)[8]) {
    constexpr uint32_t kLanes = Fmt<F>::kGroupCols / 8;  // threads per scale group; sixteen share 128 columns and an exponent
    float s = 0.f;
    uint32_t ab = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        ab = max(ab, __float_as_uint(a[i]) & 0x7FFFFFFFu);  // ordered like |x|; an infinity or NaN wins
        s += a[i];
    }
#pragma unroll
    for (uint32_t o = 1; o < 16; o <<= 1) {
        ab = max(ab, __shfl_xor_sync(0xffffffffu, ab, o));
        if (o < kLanes) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    const uint32_t eb = ab >> 23, el = eb < 30 ? 30 : eb;  // biased exponent of the largest |x|; below 2^-97 bits get lost that nobody can see
    const float scale = __uint_as_float((283u - el) << 23);  // 2^(29 − E), E = el − 127
    uint32_t m[8];  // signed base-256 digits of M, one per byte
#pragma unroll
    for (int i = 0; i < 8; i++) m[i] = ((uint32_t)__float2int_rn(a[i] * scale) + 0x80808080u) ^ 0x80808080u;
    // k order of the fragments: natural, Q4_0: even columns then odd ones
    constexpr bool kEvenOdd = F == kQ4;
    uint32_t w[4][2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int st = kEvenOdd ? 2 : 1, i0 = kEvenOdd ? q : 4 * q;
        const uint32_t t0 = __byte_perm(m[i0], m[i0 + st], 0x5140), t1 = __byte_perm(m[i0 + 2 * st], m[i0 + 3 * st], 0x5140);
        const uint32_t t2 = __byte_perm(m[i0], m[i0 + st], 0x7362), t3 = __byte_perm(m[i0 + 2 * st], m[i0 + 3 * st], 0x7362);
        w[0][q] = __byte_perm(t0, t1, 0x5410), w[1][q] = __byte_perm(t0, t1, 0x7632);
        w[2][q] = __byte_perm(t2, t3, 0x5410), w[3][q] = __byte_perm(t2, t3, 0x7632);
    }
    unsigned char *base = sm.img + (size_t)(c >> 7) * kImgHalf;
    if (F == kQ6K) {  // [group of the pair][digit][lane][32-column run]
        base += ((c >> 4) & 1u) * 256 + ((c >> 2) & 3u) * 16 + ((c >> 5) & 3u) * 4;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            *reinterpret_cast<uint32_t *>(base + j * 64) = w[j][0];
            *reinterpret_cast<uint32_t *>(base + j * 64 + 16) = w[j][1];
        }
    } else {  // [group of the pair][digit][lane][pair]
        base += ((c >> 5) & 1u) * 256 + ((c >> 3) & 3u) * 16 + ((c >> 6) & 1u) * 8;
#pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<uint2 *>(base + j * 64) = make_uint2(w[j][0], w[j][1]);
    }
    if ((threadIdx.x & (kLanes - 1)) == 0) sm.sx[c / Fmt<F>::kGroupCols] = (F == kQ6K ? -32.f : F == kQ4 ? -8.f : 1.f) * s;
    if ((threadIdx.x & 15) == 0) sm.f[c >> 7] = eb == 0xFF ? __uint_as_float(0x7FC00000u) : __uint_as_float((el - 29u) << 23);  // 2^(E − 29)
}

template <int F, bool TP, int W>
__global__ void __launch_bounds__(cta_threads(W), ctas_per_sm(W)) qmv_digits_kernel(const __grid_constant__ DigitsParams<F> p) {
    using S = Fmt<F>;
    constexpr int kBoxes = W / 8;  // boxes per stage
    constexpr uint32_t kStage = kStageBytes<F, W>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    yule_pdl_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool two = kBoxes == 2 && p.two_tiles != 0;
    const uint32_t bpr = p.n_cols / 256, chunk_blocks = two ? S::kBoxBlocks : kBoxes * S::kBoxBlocks, chunks = (bpr + chunk_blocks - 1) / chunk_blocks;
    const uint32_t nq = p.pair && !two ? 2 : 1;
    const uint32_t first = blockIdx.x, stride = gridDim.x;
    const uint32_t my_units = (p.n_units - first + stride - 1) / stride;  // the grid never exceeds the units
    const uint32_t slots = p.slots;
    const Smem sm = carve<F, W>(smem_raw, p.n_cols, slots, p.finish, nq);
    const uint32_t bar_full = smem_u32(sm.bars), bar_empty = bar_full + 8 * kMaxSlots;

    // Tile `half` of unit k (q: matrix of a pair whose tiles go one by one): its matrix and its number there.
    auto locate = [&](uint32_t k, uint32_t q, uint32_t half, uint32_t &seg) {
        uint32_t tile = first + k * stride;
        if (p.pair) {
            seg = two ? half : q;
            return tile;
        }
        if (two) tile = 2 * tile + half;
        seg = 0;
        while (seg + 1 < p.n_seg && tile >= p.seg_tiles[seg]) {
            tile -= p.seg_tiles[seg];
            seg++;
        }
        return tile;
    };
    // whether box `box` of a stage carries anything: the second tile of the last unit and the last blocks of a row may be missing
    auto box_live = [&](uint32_t k, uint32_t c, uint32_t box) {
        if (box == 0) return true;
        return two ? (p.pair || 2 * (first + k * stride) + 1 < p.n_tiles) : c * chunk_blocks + S::kBoxBlocks < bpr;
    };

    if (warp == W) {
        // ── the copying warp (one thread) ──
        if (lane == 0) {
            for (uint32_t i = 0; i < slots; i++) {
                mbar_init(bar_full + 8 * i, 1);
                mbar_init(bar_empty + 8 * i, W);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        uint32_t k = 0, q = 0, c = 0, slot = 0, phase = 0, n = 0, seg[2] = {0, 0}, row[2] = {0, 0};
        const uint32_t total = my_units * nq * chunks, ring_u32 = smem_u32(sm.ring);
        auto issue = [&]() {
            if (c == 0) {
                row[0] = locate(k, q, 0, seg[0]) * kTileRows;
                row[1] = row[0], seg[1] = seg[0];
                if (two && box_live(k, 0, 1)) row[1] = locate(k, q, 1, seg[1]) * kTileRows;
            }
            const uint32_t bar = bar_full + 8 * slot;
            const bool both = kBoxes == 2 && box_live(k, c, 1);
            mbar_arrive_expect_tx(bar, both ? kStage : S::kBoxBytes);
#pragma unroll
            for (int box = 0; box < kBoxes; box++) {
                if (box == 1 && !both) break;
                const uint32_t dst = ring_u32 + slot * kStage + box * S::kBoxBytes;
                const uint32_t blk = p.col0 / 256 + c * chunk_blocks + (two ? 0 : box * S::kBoxBlocks);
                auto copy = [&](int plane, uint32_t to, uint32_t x) {
                    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(to),
                                 "l"(reinterpret_cast<uint64_t>(&p.map[seg[box] * S::kPlanes + plane])), "r"(bar), "r"(x), "r"(row[box])
                                 : "memory");
                };
                if (F == kQ6K) {
                    copy(0, dst, blk * 16);
                    copy(1, dst + S::kQhOff, blk * 8);
                    copy(2, dst + S::kScOff, blk * 2);
                    copy(3, dst + S::kDOff, blk / 4);
                } else {
                    copy(0, dst, blk * (S::kBlockBytes / 8));
                    if (S::kCopies == 2) copy(0, dst + kTileRows * S::kPitch, (blk + S::kBoxBlocks / 2) * (S::kBlockBytes / 8));
                }
            }
            if (++c == chunks) {
                c = 0;
                if (++q == nq) {
                    q = 0;
                    k++;
                }
            }
            if (++slot == slots) {
                slot = 0;
                phase ^= 1u;
            }
            n++;
        };
        if (lane == 0)
            while (n < slots && n < total) issue();
        __syncthreads();
        if (lane == 0)
            while (n < total) {
                if (!ring_wait(bar_empty + 8 * slot, phase ^ 1u, p.status, p.wait_cycles)) break;
                issue();
            }
        return;
    }

    if (!p.late_wait) yule_pdl_wait();

    // ── x into the image ──
    {
        float ss = 0.f;
        const uint32_t pair_epoch = (TP && p.tp.wait) ? *p.tp.tick * p.tp.epochs_per_tick + p.tp.wait_index + 1u : 0u;
        auto load8 = [&](uint32_t c, float (&a)[8]) {
            if (TP && p.tp.wait) {
                tp_load8(p.tp.pair_in + c, pair_epoch, p.tp.status, p.tp.wait_cycles, a);
                return;
            }
            *reinterpret_cast<float4 *>(a) = *reinterpret_cast<const float4 *>(p.x + c);
            *reinterpret_cast<float4 *>(a + 4) = *reinterpret_cast<const float4 *>(p.x + c + 4);
        };
        for (uint32_t c = threadIdx.x * 8; c < p.n_cols; c += mul_threads(W) * 8) {  // n_cols is a multiple of 256: whole warps are in or out
            float a[8];
            load8(p.col0 + c, a);
            if (p.norm_w) {
                float w[8];
                *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(p.norm_w + p.col0 + c);
                *reinterpret_cast<float4 *>(w + 4) = *reinterpret_cast<const float4 *>(p.norm_w + p.col0 + c + 4);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    ss = fmaf(a[i], a[i], ss);
                    a[i] *= w[i];
                }
            }
            put8<F>(sm, c, a);
        }
        if (p.norm_w) {
            if (p.n_cols < p.full_cols)  // the columns of other launches count for the norm too
                for (uint32_t c = threadIdx.x * 8; c < p.full_cols; c += mul_threads(W) * 8)
                    if (c < p.col0 || c >= p.col0 + p.n_cols) {
                        float a[8];
                        load8(c, a);
#pragma unroll
                        for (int i = 0; i < 8; i++) ss = fmaf(a[i], a[i], ss);
                    }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (lane == 0) sm.red[warp] = ss;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float inv = 1.f;
        if (p.norm_w) {
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < W; i++) ss += sm.red[i];
            inv = 1.0f / sqrtf(ss / (float)p.full_cols + p.eps);  // as the CPU runner forms it (model_runner.rs:254-258)
        }
        *sm.inv = inv;  // read by finishing warps, behind a barrier that this warp passes first
    }

    const LaneView lv = {smem_u32(sm.img) + (g * 4 + t) * 16, g < 4 ? 1u : 0u, (uint32_t)t >> 1};
    const float weight = ((t & 1) ? 65536.f : 1.f) * (F == kQ4K && t >= 2 ? 0.0625f : 1.f);
    const uint32_t box = warp >> 3, local = warp & 7;  // this warp's box of a stage, its block there
    // row g of that block in slot 0 (Q6_K: the box)
    const unsigned char *r_base = sm.ring + box * S::kBoxBytes;
    if (F == kQ8) r_base += (local >> 2) * (kTileRows * S::kPitch) + g * S::kPitch + (local & 3) * S::kBlockBytes;
    else if (F != kQ6K) r_base += g * S::kPitch + local * S::kBlockBytes;
    BRegs b;
    bool dead = false;
    uint32_t slot = 0, phase = 0, buf = 0, bar_id = 1;
    for (uint32_t k = 0; k < my_units; k++) {
        float *part = sm.part + (size_t)(buf * nq) * (W * kTileRows);
        const bool mine = !two || box_live(k, 0, box);
        for (uint32_t q = 0; q < nq; q++) {
            Acc acc;
            uint32_t blk = two ? local : warp;
            for (uint32_t c = 0; c < chunks; c++, blk += chunk_blocks) {
                // A copy that never arrives: the lane waits for no other one and releases no slot (whose copy may still be on its way);
                // what the warp multiplies from here on means nothing.
                if (!dead) dead = !ring_wait(bar_full + 8 * slot, phase, p.status, p.wait_cycles);
                if (blk < bpr && mine) {
                    const unsigned char *r0 = r_base + slot * kStage;
                    if constexpr (F == kQ6K)
                        consume_q6k(r0, local, blk, g, t, lv, sm, b, acc);
                    else if constexpr (F == kQ4K || F == kQ5K)
                        consume_q4k<F == kQ5K>(r0, blk, t, lv, sm, b, acc);
                    else
                        consume_q32<F == kQ8>(r0, blk, t, lv, sm, b, acc);
                }
                __syncwarp();
                if (lane == 0 && !dead) mbar_arrive(bar_empty + 8 * slot);
                if (++slot == slots) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
            float v0 = fmaf(acc.a0, weight, acc.m0), v1 = fmaf(acc.a1, weight, acc.m1);
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
            v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
            v0 += __shfl_xor_sync(0xffffffffu, v0, 2);
            v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
            if (t == 0) {
                float *to = part + q * (W * kTileRows) + warp * kTileRows + g;
                to[0] = v0;
                to[8] = v1;
            }
        }
        // the sums of unit k are parked; its finishing warp adds them up and stores
        const bool finishes = (k & (W - 1)) == warp;
        // A warp that has given up keeps its place at the barriers, but the ring no longer holds it back: it waits for the others at
        // every unit, or it could arrive a second time at a barrier that a slower warp has yet to reach, whose phase would then be
        // over without that warp, and its wait never.  (For the same reason there is one barrier more than there are buffers: the
        // unit at which it gives up is one further on than the ring would have let it come.)
        dead = __any_sync(0xffffffffu, dead);
        if (finishes || dead)
            asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(mul_threads(W)) : "memory");
        else
            asm volatile("bar.arrive %0, %1;" ::"r"(bar_id), "n"(mul_threads(W)) : "memory");
        if (finishes) {
            const uint32_t rr = lane & 15, half = lane >> 4;  // half: of the warps (two tiles: those of box 0 or 1)
            auto collect = [&](uint32_t q) {
                const float *src = part + q * (W * kTileRows) + half * (W / 2 * kTileRows) + rr;
                float s = 0.f;  // fixed order over the warps: deterministic
#pragma unroll
                for (int w = 0; w < W / 2; w++) s += src[w * kTileRows];
                return s * *sm.inv;
            };
            float v = collect(0), other = __shfl_xor_sync(0xffffffffu, v, 16);
            if (!two) {
                v += other;
                if (p.pair) {
                    other = collect(1);
                    other += __shfl_xor_sync(0xffffffffu, other, 16);
                }
            }
            uint32_t seg = 0;
            const bool stores = two && !p.pair ? box_live(k, 0, half) : half == 0;  // one lane per row
            const uint32_t row = stores ? locate(k, 0, half, seg) * kTileRows + rr : 0;
            if (p.late_wait) yule_pdl_wait();  // everything the kernels before wrote is settled before the stores
            if (stores && row < p.seg_rows[seg]) {
                if (p.pair)
                    v = (v / (1.0f + expf(-v))) * other;  // silu_mul.cu
                else if (seg == 0 && p.residual)
                    v += p.residual[row];
                if (p.accumulate) v += p.out[seg][row];
                p.out[seg][row] = v;
                if (TP && p.tp.push && seg == 0) tp_push_value(p.tp, row, v);
            }
        }
        if (++buf == p.finish) buf = 0;
        if (++bar_id == p.finish + 2) bar_id = 1;
    }
    if (dead)  // copies of this CTA that are still on their way get time to land before its shared memory goes
        for (const long long t0 = clock64(); clock64() - t0 < 2000000LL;) {
        }
}

template <int F, bool TP, int W>
cudaError_t launch_variant(const DigitsParams<F> &p, uint32_t grid, size_t smem, bool pdl, cudaStream_t s) {
    auto kern = qmv_digits_kernel<F, TP, W>;
    static bool attr_done[64] = {};  // the opt-in for large dynamic shared memory belongs to the device
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !attr_done[dev]) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem(W == 8 ? 2 : 1));
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    return launch_kernel(kern, dim3(grid), dim3(cta_threads(W)), smem, s, pdl, p);
}

template <int F, int W>
cudaError_t launch_format(const QmvDigits &f, int sm_count, uint32_t share, cudaStream_t s, uint64_t *launches) {
    using S = Fmt<F>;
    DigitsParams<F> p = {};
    const uint32_t full_bpr = f.n_cols / 256;
    uint32_t n_tiles = 0;
    for (uint32_t i = 0; i < f.n_seg; i++) {
        cudaError_t e = cudaSuccess;
        if (F == kQ6K) {
            const uint64_t d_bytes = ((uint64_t)full_bpr * 2 + 15) & ~(uint64_t)15, rec = (uint64_t)full_bpr * 208 + d_bytes;
            const uint64_t off[4] = {0, (uint64_t)full_bpr * 128, (uint64_t)full_bpr * 192, (uint64_t)full_bpr * 208};
            const uint64_t len[4] = {(uint64_t)full_bpr * 128, (uint64_t)full_bpr * 64, (uint64_t)full_bpr * 16, d_bytes};
            const uint32_t pitch[4] = {S::kQlPitch, S::kQhPitch, S::kScPitch, S::kDPitch};
            for (int pl = 0; pl < 4 && e == cudaSuccess; pl++)
                e = cached_tensor_map_2d(f.w[i] + off[pl], 8, len[pl] / 8, f.rows[i], rec, pitch[pl] / 8, kTileRows, &p.map[(i * 4 + pl) % (3 * S::kPlanes)]);
        } else {
            const uint64_t row_bytes = (uint64_t)full_bpr * S::kBlockBytes;
            e = cached_tensor_map_2d(f.w[i], 8, row_bytes / 8, f.rows[i], row_bytes, S::kPitch / 8, kTileRows, &p.map[i]);
        }
        if (e != cudaSuccess) return e;
        p.out[i] = f.out[i];
        p.seg_rows[i] = f.rows[i];
        p.seg_tiles[i] = (f.rows[i] + kTileRows - 1) / kTileRows;
        if (!f.swiglu_pair || i == 0) n_tiles += p.seg_tiles[i];
    }
    if (n_tiles == 0) return cudaSuccess;
    p.n_seg = f.n_seg;
    p.n_tiles = n_tiles;
    p.pair = f.swiglu_pair ? 1 : 0;
    p.full_cols = f.n_cols;
    p.x = f.x;
    p.norm_w = f.norm_w;
    p.eps = f.eps;
    p.status = f.status;
    p.wait_cycles = f.wait_cycles;
    p.tp = f.tp;
    // Parts of the columns, in whole boxes of eight blocks: as few as leave room for two ring slots, of equal size (half-size CTAs: one part).
    const uint32_t units8 = (full_bpr + 7) / 8;
    uint32_t n_parts = 1;
    while (W == 16 && n_parts < units8 && 2 * (size_t)kStageBytes<F, W> + fixed_bytes<F, W>((units8 + n_parts - 1) / n_parts * 2048, 3, 2) > max_smem(share)) n_parts++;
    if (f.swiglu_pair && n_parts > 1) return cudaErrorInvalidValue;
    for (uint32_t part = 0, unit0 = 0; part < n_parts; part++) {
        const uint32_t unit1 = (uint32_t)((uint64_t)units8 * (part + 1) / n_parts);
        const uint32_t blk0 = unit0 * 8, blk1 = unit1 * 8 < full_bpr ? unit1 * 8 : full_bpr, bpr = blk1 - blk0;
        unit0 = unit1;
        p.col0 = blk0 * 256;
        p.n_cols = bpr * 256;
        // One tile per unit (sixteen blocks of a row per stage) or two (eight of each)?  The time of a CTA goes with its
        // number of stages; with few tiles two per unit would leave SMs without work.
        const uint32_t chunks1 = (bpr + W - 1) / W, chunks2 = (bpr + 7) / 8;
        const uint32_t units1 = n_tiles * (f.swiglu_pair ? 2 : 1), units2 = f.swiglu_pair ? n_tiles : (n_tiles + 1) / 2;
        const uint32_t ctas = (uint32_t)sm_count * share;
        auto rounds = [&](uint32_t units) { return (units + ctas - 1) / ctas; };
        const uint32_t rounds1 = f.swiglu_pair ? 2 * rounds(n_tiles) : rounds(units1);
        p.two_tiles = W == 16 && rounds(units2) * chunks2 < rounds1 * chunks1 ? 1u : 0u;
        p.n_units = p.two_tiles ? units2 : n_tiles;
        const uint32_t nq = f.swiglu_pair && !p.two_tiles ? 2 : 1, chunks = p.two_tiles ? chunks2 : chunks1;
        const uint32_t grid = p.n_units < ctas ? p.n_units : ctas;
        const uint32_t need = (p.n_units + grid - 1) / grid * nq * chunks;
        p.late_wait = f.pdl && f.late_wait ? 1u : 0u;  // (a part after the first reads the result of the one before, behind the wait)
        p.accumulate = part > 0 ? 1u : 0u;
        p.residual = part == 0 ? f.residual : nullptr;
        // Ring slots: what fits beside the image, no more than will be used.
        uint32_t slots = kMaxSlots, finish;
        size_t smem;
        for (;; slots--) {
            finish = 2 + (slots - 1 + nq * chunks - 1) / (nq * chunks);  // the finishing warp of a unit may lag behind a warp a whole ring ahead
            smem = (size_t)slots * kStageBytes<F, W> + fixed_bytes<F, W>(p.n_cols, finish, nq);
            if (slots == 1 || (finish <= kMaxFinish && slots <= need && smem <= max_smem(share))) break;
        }
        if (smem > max_smem(share)) return cudaErrorInvalidValue;
        p.slots = slots;
        p.finish = finish;
        p.tp.push = f.tp.push && part + 1 == n_parts;
        const bool tp = p.tp.push || f.tp.wait;
        const bool pdl = f.pdl || part > 0;  // a part reads its weights early, everything else after its wait
        cudaError_t e;
        if constexpr (F == kQ4K && W == 16)
            e = tp ? launch_variant<F, true, W>(p, grid, smem, pdl, s) : launch_variant<F, false, W>(p, grid, smem, pdl, s);
        else
            e = tp ? cudaErrorInvalidValue : launch_variant<F, false, W>(p, grid, smem, pdl, s);  // the exchange is built for Q4_K only
        if (e != cudaSuccess) return e;
        *launches += 1;
    }
    return cudaSuccess;
}

// A call whose inputs nothing before it writes overlaps with the calls before it, if an SM has room for CTAs of several: then the
// start of one, its image of x and its last sums run under the multiplying of the others.  So such calls take half-size CTAs, three
// to an SM where image and two ring slots fit a third of its shared memory, else two.  Not for rows of more than 8192 columns, whose
// image costs more than the overlap gives, and two to an SM not where a CTA has more than eight stages, which two slots do
// not keep fed.  us per independent call, 16-warp CTAs against these: Q4_K 2048x2048 2.26, 0.95, 5632x2048 3.29, 2.30, 14336x4096
// 9.1, 6.7, 28672x8192 23.3, 22.7; Q8_0 2048x2048 2.45, 1.14; two to an SM Q6_K 14336x4096 11.3, 9.5, Q8_0 4096x4096 4.5, 3.4;
// beyond the lines Q4_K 4096x14336 7.2, 8.6, Q5_K 28672x8192 27.7, 29.7.
//   In a chain of dependent launches nothing overlaps, yet over many rows of few columns, where a tile is a stage or two, three half-size CTAs keep an SM
// busier through the start and the end of a tile than one.  So they are taken from 30000 rows of up to 4096 columns on (a gate / up pair: 2048), for the two
// formats whose unpacking is shortest.  us per token, 16-warp CTAs, these, two layers and an output in Q4_K: 32000x2048 47.5, 47.1, 32000x4096 64.7, 63.1, 64000x4096
// 79.9, 74.2, 128256x4096 110.9, 98.5, 256000x3072 159.4, 126.3; 32768x8192 92.1, 93.9, 200064x5120 152.2, 159.5.  Eight layers with a gate / up pair of 30720x1024 205.1,
// 197.1, 49152x2048 295.9, 285.4; 32768x4096 326.2, 346.9, 30208x5120 389.3, 431.1, 32768x6144 419.6, 463.2.  Q4_0 alike.  28672x4096 in the 8B model
// 1563, 1650; the outputs of Q8_0 and Q6_K (32000x2048, 128256x4096) gain nothing.
template <int F>
cudaError_t launch_sized(const QmvDigits &f, int sm_count, cudaStream_t s, uint64_t *launches) {
    uint32_t all_rows = 0;
    for (uint32_t i = 0; i < f.n_seg; i++) all_rows += f.rows[i];
    const bool many_rows = all_rows >= 30000 && f.n_cols <= (f.swiglu_pair ? 2048u : 4096u) && (F == kQ4K || F == kQ4);
    if (f.pdl && (f.late_wait || many_rows) && f.n_cols <= 8192 && !f.tp.push && !f.tp.wait) {
        uint32_t n_tiles = 0;
        for (uint32_t i = 0; i < (f.swiglu_pair ? 1 : f.n_seg); i++) n_tiles += (f.rows[i] + kTileRows - 1) / kTileRows;
        const uint32_t nq = f.swiglu_pair ? 2 : 1;
        for (uint32_t share = 3; share > 1; share--) {
            const uint32_t ctas = (uint32_t)sm_count * share, stages = (n_tiles + ctas - 1) / ctas * nq * ((f.n_cols / 256 + 7) / 8);
            if (share == 2 && stages > 8) break;
            if ((stages > 1 ? 2 : 1) * (size_t)kStageBytes<F, 8> + fixed_bytes<F, 8>(f.n_cols, 3, nq) <= max_smem(share))
                return launch_format<F, 8>(f, sm_count, share, s, launches);
        }
    }
    return launch_format<F, 16>(f, sm_count, 1, s, launches);
}

}  // namespace

bool qmv_digits_supported(uint32_t type, const void *w, uint32_t n_cols) {
    switch (type) {
        case YULE_DTYPE_Q4_K: case YULE_DTYPE_Q5_K: case YULE_DTYPE_Q6_K: case YULE_DTYPE_Q8_0: case YULE_DTYPE_Q4_0: break;
        default: return false;
    }
    return n_cols != 0 && n_cols % 256 == 0 && w && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
}
bool qmv_digits_can_pair(uint32_t n_cols) { return n_cols <= 8192; }

cudaError_t launch_qmv_digits(const QmvDigits &f, int sm_count, cudaStream_t s, uint64_t *launches) {
    if (f.n_seg == 0 || f.n_seg > 3 || (reinterpret_cast<uintptr_t>(f.x) & 15)) return cudaErrorInvalidValue;
    if (f.swiglu_pair && (f.n_seg != 2 || !qmv_digits_can_pair(f.n_cols))) return cudaErrorInvalidValue;
    switch (f.type) {
        case YULE_DTYPE_Q4_K: return launch_sized<kQ4K>(f, sm_count, s, launches);
        case YULE_DTYPE_Q5_K: return launch_sized<kQ5K>(f, sm_count, s, launches);
        case YULE_DTYPE_Q6_K: return launch_sized<kQ6K>(f, sm_count, s, launches);
        case YULE_DTYPE_Q8_0: return launch_sized<kQ8>(f, sm_count, s, launches);
        case YULE_DTYPE_Q4_0: return launch_sized<kQ4>(f, sm_count, s, launches);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace yule
