// qmv_rows.cu — fused dequantise + matvec for several activation vectors (up to sixteen per pass over the weights), every
// tuned block format (Q4_K, Q5_K, Q6_K on its row-planar copy, Q8_0, Q4_0), with the neighbouring ops of a batched decode step
// folded in.
//
// Contract: yule-core/src/dequant.rs:902-1009 (and :297-338 for Q5_K) for each vector — per row the sum over scale groups
// of d·sc·Σ q·x minus the offset or min term.
//
// Arithmetic.  `mma.sync.m16n8k16` on fp16: A = 16 rows of quants as exact small integers (normal numbers: fed as subnormals, the
// cheapest way to make them, they cost seven bits of every product; relative error 1e-6 instead of 1e-7), the eight B columns
// are the hi and lo fp16 terms of four vectors (column 2v: hi of vector v, 2v + 1: lo; 22 bits of each x, every 256 columns
// of a vector with a power-of-two scale of their own).  A lane owns four consecutive quant bytes per MMA, receives hi and lo
// of one vector for two rows, adds the two and applies the group's scale in fp32.  Formats with a constant offset subtract it
// from the fp16 quants, exactly.  Q4_K and Q5_K: the middle of the quants is subtracted likewise, so that what the minimum takes
// away is not in the sums in the first place (error 2.6e-7 without that); two more MMAs per 256 columns, the mins and the scales
// times the sums of x over the sub-blocks, which enter as three fp16 terms (k slots 0-7: hi | lo, 8-15: the rest).
//
// What bounds it.  Per 512 weights and four vectors two MMAs of eight clocks per SM sub-partition, and about as many issue
// slots for unpacking and scaling: from eight vectors on the issue slots, below that HBM on the large matrices and the
// phases of a launch (start, image, meeting: 3 to 4 us) on the small ones.  A warp multiplies 32 rows at a time so that each B
// fragment read from shared memory serves two A fragments.
//
// Schedule.  The columns of a row are dealt over the CTAs of a cluster (and over warps inside a CTA), so that the digits of
// all vectors that a CTA needs are a small part of x: building them cost more than the multiplying when every CTA had
// whole rows, and rows of any length fit.  A warp multiplies (32 rows x 256 columns) units that it brings in itself, one
// tiled TMA copy per unit and plane into a ring of its own.  Row sums of the column shares meet through distributed shared
// memory, every CTA finishing a share of the rows, always in the same order.
//
// Folded in: RMSNorm of the vectors (the 1/rms factor multiplies the finished rows), up to three matrices that share x, SiLU(gate)·up
// of a pair, the residual.
//
// Measured (chain of dependent launches, before: two to four vectors per pass, or from thirteen the GEMM): Q4_K 8 vectors 4096x4096
// 17.4 -> 9.0 us, 14336x4096 32.8 -> 18.0, 4096x14336 62.7 -> 20.7; Q6_K 4096x14336 16 vectors 140 -> 38; Q8_0 128 -> 43.

#include <cuda.h>
#include <cuda_fp16.h>

#include <mutex>

#include "internal.h"

namespace yule {

namespace {

#include "ring_common.cuh"

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr uint32_t kMaxSlots = 3;     // ring slots of a warp
constexpr uint32_t kMaxCluster = 8;
constexpr uint32_t kMaxVecs = 16;
constexpr size_t kMaxSmem = 220 * 1024;

enum : int { kQ4K, kQ5K, kQ6K, kQ8, kQ4 };

template <int F>
struct Fmt {
    static constexpr uint32_t kBlockBytes = F == kQ4K ? 144 : F == kQ5K ? 176 : F == kQ8 ? 272 : F == kQ4 ? 144 : 0;  // of 256 columns
    static constexpr int kPlanes = F == kQ6K ? 4 : 1;
    // Q6_K planes of a unit of 32 rows: low nibbles (128-byte rows, 128-byte swizzle), high bit pairs (64-byte rows, 64-byte
    // swizzle), scales (16 bytes), d (the 16 bytes with those of eight blocks).  The raw formats need no swizzle: their row
    // pitches of 36, 44 and 68 words spread the eight rows of a fragment over all banks.
    static constexpr uint32_t kQhOff = 4096, kScOff = kQhOff + 2048, kDOff = kScOff + 512;
    static constexpr uint32_t kUnitBytes = F == kQ6K ? kDOff + 512 : 32 * kBlockBytes;
    static constexpr bool kMins = F == kQ4K || F == kQ5K;
    static_assert(kUnitBytes % (F == kQ6K ? 1024 : 128) == 0, "units keep the alignment of their copies");
};

template <int F>
struct RowsParams {
    CUtensorMap map[3 * Fmt<F>::kPlanes];
    float *out[3];
    uint32_t seg_rows[3], seg_tiles[3], out_stride[3];
    uint32_t n_seg, n_tiles, n_groups, pair;   // tiles: 32 rows of a matrix (pair: 16 of gate and 16 of up); groups: row_warps tiles
    uint32_t row_warps_log2, n_blocks;         // warps side by side over rows; 256-column blocks of a row
    const float *x, *norm_w, *residual;        // residual: segment 0
    uint32_t x_stride, nb;
    float eps;
    uint32_t slots, img_blocks, late_wait;
    int *status;
    long long wait_cycles;
};

// Shared memory: rings | image | min image | 2^-e | partial sums | Σx² | 1/rms | barriers
template <int NT>
constexpr uint32_t kImgBlock = 4096u * NT;   // bytes of 256 columns: [32-column group][four vectors][lane] x 16
template <int NT>
constexpr uint32_t kMinBlock = 256u * NT;
__host__ __device__ inline uint32_t part_pitch(uint32_t row_warps_log2) { return (32u << row_warps_log2) + 8; }
template <int F, int NT>
__host__ __device__ inline size_t smem_bytes(uint32_t slots, uint32_t img_blocks, uint32_t row_warps_log2) {
    return (size_t)kWarps * slots * Fmt<F>::kUnitBytes + (size_t)img_blocks * (kImgBlock<NT> + (Fmt<F>::kMins ? kMinBlock<NT> : 0) + 4 * NT * 4) +
           (size_t)(kWarps >> row_warps_log2) * 4 * NT * part_pitch(row_warps_log2) * 4 + kWarps * kMaxVecs * 4 + 2 * kMaxVecs * 4 +
           kWarps * kMaxSlots * 8 + 1024;
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16816_z(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ float half_bits(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
__device__ __forceinline__ float half_at(const unsigned char *p) { return half_bits(*reinterpret_cast<const unsigned short *>(p)); }
__device__ __forceinline__ uint32_t lds32(const unsigned char *p) { return *reinterpret_cast<const uint32_t *>(p); }
__device__ __forceinline__ uint4 lds128(const unsigned char *p) { return *reinterpret_cast<const uint4 *>(p); }
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
constexpr float kMagic = 8388608.f;
// byte `i` of w as a float
__device__ __forceinline__ float byte_f(uint32_t w, uint32_t i) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + i)) - kMagic; }
// (1024 + q) halves minus 1024 and the format's offset: exact
__device__ __forceinline__ uint32_t minus(uint32_t v, uint32_t c) {
    return h2_bits(__hsub2(*reinterpret_cast<const __half2 *>(&v), *reinterpret_cast<const __half2 *>(&c)));
}
constexpr uint32_t k1024 = 0x64006400u;

struct Img {
    const unsigned char *x;     // of the unit's block, at this lane
    const unsigned char *mins;  // same
    const float *f;             // 2^-e of the block's vectors, at this lane's vector of the first four
};

// Each of the consume routines adds one unit (32 rows x 256 columns) to the lane's sums: acc[half][nt][0 / 1] are rows
// 16·half + g and + 8 against vector 4·nt + t.
template <bool Q5, int NT>
__device__ __forceinline__ void consume_q4k(const unsigned char *u, int g, int t, const Img &im, float (&acc)[2][NT][2]) {
    constexpr uint32_t P = Q5 ? 176 : 144;
    float s[2][NT][2];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int n = 0; n < NT; n++) s[h][n][0] = s[h][n][1] = 0.f;
    const unsigned char *r = u + g * P;
    uint32_t sc[2][2][2];          // [half][row][lower / upper four sub-blocks]: 6-bit scales (dequant.rs:176-190)
    uint32_t dd[2][2], am[2][2];   // d and dmin; mins 2t, 2t + 1 as halves
    uint32_t q5[2][2][2];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            const uint4 hd = lds128(r + (16 * h + 8 * rr) * P);
            dd[h][rr] = hd.x;
            sc[h][rr][0] = hd.y & 0x3F3F3F3Fu;
            sc[h][rr][1] = (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u);
            const uint32_t mn = t < 2 ? hd.z & 0x3F3F3F3Fu : ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u);
            am[h][rr] = minus(__byte_perm(mn, 0x64u, (t & 1) ? 0x4342u : 0x4140u), k1024);
            if (Q5) q5[h][rr][0] = lds32(r + (16 * h + 8 * rr) * P + 16 + 4 * t), q5[h][rr][1] = lds32(r + (16 * h + 8 * rr) * P + 32 + 4 * t);
        }
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {  // 32 bytes: low nibbles sub-block 2jj, high nibbles 2jj + 1
        uint32_t w[2][2][2];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const unsigned char *p = r + (16 * h + 8 * rr) * P + (Q5 ? 48 : 16) + 32 * jj + 4 * t;
                w[h][rr][0] = lds32(p);
                w[h][rr][1] = lds32(p + 16);
            }
#pragma unroll
        for (int nib = 0; nib < 2; nib++) {
            const int sb = 2 * jj + nib;
            uint4 b[NT];
#pragma unroll
            for (int n = 0; n < NT; n++) b[n] = lds128(im.x + (sb * NT + n) * 512);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t a[2][4];  // [sixteen columns][register]
#pragma unroll
                for (int rr = 0; rr < 2; rr++)
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        const uint32_t v = w[h][rr][c];
                        if (Q5) {
                            // fifth bits: bit sb of byte l belongs to column l of the sub-block
                            const uint32_t e = q5[h][rr][c], q = ((nib ? v >> 4 : v) & 0x0F0F0F0Fu) | ((sb <= 4 ? e << (4 - sb) : e >> (sb - 4)) & 0x10101010u);
                            a[c][rr] = minus((q & 0x00FF00FFu) | k1024, 0x64106410u);  // 1040
                            a[c][2 + rr] = minus(((q >> 8) & 0x00FF00FFu) | k1024, 0x64106410u);
                        } else {
                            // 1024 + byte, and 1024 + 16·(high nibble) + 8: low − 8 is the difference, 16·(high − 8) the second minus 1160
                            const uint32_t b02 = __byte_perm(v, 0x64646464u, 0x4240u), b13 = __byte_perm(v, 0x64646464u, 0x4341u);
                            const uint32_t h02 = (b02 & 0xFFF0FFF0u) | 0x00080008u, h13 = (b13 & 0xFFF0FFF0u) | 0x00080008u;
                            a[c][rr] = nib ? minus(h02, 0x64886488u) : minus(b02, h02);
                            a[c][2 + rr] = nib ? minus(h13, 0x64886488u) : minus(b13, h13);
                        }
                    }
                const float up = nib && !Q5 ? 0.0625f : 1.f;
                const float s0 = byte_f(sc[h][0][sb >> 2], sb & 3) * up, s1 = byte_f(sc[h][1][sb >> 2], sb & 3) * up;
                float d[NT][4];
#pragma unroll
                for (int n = 0; n < NT; n++) mma16816_z(d[n], a[0][0], a[0][1], a[0][2], a[0][3], b[n].x, b[n].y);
#pragma unroll
                for (int n = 0; n < NT; n++) mma16816(d[n], a[1][0], a[1][1], a[1][2], a[1][3], b[n].z, b[n].w);
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    s[h][n][0] = fmaf(s0, d[n][0] + d[n][1], s[h][n][0]);
                    s[h][n][1] = fmaf(s1, d[n][2] + d[n][3], s[h][n][1]);
                }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const float d0 = half_bits(dd[h][0]), d1 = half_bits(dd[h][1]);
        // The sums of x went in with a factor 2^-5; with the scales they make up for the subtracted middle of the quants.
        const float m0 = half_bits(dd[h][0] >> 16) * -32.f, m1 = half_bits(dd[h][1] >> 16) * -32.f;
        const float c0 = d0 * (Q5 ? 512.f : 256.f), c1 = d1 * (Q5 ? 512.f : 256.f);
        uint32_t as[2];  // scales 2t, 2t + 1 as halves
#pragma unroll
        for (int rr = 0; rr < 2; rr++) as[rr] = minus(__byte_perm(t < 2 ? sc[h][rr][0] : sc[h][rr][1], 0x64u, (t & 1) ? 0x4342u : 0x4140u), k1024);
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const uint2 b = *reinterpret_cast<const uint2 *>(im.mins + n * 256);
            const float f = im.f[4 * n];
            float d[4], e[4];
            mma16816_z(d, am[h][0], am[h][1], am[h][0], am[h][1], b.x, b.y);
            mma16816_z(e, as[0], as[1], as[0], as[1], b.x, b.y);
            acc[h][n][0] = fmaf(f, fmaf(d0, s[h][n][0], fmaf(c0, e[0] + e[1], m0 * (d[0] + d[1]))), acc[h][n][0]);
            acc[h][n][1] = fmaf(f, fmaf(d1, s[h][n][1], fmaf(c1, e[2] + e[3], m1 * (d[2] + d[3]))), acc[h][n][1]);
        }
    }
}

template <int NT>
__device__ __forceinline__ void consume_q6k(const unsigned char *u, uint32_t blk, int g, int t, const Img &im, float (&acc)[2][NT][2]) {
    using S = Fmt<kQ6K>;
    float s[2][NT][2];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int n = 0; n < NT; n++) s[h][n][0] = s[h][n][1] = 0.f;
    uint4 sc[2][2];  // sixteen signed scales of a row, as byte + 128
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            sc[h][rr] = lds128(u + S::kScOff + (16 * h + 8 * rr + g) * 16);
            sc[h][rr].x ^= 0x80808080u, sc[h][rr].y ^= 0x80808080u, sc[h][rr].z ^= 0x80808080u, sc[h][rr].w ^= 0x80808080u;
        }
#pragma unroll
    for (int uu = 0; uu < 2; uu++) {  // halves of 128 columns
        uint32_t hb[2][2][2];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int rr = 0; rr < 2; rr++)
#pragma unroll
                for (int c = 0; c < 2; c++)
                    hb[h][rr][c] = lds32(u + S::kQhOff + (16 * h + 8 * rr + g) * 64 + (((2 * uu + c) ^ ((g >> 1) & 3)) << 4) + 4 * t);
#pragma unroll
        for (int jb = 0; jb < 2; jb++) {
            uint32_t w[2][2][2];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int rr = 0; rr < 2; rr++)
#pragma unroll
                    for (int c = 0; c < 2; c++)
                        w[h][rr][c] = lds32(u + (16 * h + 8 * rr + g) * 128 + (((4 * uu + 2 * jb + c) ^ g) << 4) + 4 * t);
#pragma unroll
            for (int nib = 0; nib < 2; nib++) {  // columns 32·jb (low nibbles) and 32·jb + 64 (high nibbles)
                const int j = jb + 2 * nib;
                uint4 b[NT];
#pragma unroll
                for (int n = 0; n < NT; n++) b[n] = lds128(im.x + ((4 * uu + j) * NT + n) * 512);
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int c = 0; c < 2; c++) {  // scale group 8·uu + 2·j + c
                        uint32_t a[4];
#pragma unroll
                        for (int rr = 0; rr < 2; rr++) {
                            const uint32_t e = hb[h][rr][c], v = w[h][rr][c];
                            const uint32_t eb = j == 0 ? e << 4 : j == 1 ? e << 2 : j == 2 ? e : e >> 2;
                            const uint32_t q = ((nib ? v >> 4 : v) & 0x0F0F0F0Fu) | (eb & 0x30303030u);
                            a[rr] = minus((q & 0x00FF00FFu) | k1024, 0x64206420u);  // 1056
                            a[2 + rr] = minus(((q >> 8) & 0x00FF00FFu) | k1024, 0x64206420u);
                        }
                        const int grp = 2 * j + c;
                        auto scale = [&](const uint4 &q) {
                            const uint32_t word = uu == 0 ? (grp < 4 ? q.x : q.y) : (grp < 4 ? q.z : q.w);
                            return byte_f(word, grp & 3) - 128.f;
                        };
                        const float s0 = scale(sc[h][0]), s1 = scale(sc[h][1]);
#pragma unroll
                        for (int n = 0; n < NT; n++) {
                            float d[4];
                            mma16816_z(d, a[0], a[1], a[2], a[3], c ? b[n].z : b[n].x, c ? b[n].w : b[n].y);
                            s[h][n][0] = fmaf(s0, d[0] + d[1], s[h][n][0]);
                            s[h][n][1] = fmaf(s1, d[2] + d[3], s[h][n][1]);
                        }
                    }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const unsigned char *dp = u + S::kDOff + (16 * h + g) * 16 + (blk & 7) * 2;
        const float d0 = half_at(dp), d1 = half_at(dp + 128);
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const float f = im.f[4 * n];
            acc[h][n][0] = fmaf(f * d0, s[h][n][0], acc[h][n][0]);
            acc[h][n][1] = fmaf(f * d1, s[h][n][1], acc[h][n][1]);
        }
    }
}

template <bool Q8, int NT>
__device__ __forceinline__ void consume_q32(const unsigned char *u, int g, int t, const Img &im, float (&acc)[2][NT][2]) {
    constexpr uint32_t P = Q8 ? 272 : 144, B = Q8 ? 34 : 18;
    float s[2][NT][2];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int n = 0; n < NT; n++) s[h][n][0] = s[h][n][1] = 0.f;
    const unsigned char *r = u + g * P;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint4 b[NT];
#pragma unroll
        for (int n = 0; n < NT; n++) b[n] = lds128(im.x + (i * NT + n) * 512);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            uint32_t a[2][4];
            float sc[2];
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                const unsigned char *p = r + (16 * h + 8 * rr) * P + B * i;
                sc[rr] = half_at(p);
                // the quants start two bytes into the block: on a word boundary in every other one
                auto word = [&](int at) { return (i & 1) ? lds32(p + 2 + at + 4 * t) : __byte_perm(lds32(p + at + 4 * t), lds32(p + at + 4 + 4 * t), 0x5432); };
                if (Q8) {
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        const uint32_t v = word(16 * c);  // signed byte ^ 128 = byte + 128; minus 1152
                        a[c][rr] = minus((v & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
                        a[c][2 + rr] = minus(((v >> 8) & 0x00FF00FFu) ^ 0x64806480u, 0x64806480u);
                    }
                } else {
                    const uint32_t v = word(0);  // low nibbles: even columns of the block, high ones: odd columns
#pragma unroll
                    for (int c = 0; c < 2; c++) {
                        a[c][rr] = minus(((v >> (4 * c)) & 0x000F000Fu) | k1024, 0x64086408u);
                        a[c][2 + rr] = minus(((v >> (8 + 4 * c)) & 0x000F000Fu) | k1024, 0x64086408u);
                    }
                }
            }
            float d[NT][4];
#pragma unroll
            for (int n = 0; n < NT; n++) mma16816_z(d[n], a[0][0], a[0][1], a[0][2], a[0][3], b[n].x, b[n].y);
#pragma unroll
            for (int n = 0; n < NT; n++) mma16816(d[n], a[1][0], a[1][1], a[1][2], a[1][3], b[n].z, b[n].w);
#pragma unroll
            for (int n = 0; n < NT; n++) {
                s[h][n][0] = fmaf(sc[0], d[n][0] + d[n][1], s[h][n][0]);
                s[h][n][1] = fmaf(sc[1], d[n][2] + d[n][3], s[h][n][1]);
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NT; n++) {
        const float f = im.f[4 * n];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            acc[h][n][0] = fmaf(f, s[h][n][0], acc[h][n][0]);
            acc[h][n][1] = fmaf(f, s[h][n][1], acc[h][n][1]);
        }
    }
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}

template <int F, int NT>
__global__ void __launch_bounds__(kThreads, 1) qmv_rows_kernel(const __grid_constant__ RowsParams<F> p) {
    using S = Fmt<F>;
    constexpr uint32_t V = 4 * NT;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    yule_pdl_launch_dependents();
    uint32_t n_ranks, rank;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n_ranks));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const uint32_t ranks_log2 = 31u - __clz(n_ranks);
    const uint32_t cluster = blockIdx.x >> ranks_log2, n_clusters = gridDim.x >> ranks_log2;
    const uint32_t warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t rwl = p.row_warps_log2, row_warps = 1u << rwl, col_warps = kWarps >> rwl;
    const uint32_t rw = warp & (row_warps - 1), kw = warp >> rwl;
    const uint32_t b0 = p.n_blocks * rank >> ranks_log2, b1 = p.n_blocks * (rank + 1) >> ranks_log2, nblk = b1 - b0;  // this CTA's columns

    // 128-byte swizzle wants 1024-byte boundaries: rounded up, smem_bytes() has the room
    unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char *ring = base + (size_t)warp * p.slots * S::kUnitBytes;
    unsigned char *img = base + (size_t)kWarps * p.slots * S::kUnitBytes;
    unsigned char *mins = img + (size_t)p.img_blocks * kImgBlock<NT>;
    float *fx = reinterpret_cast<float *>(mins + (S::kMins ? (size_t)p.img_blocks * kMinBlock<NT> : 0));
    float *part = fx + p.img_blocks * V;
    const uint32_t pitch = part_pitch(rwl);
    float *ssq = part + col_warps * V * pitch;             // [warp][vector]
    float *ssum = ssq + kWarps * kMaxVecs;                 // Σx² of this CTA's columns
    float *inv = ssum + kMaxVecs;
    uint64_t *bars = reinterpret_cast<uint64_t *>(inv + kMaxVecs) + warp * kMaxSlots;

    // The 16 rows `half` of a tile: matrix and first row.
    auto locate = [&](uint32_t tile, uint32_t half, uint32_t &row0) {
        if (p.pair) {
            row0 = tile * 16;
            return half;
        }
        uint32_t seg = 0;
        while (seg + 1 < p.n_seg && tile >= p.seg_tiles[seg]) tile -= p.seg_tiles[seg++];
        row0 = tile * 32 + 16 * half;
        return seg;
    };

    // ── this warp's copies: units in the order in which it multiplies them ──
    const uint32_t full = smem_u32(bars), ring_u32 = smem_u32(ring);
    uint32_t ig = cluster, ib = kw, islot = 0;  // next unit to bring in: group, block
    auto issue = [&]() {  // one thread
        const uint32_t tile = ig * row_warps + rw;
        if (ig >= p.n_groups || tile >= p.n_tiles || ib >= nblk) return;  // (only the last group has missing tiles)
        const uint32_t bar = full + 8 * islot, dst = ring_u32 + islot * S::kUnitBytes, blk = b0 + ib;
        mbar_arrive_expect_tx(bar, S::kUnitBytes);
        const uint32_t copies = p.pair ? 2 : 1, rows = p.pair ? 16 : 32;
        for (uint32_t c = 0; c < copies; c++) {
            uint32_t row0;
            const uint32_t seg = locate(tile, c, row0);
            auto copy = [&](int plane, uint32_t to, uint32_t x) {
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(to),
                             "l"(reinterpret_cast<uint64_t>(&p.map[seg * S::kPlanes + plane])), "r"(bar), "r"(x), "r"(row0)
                             : "memory");
            };
            if (F == kQ6K) {
                copy(0, dst + c * rows * 128, blk * 16);
                copy(1, dst + S::kQhOff + c * rows * 64, blk * 8);
                copy(2, dst + S::kScOff + c * rows * 16, blk * 2);
                copy(3, dst + S::kDOff + c * rows * 16, (blk / 8) * 2);
            } else {
                copy(0, dst + c * rows * S::kBlockBytes, blk * (S::kBlockBytes / 8));
            }
        }
        if (++islot == p.slots) islot = 0;
        ib += col_warps;
        if (ib >= nblk) ib = kw, ig += n_clusters;
    };
    if (lane == 0) {
        for (uint32_t i = 0; i < p.slots; i++) mbar_init(full + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (uint32_t i = 0; i < p.slots; i++) issue();
    }
    __syncwarp();

    if (!p.late_wait) yule_pdl_wait();

    // ── image of the vectors over blocks [f0, f1) of this CTA's: a warp takes (block, vector) pairs ──
    auto convert = [&](uint32_t f0, uint32_t li, uint32_t v, float4 (&a)[2], bool sums) {
        float sq = 0.f;
        if (p.norm_w) {
            const float *nw = p.norm_w + (b0 + f0 + li) * 256 + lane * 4;
            const float4 w0 = *reinterpret_cast<const float4 *>(nw), w1 = *reinterpret_cast<const float4 *>(nw + 128);
#pragma unroll
            for (int i = 0; i < 2; i++) sq = fmaf(a[i].x, a[i].x, fmaf(a[i].y, a[i].y, fmaf(a[i].z, a[i].z, fmaf(a[i].w, a[i].w, sq))));
            a[0].x *= w0.x, a[0].y *= w0.y, a[0].z *= w0.z, a[0].w *= w0.w;
            a[1].x *= w1.x, a[1].y *= w1.y, a[1].z *= w1.z, a[1].w *= w1.w;
        }
        uint32_t mx = 0;  // ordered like |x|; an infinity or NaN wins
#pragma unroll
        for (int i = 0; i < 2; i++) {
            mx = max(max(mx, __float_as_uint(a[i].x) & 0x7FFFFFFFu), __float_as_uint(a[i].y) & 0x7FFFFFFFu);
            mx = max(max(mx, __float_as_uint(a[i].z) & 0x7FFFFFFFu), __float_as_uint(a[i].w) & 0x7FFFFFFFu);
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        // 2^e with max|x|·2^e in [2^13, 2^14); both 2^e and 2^-e stay finite normals
        int eb = (int)(mx >> 23);
        if (mx == 0u || eb == 0xFF) eb = 127 + 13;
        int se = 127 + 13 - (eb - 127);
        se = se < 1 ? 1 : (se > 253 ? 253 : se);
        const float sc = __uint_as_float((uint32_t)se << 23);
        const uint32_t nt = v >> 2, n = 2 * (v & 3);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            a[i].x *= sc, a[i].y *= sc, a[i].z *= sc, a[i].w *= sc;  // exact
            const __half2 h02 = __floats2half2_rn(a[i].x, a[i].z), h13 = __floats2half2_rn(a[i].y, a[i].w);
            const float2 c02 = __half22float2(h02), c13 = __half22float2(h13);
            uint2 hi = make_uint2(h2_bits(h02), h2_bits(h13));
            uint2 lo = make_uint2(h2_bits(__floats2half2_rn(a[i].x - c02.x, a[i].z - c02.y)), h2_bits(__floats2half2_rn(a[i].y - c13.x, a[i].w - c13.y)));
            const uint32_t s = 4 * i + ((uint32_t)lane >> 3);
            unsigned char *dst = img + (size_t)li * kImgBlock<NT> + (s * NT + nt) * 512 + n * 64;
            if (F == kQ4) {
                // byte 4t + b of a block holds columns 8t + 2b (low nibble) and 8t + 2b + 1: the even columns make the first
                // sixteen k, the odd ones the second; two lanes swap what the other one stores
                const bool odd = lane & 1;
                auto deal = [&](uint2 w) {
                    const uint32_t mine = odd ? w.y : w.x, other = __shfl_xor_sync(0xffffffffu, odd ? w.x : w.y, 1);
                    const uint32_t first = odd ? other : mine, second = odd ? mine : other;
                    return make_uint2(__byte_perm(first, second, 0x5410), __byte_perm(first, second, 0x7632));
                };
                hi = deal(hi), lo = deal(lo);
                dst += (((uint32_t)lane & 7u) >> 1) * 16 + (lane & 1) * 8;
            } else {  // columns 32·s + 16·h + 4·t + {0, 2} and {1, 3}
                dst += (lane & 3) * 16 + (((uint32_t)lane >> 2) & 1u) * 8;
            }
            *reinterpret_cast<uint2 *>(dst) = hi;
            *reinterpret_cast<uint2 *>(dst + 64) = lo;
            if (S::kMins) {
                float sx = (a[i].x + a[i].y) + (a[i].z + a[i].w);
                sx += __shfl_xor_sync(0xffffffffu, sx, 1);
                sx += __shfl_xor_sync(0xffffffffu, sx, 2);
                sx += __shfl_xor_sync(0xffffffffu, sx, 4);
                if ((lane & 7) == 0) {
                    sx *= 0.03125f;  // 32 values of up to 2^14: inside fp16's range
                    const __half first = __float2half_rn(sx);
                    const float r1 = sx - __half2float(first);
                    const __half second = __float2half_rn(r1);
                    unsigned char *to = mins + (size_t)li * kMinBlock<NT> + nt * 256 + (n * 4 + (s >> 1)) * 8 + (s & 1) * 2;
                    *reinterpret_cast<__half *>(to) = first;
                    *reinterpret_cast<__half *>(to + 4) = __float2half_rn(r1 - __half2float(second));
                    *reinterpret_cast<__half *>(to + 32) = second;
                    *reinterpret_cast<__half *>(to + 36) = __ushort_as_half(0);
                }
            }
        }
        if (lane == 0) fx[li * V + v] = __uint_as_float((uint32_t)(254 - se) << 23);
        if (sums && p.norm_w) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
            if (lane == 0) ssq[warp * kMaxVecs + v] += sq;
        }
    };
    auto build = [&](uint32_t f0, uint32_t f1, bool sums) {
        constexpr int kAhead = 4;  // pairs whose loads are in flight together
        const uint32_t n_pairs = (f1 - f0) * V;
        for (uint32_t k0 = warp; k0 < n_pairs; k0 += kWarps * kAhead) {
            float4 xin[kAhead][2];
#pragma unroll
            for (int j = 0; j < kAhead; j++) {
                const uint32_t k = k0 + j * kWarps, v = k % V;
                xin[j][0] = xin[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k < n_pairs && v < p.nb) {
                    const float *xv = p.x + (size_t)v * p.x_stride + (b0 + f0 + k / V) * 256 + lane * 4;
                    xin[j][0] = *reinterpret_cast<const float4 *>(xv);
                    xin[j][1] = *reinterpret_cast<const float4 *>(xv + 128);
                }
            }
#pragma unroll
            for (int j = 0; j < kAhead; j++) {
                const uint32_t k = k0 + j * kWarps;
                if (k >= n_pairs) break;
                convert(f0, k / V, k % V, xin[j], sums);
            }
        }
    };
    for (uint32_t i = threadIdx.x; i < kWarps * kMaxVecs; i += kThreads) ssq[i] = 0.f;
    const bool whole = nblk <= p.img_blocks;
    __syncthreads();
    if (whole) {
        build(0, nblk, true);
        __syncthreads();
    }

    bool dead = false, pending_read = false, settled = !p.late_wait;
    uint32_t slot = 0, phase = 0;
    for (uint32_t grp = cluster; grp < p.n_groups; grp += n_clusters) {
        float acc[2][NT][2];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int n = 0; n < NT; n++) acc[h][n][0] = acc[h][n][1] = 0.f;
        const bool live = grp * row_warps + rw < p.n_tiles;
        for (uint32_t f0 = 0; f0 < nblk; f0 += p.img_blocks) {  // img_blocks is a multiple of col_warps, or holds everything
            const uint32_t f1 = f0 + p.img_blocks < nblk ? f0 + p.img_blocks : nblk;
            if (!whole) {
                __syncthreads();  // the part of x before is done with
                build(f0, f1, grp == cluster);
                __syncthreads();
            }
            for (uint32_t i = f0 + kw; live && i < f1; i += col_warps) {
                // A copy that never arrives: the warp stops multiplying but keeps its place at the barriers, so that nobody hangs.
                if (!dead) dead = !ring_wait(full + 8 * slot, phase, p.status, p.wait_cycles);
                if (!dead) {
                    const unsigned char *u = ring + slot * S::kUnitBytes;
                    Img im;
                    im.x = img + (size_t)(i - f0) * kImgBlock<NT> + lane * 16;
                    im.mins = mins + (size_t)(i - f0) * kMinBlock<NT> + lane * 8;
                    im.f = fx + (i - f0) * V + t;
                    if constexpr (F == kQ6K)
                        consume_q6k<NT>(u, b0 + i, g, t, im, acc);
                    else if constexpr (F == kQ4K || F == kQ5K)
                        consume_q4k<F == kQ5K, NT>(u, g, t, im, acc);
                    else
                        consume_q32<F == kQ8, NT>(u, g, t, im, acc);
                    __syncwarp();
                    if (lane == 0) issue();
                }
                if (++slot == p.slots) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
        }
        // ── the column shares meet ──
        if (pending_read) cluster_wait();  // everybody has read the sums of the group before
#pragma unroll
        for (int n = 0; n < NT; n++) {
            float *to = part + (size_t)(kw * V + 4 * n + t) * pitch + rw * 32 + g;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                to[16 * h] = acc[h][n][0];
                to[16 * h + 8] = acc[h][n][1];
            }
        }
        if (grp == cluster && threadIdx.x < kMaxVecs && p.norm_w) {
            // (every warp's sums of squares lie before the barrier behind build())
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; w++) s += ssq[w * kMaxVecs + threadIdx.x];
            ssum[threadIdx.x] = s;
        }
        cluster_arrive();
        cluster_wait();
        if (grp == cluster) {
            if (threadIdx.x < kMaxVecs) {
                float v = 1.f;
                if (p.norm_w) {
                    float s = 0.f;
                    for (uint32_t c = 0; c < n_ranks; c++) s += ld_cluster(map_rank(smem_u32(ssum + threadIdx.x), c));
                    v = 1.0f / sqrtf(s / (float)(p.n_blocks * 256) + p.eps);  // as the CPU runner forms it (model_runner.rs:254-258)
                }
                inv[threadIdx.x] = v;
            }
            __syncthreads();
        }
        if (!settled) {  // everything the kernels before wrote is settled before the stores
            yule_pdl_wait();
            settled = true;
        }
        // This CTA finishes a share of the group's rows (pair: of the rows of its products).
        const uint32_t rows_log2 = (p.pair ? 4u : 5u) + rwl - ranks_log2, rows_cta = 1u << rows_log2, row_lo = rank << rows_log2;
        for (uint32_t k = threadIdx.x; k < rows_cta * p.nb; k += kThreads) {
            const uint32_t v = k >> rows_log2, lr = row_lo + (k & (rows_cta - 1));
            const uint32_t trw = p.pair ? lr >> 4 : lr >> 5, in = p.pair ? lr & 15 : lr & 31, tile = grp * row_warps + trw;
            uint32_t row0;
            const uint32_t seg = p.pair ? (locate(tile, 0, row0), 0u) : locate(tile, 0, row0);
            const uint32_t row = row0 + in;
            if (tile >= p.n_tiles || row >= p.seg_rows[seg]) continue;
            const uint32_t at = smem_u32(part + (size_t)v * pitch + trw * 32 + in), share = V * pitch * 4;
            // The shares of all ranks and column warps, four loads in flight at a time, added in a fixed order.
            auto collect = [&](uint32_t off) {
                const uint32_t n = n_ranks << (4 - rwl);
                float sum = 0.f;
                for (uint32_t i = 0; i < n; i += 4) {
                    float w[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) w[j] = i + j < n ? ld_cluster(map_rank(at, (i + j) & (n_ranks - 1)) + off + ((i + j) >> ranks_log2) * share) : 0.f;
                    sum += (w[0] + w[1]) + (w[2] + w[3]);
                }
                return sum;
            };
            float a = collect(0) * inv[v];
            if (p.pair) {
                const float b = collect(64) * inv[v];
                a = (a / (1.0f + expf(-a))) * b;  // silu_mul.cu
            } else if (seg == 0 && p.residual) {
                a += p.residual[(size_t)v * p.out_stride[0] + row];
            }
            p.out[seg][(size_t)v * p.out_stride[seg] + row] = a;
        }
        cluster_arrive();
        pending_read = true;
    }
    if (pending_read) cluster_wait();  // nobody leaves while its sums may still be read
    if (dead)  // copies of this CTA that are still on their way get time to land before its shared memory goes
        for (const long long t0 = clock64(); clock64() - t0 < 2000000LL;) {
        }
}

// How many clusters of a size are resident at once (they have to find their SMs in one GPC), asked once per device.
template <int F, int NT>
cudaError_t resident_clusters(uint32_t size_log2, uint32_t *out) {
    auto kern = qmv_rows_kernel<F, NT>;
    static std::mutex mu;
    static uint32_t known[64][4] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (!known[dev][0]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
        if (e != cudaSuccess) return e;
        uint32_t k[4];
        for (int i = 0; i < 4; i++) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(8);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kMaxSmem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 1u << i;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
            if (e != cudaSuccess) return e;
            k[i] = n < 1 ? 1u : (uint32_t)n;
        }
        for (int i = 0; i < 4; i++) known[dev][i] = k[i];
    }
    *out = known[dev][size_log2];
    return cudaSuccess;
}

template <int F, int NT>
cudaError_t launch_pass(const QmvRows &f, uint32_t v0, uint32_t nb, cudaStream_t s, bool pdl, bool late_wait, uint64_t *launches) {
    using S = Fmt<F>;
    RowsParams<F> p = {};
    const uint32_t bpr = f.n_cols / 256, box_rows = f.swiglu_pair ? 16 : 32;
    uint32_t n_tiles = 0;
    for (uint32_t i = 0; i < f.n_seg; i++) {
        cudaError_t e = cudaSuccess;
        if (F == kQ6K) {
            const uint64_t d_bytes = ((uint64_t)bpr * 2 + 15) & ~(uint64_t)15, rec = (uint64_t)bpr * 208 + d_bytes;
            const uint64_t off[4] = {0, (uint64_t)bpr * 128, (uint64_t)bpr * 192, (uint64_t)bpr * 208};
            const uint64_t len[4] = {(uint64_t)bpr * 128, (uint64_t)bpr * 64, (uint64_t)bpr * 16, d_bytes};
            const uint32_t box[4] = {128, 64, 16, 16}, swizzle[4] = {128, 64, 0, 0};
            for (int pl = 0; pl < 4 && e == cudaSuccess; pl++)
                e = cached_tensor_map_2d(f.w[i] + off[pl], 8, len[pl] / 8, f.rows[i], rec, box[pl] / 8, box_rows, &p.map[(i * 4 + pl) % (3 * S::kPlanes)], swizzle[pl]);
        } else {
            const uint64_t row_bytes = (uint64_t)bpr * S::kBlockBytes;
            e = cached_tensor_map_2d(f.w[i], 8, row_bytes / 8, f.rows[i], row_bytes, S::kBlockBytes / 8, box_rows, &p.map[i]);
        }
        if (e != cudaSuccess) return e;
        p.out[i] = f.out[i] + (size_t)v0 * f.out_stride[i];
        p.out_stride[i] = f.out_stride[i];
        p.seg_rows[i] = f.rows[i];
        p.seg_tiles[i] = (f.rows[i] + box_rows - 1) / box_rows;
        if (!f.swiglu_pair || i == 0) n_tiles += p.seg_tiles[i];
    }
    if (n_tiles == 0) return cudaSuccess;
    p.n_seg = f.n_seg;
    p.n_tiles = n_tiles;
    p.pair = f.swiglu_pair ? 1 : 0;
    p.n_blocks = bpr;
    p.x = f.x + (size_t)v0 * f.x_stride;
    p.x_stride = f.x_stride;
    p.nb = nb;
    p.norm_w = f.norm_w;
    p.eps = f.eps;
    p.residual = f.residual ? f.residual + (size_t)v0 * f.out_stride[0] : nullptr;
    p.late_wait = late_wait ? 1u : 0u;
    p.status = f.status;
    p.wait_cycles = f.wait_cycles;

    // Cluster size, and how many warps stand side by side over rows: the choice with the least estimated time, in clocks of this
    // kernel's phases as measured (Q4_K; the other formats keep the proportions).  Units of a CTA cost kUnit each, a warp's own
    // units one after the other at least kAlone each; a group's meeting costs kMeet, and kAdd per output of a thread and four
    // shares; the image kImage per (block, vector) pair of a warp.  Against counting rounds of units alone: 8 vectors
    // 2048x2048 7.5 -> 5.9 us, 14336x4096 19.1 -> 18.0.
    constexpr uint32_t kUnit = 220 + 70 * NT, kAlone = 1100 + 250 * NT, kMeet = 2500, kAdd = 350, kImage = 250;
    uint32_t best = ~0u, best_size = 0, best_rwl = 0, best_clusters = 0, best_slots = 0, best_img = 0;
    for (uint32_t sl = 4; sl-- > 0;) {
        const uint32_t size = 1u << sl;
        if (size > kMaxCluster || size > bpr) continue;
        uint32_t resident = 0;
        cudaError_t e = resident_clusters<F, NT>(sl, &resident);
        if (e != cudaSuccess) return e;
        const uint32_t nblk = (bpr + size - 1) / size;
        for (uint32_t rwl = 4; rwl >= 1; rwl--) {
            const uint32_t row_warps = 1u << rwl, col_warps = kWarps >> rwl;
            if ((box_rows << rwl) < size * 4) continue;
            // ring slots and blocks of the image that fit: everything with as many slots as it leaves, or a part with one
            uint32_t slots = kMaxSlots, img = nblk;
            const uint32_t rounds = (nblk + col_warps - 1) / col_warps;
            while (slots > 1 && smem_bytes<F, NT>(slots, img, rwl) > kMaxSmem) slots--;
            if (smem_bytes<F, NT>(slots, img, rwl) > kMaxSmem) {
                img = col_warps;
                if (smem_bytes<F, NT>(1, img, rwl) > kMaxSmem) continue;
                while (smem_bytes<F, NT>(1, img + col_warps, rwl) <= kMaxSmem) img += col_warps;
            }
            const uint32_t groups = (n_tiles + row_warps - 1) / row_warps, clusters = groups < resident ? groups : resident;
            const uint32_t per = (groups + clusters - 1) / clusters;
            const uint32_t units = row_warps * nblk, group_clocks = units * kUnit > rounds * kAlone ? units * kUnit : rounds * kAlone;
            const uint32_t outputs = ((box_rows << rwl) / size * nb + kThreads - 1) / kThreads, shares = (size * col_warps + 3) / 4;
            const uint32_t image = (nblk * 4 * NT + kWarps - 1) / kWarps * kImage + (nblk + img - 1) / img * 1000;
            const uint32_t cost = per * (group_clocks + kMeet + outputs * shares * kAdd) + (img < nblk ? per : 1) * image;
            if (cost < best) best = cost, best_size = size, best_rwl = rwl, best_clusters = clusters, best_slots = slots, best_img = img;
        }
    }
    if (best == ~0u) return cudaErrorInvalidValue;
    p.row_warps_log2 = best_rwl;
    p.n_groups = (n_tiles + (1u << best_rwl) - 1) >> best_rwl;
    p.slots = best_slots;
    p.img_blocks = best_img;

    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(best_clusters * best_size);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes<F, NT>(best_slots, best_img, best_rwl);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = best_size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, qmv_rows_kernel<F, NT>, p);
    if (e != cudaSuccess) return e;
    *launches += 1;
    return cudaSuccess;
}

template <int F>
cudaError_t launch_format(const QmvRows &f, cudaStream_t s, uint64_t *launches) {
    // passes of up to sixteen vectors, as equal as they come in fours
    const uint32_t n_pass = (f.batch + kMaxVecs - 1) / kMaxVecs, fours = (f.batch + 3) / 4, per = (fours + n_pass - 1) / n_pass * 4;
    for (uint32_t v = 0; v < f.batch; v += per) {
        const uint32_t nb = f.batch - v < per ? f.batch - v : per;
        const bool pdl = f.pdl || v > 0, late = f.pdl && f.late_wait && v == 0;  // a later pass reads its weights early, the rest after its wait
        cudaError_t e;
        switch ((nb + 3) / 4) {
            case 1: e = launch_pass<F, 1>(f, v, nb, s, pdl, late, launches); break;
            case 2: e = launch_pass<F, 2>(f, v, nb, s, pdl, late, launches); break;
            case 3: e = launch_pass<F, 3>(f, v, nb, s, pdl, late, launches); break;
            default: e = launch_pass<F, 4>(f, v, nb, s, pdl, late, launches); break;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

// Measured per launch, this kernel against the other matvecs.  Two to four vectors: the kernels for so few read rows of up to 4096 columns
// whole and overlap independent calls (Q4_K 2048x2048, 4 vectors: 2.8 against 4.0 us), longer ones take several launches there (8192x8192
// 29 against 17 us).  More vectors take several launches there, or run without the tensor pipe.
bool qmv_rows_over_matvecs(uint32_t type, uint64_t n_rows, uint32_t n_cols, uint32_t batch) {
    if (batch < 2) return false;
    if (batch <= 4 && type != YULE_DTYPE_Q5_K) return n_cols > 4096;
    if (type == YULE_DTYPE_Q4_K) return batch <= 12 || (batch <= 16 && n_rows * n_cols <= (17ull << 20));
    return batch <= 32 || (batch <= 48 && (n_rows * n_cols > (17ull << 20) || type == YULE_DTYPE_Q4_0 || type == YULE_DTYPE_Q5_K));
}

// And against the GEMM with its re-layout.  Q4_K (GEMM, this): 8 vectors 8192x28672 67.5, 68.3 us, smaller ones 6 to 9 us for this; 9 to 12 vectors
// 14336x4096 26.7, 24.0, 28672x4096 42.3, 42.4, 28672x8192 71.8, 83.5, 8192x28672 67.8, 84.4; 16 vectors 4096x4096 17.7, 13.7, 14336x4096 27.2, 29.2,
// 8192x8192 28.8, 33.4.  (Up to twelve vectors it is this one also where the GEMM is faster: its accumulators truncate, and the error against
// 64 bits would go from 1.6e-7 to 3.2e-7 to 4.0e-7, 4608x28672.)
// The other formats' GEMM (qgemm_int.cu) has the error of this kernel up to 4096 columns (Q8_0 by 24 vectors 1.0e-7 both, Q5_K 1.1e-7 both) and up to 6 % more beyond (14336 columns:
// Q8_0 1.07e-7, 1.12e-7, Q5_K 1.17, 1.19, Q6_K 1.14, 1.20; 65536: Q6_K 1.25, 1.35), so time decides; a seventeenth vector is a second pass here.  17, 24, 32 vectors, GEMM against this: Q5_K 2048x2048 17, 17, 17 against 15, 17, 20 us, 2048x5632 20, 20, 20
// against 22, 24, 33, 8192x28672 112, 113, 114 against 170, 188, 232; Q6_K 2048x2048 18, 18, 18 against 15, 17, 19, 4096x4096 18, 19, 19 against 23, 24, 27; Q8_0 2048x2048 20, 21, 21
// against 14, 15, 16, 2048x5632 23, 23, 24 against 21, 24, 27, 8192x8192 47, 47, 47 against 44, 50, 61, 4096x14336 40, 40, 41 against 47, 52, 81; Q4_0 the same within 10 %.
bool qmv_rows_preferred(uint32_t type, uint64_t n_rows, uint32_t n_cols, uint32_t batch) {
    if (batch <= 16 || type == YULE_DTYPE_Q4_K) return qmv_rows_over_matvecs(type, n_rows, n_cols, batch);
    const bool small = n_rows * n_cols <= (8ull << 20);
    if (type == YULE_DTYPE_Q5_K || type == YULE_DTYPE_Q6_K) return small && batch <= 24;
    return batch <= (small ? 32u : n_cols <= 8192 ? 20u : 16u);
}

bool qmv_rows_supported(uint32_t type, const void *w, const float *x, uint32_t n_cols, uint32_t x_stride) {
    switch (type) {
        case YULE_DTYPE_Q4_K: case YULE_DTYPE_Q5_K: case YULE_DTYPE_Q6_K: case YULE_DTYPE_Q8_0: case YULE_DTYPE_Q4_0: break;
        default: return false;
    }
    return n_cols != 0 && n_cols % 256 == 0 && w && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 &&
           x_stride % 4 == 0;
}

cudaError_t launch_qmv_rows(const QmvRows &f, cudaStream_t s, uint64_t *launches) {
    if (f.n_seg == 0 || f.n_seg > 3 || f.batch == 0 || (f.swiglu_pair && (f.n_seg != 2 || f.rows[0] != f.rows[1]))) return cudaErrorInvalidValue;
    for (uint32_t i = 0; i < f.n_seg; i++)
        if (!qmv_rows_supported(f.type, f.w[i], f.x, f.n_cols, f.x_stride)) return cudaErrorInvalidValue;
    switch (f.type) {
        case YULE_DTYPE_Q4_K: return launch_format<kQ4K>(f, s, launches);
        case YULE_DTYPE_Q5_K: return launch_format<kQ5K>(f, s, launches);
        case YULE_DTYPE_Q6_K: return launch_format<kQ6K>(f, s, launches);
        case YULE_DTYPE_Q8_0: return launch_format<kQ8>(f, s, launches);
        case YULE_DTYPE_Q4_0: return launch_format<kQ4>(f, s, launches);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace yule
