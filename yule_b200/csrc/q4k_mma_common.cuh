// q4k_mma_common.cuh — Q4_K device code of the persistent decode kernel (decode_mega.cu, weights staged in shared memory): the
// fp16 MMA and the 6-bit scale unpack.  Include inside namespace yule { namespace { … } }.
#pragma once

constexpr int kWarps = 8;        // warps per group: one per super-block slot of a tile
constexpr int kGroups = 2;       // independent 8-warp groups per CTA
constexpr int kThreadsCta = kGroups * kWarps * 32;  // 512

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t h2_as_u32(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }

#include "tp_pairs.cuh"

// ── sub-blocks in the N dimension ───────────────────────────────────────────────────────────
// B column n = 4·part + t' carries x (part 0 = hi, 1 = lo) only at the k slots that lane t' feeds,
// zeros elsewhere.  Those slots belong to one sub-block (2t' for the low-nibble MMA, 2t'+1 for the
// high-nibble one), so D[row][n] is that sub-block's Σ q·x whatever the k order — and the weights
// go in unscaled: the nibble's bits are used as an fp16 subnormal (q·2^-24, or 16q·2^-24 for a
// high nibble), one AND per pair of weights.  Lane (g, t) ends up with columns 2t, 2t+1 =
// groups 2u, 2u+1 (u = t&1) of part t>>1, i.e. sub-blocks 4u..4u+3, and applies their scales.
struct RowScalesF {
    float sc[4];  // sc[4u + i] · d · 2^24 (i even: low-nibble MMAs) or · d · 2^20 (i odd)
    float mn[4];  // mn[4u + i] · dmin, zero in the lanes of the lo part (mins are charged once)
};

template <bool Q5>
__device__ __forceinline__ RowScalesF unpack_scales_f(const uint4 &hdr, int u, bool charge_mins) {
    uint32_t sc4, mn4;  // four 6-bit values each, one per byte (dequant.rs:176-190)
    if (u == 0) {
        sc4 = hdr.y & 0x3F3F3F3Fu;
        mn4 = hdr.z & 0x3F3F3F3Fu;
    } else {
        sc4 = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
        mn4 = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
    }
    const float d = __half2float(__ushort_as_half((unsigned short)(hdr.x & 0xFFFFu)));
    const float dmin = charge_mins ? __half2float(__ushort_as_half((unsigned short)(hdr.x >> 16))) : 0.f;
    // Q5_K operands carry q·2^-24 in both halves; Q4_K's high nibbles stay in place (16q·2^-24)
    const float d24 = d * 16777216.0f, d20 = Q5 ? d24 : d * 1048576.0f;
    const float k23 = 8388608.0f;
    RowScalesF r;
    r.sc[0] = (__uint_as_float(__byte_perm(sc4, 0x4B000000u, 0x7440)) - k23) * d24;
    r.sc[1] = (__uint_as_float(__byte_perm(sc4, 0x4B000000u, 0x7441)) - k23) * d20;
    r.sc[2] = (__uint_as_float(__byte_perm(sc4, 0x4B000000u, 0x7442)) - k23) * d24;
    r.sc[3] = (__uint_as_float(__byte_perm(sc4, 0x4B000000u, 0x7443)) - k23) * d20;
    r.mn[0] = (__uint_as_float(__byte_perm(mn4, 0x4B000000u, 0x7440)) - k23) * dmin;
    r.mn[1] = (__uint_as_float(__byte_perm(mn4, 0x4B000000u, 0x7441)) - k23) * dmin;
    r.mn[2] = (__uint_as_float(__byte_perm(mn4, 0x4B000000u, 0x7442)) - k23) * dmin;
    r.mn[3] = (__uint_as_float(__byte_perm(mn4, 0x4B000000u, 0x7443)) - k23) * dmin;
    return r;
}
