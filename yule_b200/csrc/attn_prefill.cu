// attn_prefill.cu — causal grouped-query attention of many query tokens over the fp32 KV cache, on the tensor pipe.
//
// What it computes is the per-head loop of yule-infer/src/model_runner.rs:672-758 for every token of a prompt chunk: the
// reference feeds a prompt token by token (yule-infer/src/gpu_runner.rs:146-160), so token i attends to positions [0, i].
// One query per CTA (attention.cu) reads every K and V row once per token and multiplies on the FMA pipe: 2.4 ms per layer
// for a 2048-token prompt of the 8B shape.  Here 128 query rows share each K / V tile and the products run on mma.sync.
//
// Precision.  The cache and the queries are fp32; every operand is scaled by a power of two (per query row; per tile of K
// and of V) and split into fp16 hi + lo (22 significant bits); a product is four MMAs.  Probabilities are split the same way.
// The tensor core truncates what it adds to, so every hi·hi MMA starts from zero and its result is added in fp32, and what
// truncation takes on average (kTruncation) is given back; the three smaller products have an accumulator of their own, whose
// truncation nobody sees.  For the scores it also collects what the fp32 additions and the scaling round off, and
// multiplies the probability as 1 + rest.  Soft-max is fp32 with a running maximum.  Error against 64 bits (2-norm, N(0, 1) K and V)
// as a multiple of that of one query per CTA on the FMA pipe: 40 tokens 0.98 to 1.08, 200 to 2048 tokens 0.85 to 0.98, with queries
// four times as large 0.60 to 0.84, with a few channels of K and V 20 times as large 0.55 to 0.85.  (All MMAs of a sum on one
// accumulator: 2.3 to 4.6, 532 us where this takes 718; without lo·lo up to 1.11, 636 us.)
//
// What a query does not see.  One scale for a tile's rows is a loss to the small ones, and a masked position's probability of
// zero makes NaN of an infinite V row.  Either would let a token change what tokens before it get.  So a CTA that
// meets rows of K or V whose largest elements lie more than kRange binary orders apart (the small ones would lose bits), or
// a value that is not finite, computes its rows over again on the FMA pipe (exact_rows), where a query touches the
// positions that it attends to and no others.  With rows of one model's layer neither happens; looking takes 3 to 4 %.  Powers
// of two of their own for the rows of K and V, the latter's in the probabilities, would keep wide ranges on the tensor pipe, at 2 % more.
//
// Work split.  CTA (query tile, KV head, sequence): 128 rows = GROUP query heads x 128/GROUP tokens, so that all rows share
// the K / V tiles of one KV head and the causal edge cuts few tiles; warp w has rows 16w .. 16w + 15.  K / V come in tiles of
// 64 positions: asynchronous copies of the next tile's fp32 rows run under the MMAs of the current one; every thread then
// converts the pieces it copied itself.  The split queries stay in shared memory (in registers they left too few for the scores
// and their rest).  Per layer, 2048 tokens of the 8B shape 718 us, of the 1.1B shape 378.

#include <cfloat>
#include <mutex>

#include <cuda_fp16.h>

#include "internal.h"

namespace yule {

namespace {

constexpr int kThreads = 256;
constexpr int kRows = 128;  // query rows per CTA
constexpr int kKeys = 64;   // positions per K / V tile
// Mean of the part that truncation to 24 bits takes of a sum: half a unit of the last place, over mantissas of equal density in the
// logarithm, 2^-24 / (2 ln 2).
constexpr float kTruncation = 4.3e-8f;
constexpr uint32_t kRange = 14;  // scaled, a tile's largest element is 2^13 to 2^14 and lo ends at 2^-24: 2^-1 keeps its 22 bits
constexpr float kProbScale = 4096.f;  // keeps small probabilities clear of fp16's subnormals; cancels in the division by the sum

struct PrefillParams {
    const float *q;
    const float *k_cache, *v_cache;
    float *out;
    uint32_t n_tokens, pos0, n_kv_heads, kv_stride, q_stride, out_stride;
    size_t kv_batch_stride;
};

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ uint32_t h2(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
// (a, b) → packed fp16 pairs hi and lo
__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = h2(h);
    lo = h2(__floats2half2_rn(a - f.x, b - f.y));
}
// 2^e with m·2^e in [2^13, 2^14) and its inverse; m == 0, inf and NaN give 1 and 1 (they stay what they are)
__device__ __forceinline__ void pow2_scale(float m, float &scale, float &inv) {
    const int eb = (int)((__float_as_uint(m) >> 23) & 0xFFu);
    int se = (m == 0.f || eb == 0xFF) ? 127 : 127 + 13 - (eb - 127);
    se = se < 1 ? 1 : (se > 253 ? 253 : se);
    scale = __uint_as_float((uint32_t)se << 23);
    inv = __uint_as_float((uint32_t)(254 - se) << 23);
}

template <int HD>
struct Layout {
    static constexpr uint32_t kPitch = HD * 2 + 16;               // bytes of an fp16 row: rows 16 bytes apart in bank terms
    static constexpr uint32_t kPlane = kKeys * kPitch;            // one of K hi, K lo, V hi, V lo
    static constexpr uint32_t kRaw = kKeys * HD * 4;              // fp32 tile of K or V
    static constexpr uint32_t kQPlane = kRows * kPitch;           // Q hi or lo
    static constexpr uint32_t kSmem = 4 * kPlane + 2 * kQPlane + 2 * kRaw + 128;
};

// The 16 rows of a warp, position by position in fp32.
template <int HD, int GROUP>
__device__ __noinline__ void exact_rows(const PrefillParams &p, const float *kc, const float *vc, uint32_t seq, uint32_t kvh, uint32_t first, uint32_t n_rows) {
    constexpr int N = HD / 32;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t row = first; row < first + 16 && row < n_rows; row++) {
        const size_t tok = (size_t)seq * p.n_tokens + row / GROUP;
        const uint32_t head = (kvh * GROUP + row % GROUP) * HD + lane, pos = p.pos0 + row / GROUP;
        float q[N], o[N], m = -FLT_MAX, l = 0.f;
#pragma unroll
        for (int i = 0; i < N; i++) q[i] = p.q[tok * p.q_stride + head + 32 * i], o[i] = 0.f;
        for (uint32_t k = 0; k <= pos; k++) {
            const float *kr = kc + (size_t)k * p.kv_stride + lane, *vr = vc + (size_t)k * p.kv_stride + lane;
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < N; i++) s = fmaf(q[i], kr[32 * i], s);
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
            s *= 1.0f / sqrtf((float)HD);
            const float mn = fmaxf(m, s), alpha = expf(m - mn), e = expf(s - mn);
            m = mn;
            l = fmaf(l, alpha, e);
#pragma unroll
            for (int i = 0; i < N; i++) o[i] = fmaf(o[i], alpha, e * vr[32 * i]);
        }
        const float inv = 1.0f / l;
#pragma unroll
        for (int i = 0; i < N; i++) p.out[tok * p.out_stride + head + 32 * i] = o[i] * inv;
    }
}

template <int HD, int GROUP>
__global__ void __launch_bounds__(kThreads, 1) attn_prefill_kernel(const __grid_constant__ PrefillParams p) {
    using L = Layout<HD>;
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int KS = HD / 16;      // k16 steps of a score
    constexpr int NT = HD / 8;       // n8 tiles of the output
    constexpr int CH = HD / 4;       // 16-byte pieces per row
    constexpr int PER = kKeys * CH / kThreads;  // pieces of K (and of V) per thread and tile
    unsigned char *planes = smem, *q_planes = smem + 4 * L::kPlane, *raw = q_planes + 2 * L::kQPlane;
    uint4 *red = reinterpret_cast<uint4 *>(raw + 2 * L::kRaw);  // per warp: largest |K|, |V|, and the smallest of its rows' largest
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const uint32_t kvh = blockIdx.y, seq = blockIdx.z;
    // the longest tiles first: the last query tiles see the most keys
    const uint32_t tile = gridDim.x - 1 - blockIdx.x;
    const uint32_t n_rows = p.n_tokens * GROUP, row0 = tile * kRows;
    const uint32_t last_row = row0 + kRows < n_rows ? row0 + kRows - 1 : n_rows - 1;
    const uint32_t last_pos = p.pos0 + last_row / GROUP;
    const uint32_t n_tiles = last_pos / kKeys + 1;
    yule_pdl_launch_dependents();
    yule_pdl_wait();

    const float *kc = p.k_cache + seq * p.kv_batch_stride + (size_t)kvh * HD, *vc = p.v_cache + seq * p.kv_batch_stride + (size_t)kvh * HD;
    const uint32_t raw_u32 = (uint32_t)__cvta_generic_to_shared(raw), planes_u32 = (uint32_t)__cvta_generic_to_shared(planes);
    auto copy_tile = [&](uint32_t j) {
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const uint32_t e = tid + i * kThreads, r = e / CH, c = e % CH;
            uint32_t pos = j * kKeys + r;
            pos = pos < last_pos ? pos : last_pos;  // rows past the end are masked; the copy stays inside what has been written
            const size_t src = (size_t)pos * p.kv_stride + 4 * c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(raw_u32 + e * 16), "l"(kc + src) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(raw_u32 + L::kRaw + e * 16), "l"(vc + src) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    copy_tile(0);

    // this lane's two query rows to shared memory, and the factor of their scores
    float row_scale[2];
    uint32_t qpos[2];
    {
        float mx[2] = {0.f, 0.f};
        const float *qp[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            uint32_t row = row0 + warp * 16 + g + 8 * r;
            row = row < n_rows ? row : n_rows - 1;
            qpos[r] = p.pos0 + row / GROUP;
            qp[r] = p.q + ((size_t)seq * p.n_tokens + row / GROUP) * p.q_stride + (size_t)(kvh * GROUP + row % GROUP) * HD + 2 * t;
#pragma unroll
            for (int k = 0; k < 2 * KS; k++) {
                const float2 v = *reinterpret_cast<const float2 *>(qp[r] + 8 * k);
                mx[r] = fmaxf(mx[r], fmaxf(fabsf(v.x), fabsf(v.y)));
            }
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
            mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
            float sc;
            pow2_scale(mx[r], sc, row_scale[r]);
            unsigned char *to = q_planes + (warp * 16 + g + 8 * r) * L::kPitch + 4 * t;
#pragma unroll
            for (int k = 0; k < 2 * KS; k++) {
                const float2 v = *reinterpret_cast<const float2 *>(qp[r] + 8 * k);
                uint32_t hi, lo;
                split2(v.x * sc, v.y * sc, hi, lo);
                *reinterpret_cast<uint32_t *>(to + 16 * k) = hi;
                *reinterpret_cast<uint32_t *>(to + L::kQPlane + 16 * k) = lo;
            }
            row_scale[r] *= 1.0f / sqrtf((float)HD);
        }
    }
    float o[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.f, 0.f};

    for (uint32_t j = 0; j < n_tiles; j++) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // this thread's own pieces: the tile's largest |K| and |V|, and the largest of each row (the pieces of CH neighbouring lanes)
        auto bits = [](float x) { return __float_as_uint(x) & 0x7FFFFFFFu; };  // ordered like |x|; an infinity or NaN wins
        uint4 mm = make_uint4(0u, 0u, 0x7F800000u, 0x7F800000u);
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const uint32_t e = tid + i * kThreads;
            const float4 a = *reinterpret_cast<const float4 *>(raw + e * 16), b = *reinterpret_cast<const float4 *>(raw + L::kRaw + e * 16);
            const uint32_t kb = max(max(bits(a.x), bits(a.y)), max(bits(a.z), bits(a.w))), vb = max(max(bits(b.x), bits(b.y)), max(bits(b.z), bits(b.w)));
#pragma unroll
            for (uint32_t h = 0; h < 32; h += CH) {  // (a partial member mask would take the two halves of the warp one after the other, by a slow path)
                const bool own = CH >= 32 || (lane & 16) == h;
                const uint32_t km = __reduce_max_sync(0xffffffffu, own ? kb : 0u), vm = __reduce_max_sync(0xffffffffu, own ? vb : 0u);
                mm.x = max(mm.x, km), mm.y = max(mm.y, vm);
                mm.z = min(mm.z, km ? km : mm.z), mm.w = min(mm.w, vm ? vm : mm.w);  // rows of zeros lose nothing
            }
        }
        if (lane == 0) red[warp] = mm;
        __syncthreads();  // and everyone is done with the planes of the tile before
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const uint4 o = red[w];
            mm.x = max(mm.x, o.x), mm.y = max(mm.y, o.y), mm.z = min(mm.z, o.z), mm.w = min(mm.w, o.w);
        }
        if (max(mm.x, mm.y) >= 0x7F800000u || mm.x > mm.z + (kRange << 23) || mm.y > mm.w + (kRange << 23)) {
            exact_rows<HD, GROUP>(p, kc, vc, seq, kvh, row0 + warp * 16, n_rows);
            return;
        }
        const float km = __uint_as_float(mm.x), vm = __uint_as_float(mm.y);
        float ks, ki, vs, vi;
        pow2_scale(km, ks, ki);
        pow2_scale(vm, vs, vi);
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const uint32_t e = tid + i * kThreads, at = (e / CH) * L::kPitch + (e % CH) * 8;
            const float4 a = *reinterpret_cast<const float4 *>(raw + e * 16), b = *reinterpret_cast<const float4 *>(raw + L::kRaw + e * 16);
            uint2 hi, lo;
            split2(a.x * ks, a.y * ks, hi.x, lo.x);
            split2(a.z * ks, a.w * ks, hi.y, lo.y);
            *reinterpret_cast<uint2 *>(planes + at) = hi;
            *reinterpret_cast<uint2 *>(planes + L::kPlane + at) = lo;
            split2(b.x * vs, b.y * vs, hi.x, lo.x);
            split2(b.z * vs, b.w * vs, hi.y, lo.y);
            *reinterpret_cast<uint2 *>(planes + 2 * L::kPlane + at) = hi;
            *reinterpret_cast<uint2 *>(planes + 3 * L::kPlane + at) = lo;
        }
        __syncthreads();
        if (j + 1 < n_tiles) copy_tile(j + 1);  // the raw pieces have been read by the threads that own them

        // scores of 16 rows x 64 keys
        float s[kKeys / 8][4], c[kKeys / 8][4];  // sums of hi·hi; everything smaller
        // ldmatrix: lanes 0-7 rows of (n, k low), 8-15 (n, k high), 16-23 (n + 1, k low), 24-31 (n + 1, k high)
        const uint32_t k_addr = planes_u32 + ((lane & 7) + ((lane >> 4) & 1) * 8) * L::kPitch + ((lane >> 3) & 1) * 16;
        // A fragments: lanes 0-7 rows 0-7, 8-15 rows 8-15 of the k low half, 16-31 the same of the k high half
        const uint32_t q_addr = planes_u32 + 4 * L::kPlane + (warp * 16 + (lane & 15)) * L::kPitch + (lane >> 4) * 16;
#pragma unroll
        for (int k = 0; k < KS; k++) {
            uint32_t qh[4], ql[4];
            ldsm4(qh, q_addr + k * 32);
            ldsm4(ql, q_addr + L::kQPlane + k * 32);
#pragma unroll
            for (int n = 0; n < kKeys / 8; n += 2) {
                uint32_t bh[4], bl[4];
                ldsm4(bh, k_addr + n * 8 * L::kPitch + k * 32);
                ldsm4(bl, k_addr + L::kPlane + n * 8 * L::kPitch + k * 32);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    float d[4];
                    mma_f16_z(d, qh, bh[2 * i], bh[2 * i + 1]);
                    if (k == 0) mma_f16_z(c[n + i], ql, bl[2 * i], bl[2 * i + 1]);
                    else mma_f16(c[n + i], ql, bl[2 * i], bl[2 * i + 1]);
                    mma_f16(c[n + i], ql, bh[2 * i], bh[2 * i + 1]);
                    mma_f16(c[n + i], qh, bl[2 * i], bl[2 * i + 1]);
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        if (k == 0) {
                            s[n + i][x] = d[x];
                        } else {  // what the addition rounds off goes to the small terms
                            const float sum = s[n + i][x] + d[x];
                            c[n + i][x] += d[x] - (sum - s[n + i][x]);
                            s[n + i][x] = sum;
                        }
                    }
                }
            }
        }
        // scale, mask, running soft-max
        const uint32_t key0 = j * kKeys + 2 * t;
        const bool edge = (j + 1) * kKeys - 1 > p.pos0 + row0 / GROUP;  // some row of the tile may not see all keys
        float alpha[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const float f = row_scale[r] * ki;
            float mx = -FLT_MAX;
#pragma unroll
            for (int n = 0; n < kKeys / 8; n++)
#pragma unroll
                for (int x = 2 * r; x < 2 * r + 2; x++) {
                    c[n][x] = fmaf(s[n][x], kTruncation, c[n][x]);
                    const float sum = s[n][x] + c[n][x];
                    float v = sum * f;
                    c[n][x] = fmaf(c[n][x] - (sum - s[n][x]), f, fmaf(sum, f, -v));  // what sum and product round off
                    if (edge && key0 + 8 * n + (x & 1) > qpos[r]) v = -FLT_MAX;
                    s[n][x] = v;
                    mx = fmaxf(mx, v);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float mn = fmaxf(m[r], mx);
            alpha[r] = expf(m[r] - mn);
            m[r] = mn;
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < kKeys / 8; n++)
#pragma unroll
                for (int x = 2 * r; x < 2 * r + 2; x++) {
                    // e^(v + c - mn), what the subtraction rounds off included: it is the first power that the small terms enter by
                    const float v = s[n][x], d = v - mn, w = expf(d), small = c[n][x] + (v - (d + mn));
                    const float e = v == -FLT_MAX ? 0.f : fmaf(w, small, w) * kProbScale;
                    s[n][x] = e;
                    sum += e;
                }
            l[r] = fmaf(l[r], alpha[r], sum);
        }
        // P as A fragments
        uint32_t ph[kKeys / 16][4], pl[kKeys / 16][4];
#pragma unroll
        for (int k = 0; k < kKeys / 16; k++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                split2(s[2 * k + h][0], s[2 * k + h][1], ph[k][2 * h], pl[k][2 * h]);
                split2(s[2 * k + h][2], s[2 * k + h][3], ph[k][2 * h + 1], pl[k][2 * h + 1]);
            }
        // ldmatrix.trans: lanes 0-7 keys (k low, n), 8-15 (k high, n), 16-23 (k low, n + 1), 24-31 (k high, n + 1)
        const uint32_t v_addr = planes_u32 + 2 * L::kPlane + ((lane & 7) + ((lane >> 3) & 1) * 8) * L::kPitch + ((lane >> 4) & 1) * 16;
#pragma unroll
        for (int n = 0; n < NT; n += 2) {
            float small[2][4], sum[2][4];
#pragma unroll
            for (int k = 0; k < kKeys / 16; k++) {
                uint32_t bh[4], bl[4];
                ldsm4t(bh, v_addr + k * 16 * L::kPitch + n * 16);
                ldsm4t(bl, v_addr + L::kPlane + k * 16 * L::kPitch + n * 16);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    float d[4];
                    mma_f16_z(d, ph[k], bh[2 * i], bh[2 * i + 1]);
                    if (k == 0) mma_f16_z(small[i], pl[k], bl[2 * i], bl[2 * i + 1]);
                    else mma_f16(small[i], pl[k], bl[2 * i], bl[2 * i + 1]);
                    mma_f16(small[i], pl[k], bh[2 * i], bh[2 * i + 1]);
                    mma_f16(small[i], ph[k], bl[2 * i], bl[2 * i + 1]);
#pragma unroll
                    for (int x = 0; x < 4; x++) sum[i][x] = k == 0 ? d[x] : sum[i][x] + d[x];
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int x = 0; x < 4; x++) o[n + i][x] = fmaf(o[n + i][x], alpha[x >> 1], (sum[i][x] + fmaf(sum[i][x], kTruncation, small[i][x])) * vi);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        const float inv = 1.0f / l[r];
        const uint32_t row = row0 + warp * 16 + g + 8 * r;
        if (row < n_rows) {
            float *op = p.out + ((size_t)seq * p.n_tokens + row / GROUP) * p.out_stride + (size_t)(kvh * GROUP + row % GROUP) * HD + 2 * t;
#pragma unroll
            for (int n = 0; n < NT; n++) *reinterpret_cast<float2 *>(op + 8 * n) = make_float2(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
        }
    }
}

template <int HD, int GROUP>
cudaError_t launch_variant(const PrefillParams &p, uint32_t n_seq, bool pdl, cudaStream_t s) {
    auto kern = attn_prefill_kernel<HD, GROUP>;
    static bool attr_done[64] = {};  // the opt-in for large dynamic shared memory belongs to the device
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !attr_done[dev]) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<HD>::kSmem);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    const uint32_t tiles = (p.n_tokens * GROUP + kRows - 1) / kRows;
    return launch_kernel(kern, dim3(tiles, p.n_kv_heads, n_seq), dim3(kThreads), Layout<HD>::kSmem, s, pdl, p);
}

}  // namespace

// Whether the tiled kernel is the faster one: its time goes with (waves of CTAs) x (K / V tiles of the longest CTA), about
// 7 us each at head_dim 128; one query per CTA (attn_decode_gqa_kernel) takes about 1.1 ns per query and key of eight KV
// heads of 512 output columns, and spreads a few queries over all SMs.
bool attn_prefill_preferred(uint32_t hd, uint32_t n_heads, uint32_t n_kv_heads, uint32_t n_tokens, uint32_t n_seq, uint32_t pos0, int sm_count) {
    if (!attn_gqa_supported(hd, n_heads, n_kv_heads)) return false;
    const uint32_t group = n_heads / n_kv_heads;
    const uint64_t ctas = (uint64_t)((n_tokens * group + kRows - 1) / kRows) * n_kv_heads * n_seq;
    const uint64_t waves = (ctas + sm_count - 1) / sm_count;
    const double keys = pos0 + 0.5 * n_tokens;
    const double tiled = (double)waves * ((pos0 + n_tokens + kKeys - 1) / kKeys) * 7.0 * hd / 128;
    const double single = 1.1e-3 * n_seq * n_tokens * keys * ((double)n_heads * hd / 4096);
    return tiled < single;
}

cudaError_t launch_attn_prefill(const AttnPrefill &a, cudaStream_t s, uint64_t *launches) {
    if (a.n_tokens == 0 || a.n_seq == 0) return cudaSuccess;
    if (!attn_gqa_supported(a.hd, a.n_heads, a.n_kv_heads) || a.q_stride % 2 || a.out_stride % 2 || a.kv_stride % 4) return cudaErrorInvalidValue;
    PrefillParams p = {};
    p.q = a.q;
    p.k_cache = a.k_cache;
    p.v_cache = a.v_cache;
    p.out = a.out;
    p.n_tokens = a.n_tokens;
    p.pos0 = a.pos0;
    p.n_kv_heads = a.n_kv_heads;
    p.kv_stride = a.kv_stride;
    p.q_stride = a.q_stride;
    p.out_stride = a.out_stride;
    p.kv_batch_stride = a.kv_batch_stride;
    const uint32_t g = a.n_heads / a.n_kv_heads;
    cudaError_t e = cudaErrorInvalidValue;
#define YULE_PREFILL_CASE(G, H) if (g == G && a.hd == H) e = launch_variant<H, G>(p, a.n_seq, a.pdl, s)
    YULE_PREFILL_CASE(1, 64); YULE_PREFILL_CASE(2, 64); YULE_PREFILL_CASE(4, 64); YULE_PREFILL_CASE(8, 64);
    YULE_PREFILL_CASE(1, 128); YULE_PREFILL_CASE(2, 128); YULE_PREFILL_CASE(4, 128); YULE_PREFILL_CASE(8, 128);
#undef YULE_PREFILL_CASE
    if (e == cudaSuccess) *launches += 1;
    return e;
}

}  // namespace yule
