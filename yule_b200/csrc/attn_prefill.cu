// attn_prefill.cu — causal grouped-query attention of many query tokens over the fp32 KV cache, on tcgen05 with its operands and sums in shared and tensor memory.
//
// What it computes is the per-head loop of yule-infer/src/model_runner.rs:672-758 for every token of a prompt chunk: the
// reference feeds a prompt token by token (yule-infer/src/gpu_runner.rs:146-160), so token i attends to positions [0, i].
// One query per CTA (attention.cu) reads every K and V row once per token and multiplies on the FMA pipe: 2.4 ms per layer
// for a 2048-token prompt of the 8B shape.  Here 128 query rows share each K / V tile of 64 positions.
//
// Precision.  The cache and the queries are fp32, the tensor core multiplies fp16 and truncates what it adds to.  Scores: a query row and a tile of K are scaled by powers
// of two and split into three terms, the first a multiple of 64 of at most 2^14, so that the sum of first by first terms over all dimensions is exact in 24 bits and
// the truncation falls on products 2^-8 as large; the two are added in fp32, and what that and the scaling round off multiplies the probability as 1 + rest.
// Probabilities and V are fp16 hi + lo (22 bits), small products first, one accumulator per tile, added up in fp32 with what truncation takes on
// average given back.  Soft-max is fp32 with a running maximum.  Error against 64 bits (2-norm, units of 2^-24; before: the mma.sync kernel that had an accumulator per
// MMA): 700 tokens, scores of N(0, 1) 2.5 (3.3), N(0, 4^2) 2.6 (4.1), 2000 tokens 2.7 (4.3), a few channels 20 times as large 2.4 to 3.5 (22).  (hi + lo for
// scores too, in two chains of four additions: 2.8, 4.9 and 46.)
//
// What a query does not see.  One scale for a tile's rows is a loss to the small ones, and a masked position's probability of
// zero makes NaN of an infinite V row.  Either would let a token change what tokens before it get.  So a CTA that
// meets rows of K or V whose largest elements lie more than kRange binary orders apart (the small ones would lose bits), or
// a value that is not finite, computes its rows on the FMA pipe (exact_rows), where a query touches the
// positions that it attends to and no others.  With rows of one model's layer neither happens.
//
// Work split.  A first kernel writes K and V once per layer as the tensor core reads them (attn_prefill_operands_kernel; the GEMM's scratch, which is free between two GEMMs,
// holds them, or as many KV heads at a time as fit).  CTA (query tile, KV head, sequence): 128 rows = GROUP query heads x 128/GROUP tokens, so that all rows share
// the K / V tiles of one KV head and the causal edge cuts few tiles; 16 warps: 0-7 soft-max, a thread per row and half of a tile's positions, 8-11 output sums, a thread per
// row, 12 issues the MMAs, 13 and 14 the bulk copies of K (two buffers) and V (one).  Scores and probabilities have two buffers in tensor memory, so that the MMAs
// of the next tile's scores and of the last one's output run under the soft-max.
//
// What bounds it: the soft-max, some 850 instructions per warp and tile of which the scheduler issues one in two clocks, and the chain of hand-offs around it; the tensor pipe has 48 + 16 MMAs
// of 42 to 64 clocks a tile.  Per layer, us, the mma.sync kernel (fp32 tiles converted in every CTA, fp32 additions behind every MMA) and this with its operands kernel: 2048 tokens of the 8B
// shape 750, 268, 777 tokens of the 1.1B shape 81, 43.

#include <cfloat>
#include <mutex>
#include <type_traits>

#include <cuda_fp16.h>

#include "internal.h"
#include "qgemm_common.cuh"

namespace yule {

namespace {

constexpr int kRows = 128;  // query rows per CTA = TMEM lanes
constexpr int kKeys = 64;   // positions per K / V tile
// Warpgroups of a CTA: two for the soft-max (a thread per query row and half of a tile's positions), one for the output sums (a thread per row), and one whose first
// three warps issue the MMAs and the copies of K and of V.
constexpr int kThreads = 512, kMmaWarp = 12, kLoadK = 13, kLoadV = 14;
constexpr int kLaunchRegs = 128;  // registers per thread that 512 threads are launched with (the build checks that the kernels get them)
constexpr int kSoftRegs = 136, kSumRegs = 192, kIssueRegs = 48;
static_assert(2 * kSoftRegs + kSumRegs + kIssueRegs <= 4 * kLaunchRegs, "register split");
// What truncation takes of a sum on average, as a fraction (four additions at full size): given back.
constexpr float kTruncation = 0.8e-7f;
constexpr uint32_t kRange = 14;  // scaled, a tile's largest element is 2^13 to 2^14 and lo ends at 2^-24: 2^-1 keeps its 22 bits
constexpr float kProbScale = 4096.f;  // keeps small probabilities clear of fp16's subnormals; cancels in the division by the sum

struct PrefillParams {
    const float *q;
    const float *k_cache, *v_cache;
    float *out;
    // A launch is over pairs (sequence, KV head) from pair0 on; what follows is per (pair of the launch, tile).
    uint32_t pair0;
    float4 *stats;  // scale of K, its inverse, scale of V, its inverse; the first is 0 where a tile is not for the tensor core
    unsigned char *planes;  // K hi, K lo, V hi, V lo in the operands' layout
    uint32_t n_tokens, pos0, n_kv_heads, kv_stride, q_stride, out_stride, all_tiles;
    size_t kv_batch_stride;
    int *status;
};

__device__ __forceinline__ uint32_t h2(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
// (a, b) → packed fp16 pairs hi and lo
__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = h2(h);
    lo = h2(__floats2half2_rn(a - f.x, b - f.y));
}
// (a, b), of at most 2^14, as three fp16 terms: multiples of 64, and 11 bits of what is left twice over.  Products of two first terms are multiples of 2^12 and at most
// 2^28, so their sum over 128 dimensions is exact in 24 bits, whatever the tensor core does with the 25th; the others are 2^-8 of it and less.
__device__ __forceinline__ void split3(float a, float b, uint32_t (&t)[3]) {
    constexpr float kRound = 805306368.f;  // 1.5 · 2^29
    const float a0 = __fsub_rn(__fadd_rn(a, kRound), kRound), b0 = __fsub_rn(__fadd_rn(b, kRound), kRound);
    t[0] = h2(__floats2half2_rn(a0, b0));
    split2(a - a0, b - b0, t[1], t[2]);
}
// 2^e with m·2^e in [2^13, 2^14) and its inverse; m == 0, inf and NaN give 1 and 1 (they stay what they are)
__device__ __forceinline__ void pow2_scale(float m, float &scale, float &inv) {
    const int eb = (int)((__float_as_uint(m) >> 23) & 0xFFu);
    int se = (m == 0.f || eb == 0xFF) ? 127 : 127 + 13 - (eb - 127);
    se = se < 1 ? 1 : (se > 253 ? 253 : se);
    scale = __uint_as_float((uint32_t)se << 23);
    inv = __uint_as_float((uint32_t)(254 - se) << 23);
}

// The eight rows of a warp, position by position in fp32.  (Inlined: the kernel moves registers between its warps, which calls know nothing of.)
template <int HD, int GROUP>
__device__ __forceinline__ void exact_rows(const PrefillParams &p, const float *kc, const float *vc, uint32_t seq, uint32_t kvh, uint32_t first, uint32_t n_rows) {
    constexpr int N = HD / 32;
    const uint32_t lane = threadIdx.x & 31;
    #pragma unroll 1
    for (uint32_t row = first; row < first + 8 && row < n_rows; row++) {
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


template <int HD>
struct Layout {
    // Operands in the no-swizzle core-matrix layout (8 rows x 16 bytes; core matrices of one step of eight contiguous along the rows): Q and K rows by
    // dimension, V transposed: dimensions by position.
    static constexpr uint32_t kQPlane = kRows * HD * 2;   // three terms
    static constexpr uint32_t kKPlane = kKeys * HD * 2;   // three terms
    static constexpr uint32_t kVPlane = kKeys * HD * 2;   // two
    static constexpr uint32_t kTile = 3 * kKPlane + 2 * kVPlane;  // in memory
    static constexpr uint32_t kOffK = 3 * kQPlane, kOffV = kOffK + 2 * 3 * kKPlane, kOffRows = kOffV + 2 * kVPlane;  // two buffers of K, one of V
    // per row: alpha (two tiles), soft-max sums of both halves (before them, in the same words, their largest scores), score factor; then barriers
    static constexpr uint32_t kOffBars = kOffRows + 5 * kRows * 4;
    static constexpr uint32_t kSmem = kOffBars + 24 * 8 + 16;
    // tensor memory columns: two buffers of scores (product of the first terms | all others), output, two buffers of probabilities (hi, lo)
    static constexpr uint32_t kS = 0, kO = 256, kP = 384;
    static_assert(kSmem <= 227 * 1024, "shared memory");
};

// A tile of K and V as the tensor core reads it: scaled by a power of two, in fp16 terms (K three, V two), in the operands' layout; its scales, and whether its rows can share
// them.  Once per layer and pass: every query tile reads these (converting them in the CTAs that use them, 32 times over for 2048 tokens, took
// a third of the time, and 256 threads).
template <int HD>
__global__ void __launch_bounds__(256) attn_prefill_operands_kernel(const __grid_constant__ PrefillParams p) {
    using L = Layout<HD>;
    yule_pdl_launch_dependents();
    yule_pdl_wait();
    __shared__ uint32_t row_max[2][kKeys];
    __shared__ float scales[2];
    const uint32_t tile = blockIdx.x, kvh = (p.pair0 + blockIdx.y) % p.n_kv_heads, seq = (p.pair0 + blockIdx.y) / p.n_kv_heads, t = threadIdx.x, lane = t & 31;
    const uint32_t n_keys = p.pos0 + p.n_tokens - tile * kKeys;  // positions of the tile that are there (or more); zeros for the others, which are masked
    const size_t at = seq * p.kv_batch_stride + (size_t)kvh * HD + (size_t)tile * kKeys * p.kv_stride, slot = (size_t)blockIdx.y * p.all_tiles + tile;
    const float *kc = p.k_cache + at, *vc = p.v_cache + at;
    if (t < 2 * kKeys) row_max[t / kKeys][t % kKeys] = 0;
    __syncthreads();
    auto bits = [](float x) { return __float_as_uint(x) & 0x7FFFFFFFu; };  // ordered like |x|; an infinity or NaN wins
    // K: eight dimensions of a key; eight neighbouring lanes take eight keys (whole rows of core matrices), the four groups of a warp four steps (whole lines).
    // V: eight positions of a dimension; neighbouring lanes take neighbouring dimensions.
    constexpr int N = HD / 32;  // pieces of each per thread
    float k[N][8], v[N][8];
    auto place = [&](uint32_t i, uint32_t &key, uint32_t &step) {
        const uint32_t unit = i * 8 + (t >> 5);
        key = (unit & 7u) * 8 + (t & 7u), step = (unit >> 3) * 4 + ((t >> 3) & 3u);
    };
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        uint32_t key, step;
        place(i, key, step);
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (key < n_keys) {
            const float4 *src = reinterpret_cast<const float4 *>(kc + (size_t)key * p.kv_stride + 8 * step);
            a = __ldcg(src), b = __ldcg(src + 1);
        }
        k[i][0] = a.x, k[i][1] = a.y, k[i][2] = a.z, k[i][3] = a.w, k[i][4] = b.x, k[i][5] = b.y, k[i][6] = b.z, k[i][7] = b.w;
        const uint32_t unit = i * 256 + t, dim = unit % HD, k8 = unit / HD;
#pragma unroll
        for (uint32_t e = 0; e < 8; e++) v[i][e] = k8 * 8 + e < n_keys ? __ldcg(vc + (size_t)(k8 * 8 + e) * p.kv_stride + dim) : 0.f;
    }
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        uint32_t key, step, most = 0;
        place(i, key, step);
#pragma unroll
        for (int e = 0; e < 8; e++) most = max(most, bits(k[i][e]));
        atomicMax(&row_max[0][key], most);
        const uint32_t k8 = (i * 256 + t) / HD;  // the same for a warp
#pragma unroll
        for (uint32_t e = 0; e < 8; e++) {
            const uint32_t all = __reduce_max_sync(0xffffffffu, bits(v[i][e]));
            if (lane == 0) atomicMax(&row_max[1][k8 * 8 + e], all);
        }
    }
    __syncthreads();
    if (t < 32) {
        uint32_t most[2], least[2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const uint32_t a = row_max[m][lane], b = row_max[m][lane + 32];
            most[m] = __reduce_max_sync(0xffffffffu, max(a, b));
            least[m] = __reduce_min_sync(0xffffffffu, min(a ? a : 0x7F800000u, b ? b : 0x7F800000u));  // rows of zeros lose nothing
        }
        float4 s;
        pow2_scale(__uint_as_float(most[0]), s.x, s.y);
        pow2_scale(__uint_as_float(most[1]), s.z, s.w);
        if (lane == 0) {
            scales[0] = s.x, scales[1] = s.z;
            if (max(most[0], most[1]) >= 0x7F800000u || most[0] > least[0] + (kRange << 23) || most[1] > least[1] + (kRange << 23)) s.x = 0.f;
            p.stats[slot] = s;
        }
    }
    __syncthreads();
    unsigned char *to = p.planes + slot * L::kTile;
    const float ks = scales[0], vs = scales[1];
#pragma unroll
    for (uint32_t i = 0; i < N; i++) {
        uint32_t key, step, t3[4][3], h[4], l[4];
        place(i, key, step);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            split3(k[i][2 * e] * ks, k[i][2 * e + 1] * ks, t3[e]);
            split2(v[i][2 * e] * vs, v[i][2 * e + 1] * vs, h[e], l[e]);
        }
        unsigned char *kd = to + step * (kKeys * 16) + key * 16, *vd = to + 3 * L::kKPlane + (i * 256 + t) * 16;
#pragma unroll
        for (int m = 0; m < 3; m++) *reinterpret_cast<uint4 *>(kd + m * L::kKPlane) = make_uint4(t3[0][m], t3[1][m], t3[2][m], t3[3][m]);
        *reinterpret_cast<uint4 *>(vd) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4 *>(vd + L::kVPlane) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

template <int HD, int GROUP>
__global__ void __launch_bounds__(kThreads, 1) attn_prefill_kernel(const __grid_constant__ PrefillParams p) {
    using L = Layout<HD>;
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int KS = HD / 16;  // k16 steps of a score
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t kvh = (p.pair0 + blockIdx.y) % p.n_kv_heads, seq = (p.pair0 + blockIdx.y) / p.n_kv_heads;
    // the longest tiles first: the last query tiles see the most keys
    const uint32_t tile = gridDim.x - 1 - blockIdx.x;
    const uint32_t n_rows = p.n_tokens * GROUP, row0 = tile * kRows;
    const uint32_t last_row = row0 + kRows < n_rows ? row0 + kRows - 1 : n_rows - 1;
    const uint32_t last_pos = p.pos0 + last_row / GROUP;
    const uint32_t n_tiles = last_pos / kKeys + 1;
    yule_pdl_launch_dependents();

    float *alpha_row = reinterpret_cast<float *>(smem + L::kOffRows), *sum_row = alpha_row + 2 * kRows, *factor_row = sum_row + 2 * kRows;
    float *most_row = sum_row;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L::kOffBars);
    const uint32_t bar0 = smem_u32(bars);
    // pairs by tile parity: K there, free; scores there, free; probabilities there, free; alpha free; else one: V there, free; output there, free; sums there
    const uint32_t k_full = bar0, v_full = bar0 + 16, k_empty = bar0 + 32, v_empty = bar0 + 48, s_full = bar0 + 64, s_empty = bar0 + 80, p_full = bar0 + 96, p_empty = bar0 + 112,
                   o_full = bar0 + 128, o_empty = bar0 + 136, l_full = bar0 + 144, a_empty = bar0 + 152;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 24);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    if (tid == 0) {
        for (uint32_t b = 0; b < 2; b++) {
            mbar_init(k_full + 8 * b, 1);   // the loader's expect_tx
            mbar_init(k_empty + 8 * b, 1);  // tcgen05.commit
            mbar_init(s_full + 8 * b, 1);
            mbar_init(s_empty + 8 * b, 8);
            mbar_init(p_full + 8 * b, 8);
            mbar_init(p_empty + 8 * b, 1);
            mbar_init(a_empty + 8 * b, 4);
        }
        mbar_init(v_full, 1);
        mbar_init(v_empty, 1);
        mbar_init(o_full, 2);  // tcgen05.commit, and the thread that saw the probabilities (and with them alpha) arrive
        mbar_init(o_empty, 4);
        mbar_init(l_full, 8);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    yule_pdl_wait();
    const float *kc = p.k_cache + seq * p.kv_batch_stride + (size_t)kvh * HD, *vc = p.v_cache + seq * p.kv_batch_stride + (size_t)kvh * HD;
    const float4 *stats = p.stats + (size_t)blockIdx.y * p.all_tiles;
    bool exact = false;
    for (uint32_t j = tid; j < n_tiles; j += kThreads) exact = exact || __ldcg(stats + j).x == 0.f;

    // The query rows: four threads a row, each with the largest of all four, three fp16 terms.
    {
        static_assert(kThreads == 4 * kRows, "query rows");
        const uint32_t r = tid >> 2, part = tid & 3;
        uint32_t row = row0 + r;
        row = row < n_rows ? row : n_rows - 1;
        const float *qp = p.q + ((size_t)seq * p.n_tokens + row / GROUP) * p.q_stride + (size_t)(kvh * GROUP + row % GROUP) * HD;
        float mx = 0.f, sc, inv;
        float v[HD / 32][8];
#pragma unroll
        for (int i = 0; i < HD / 32; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) {  // (rows start on 8-byte boundaries)
                const float2 x = __ldcg(reinterpret_cast<const float2 *>(qp + (4 * i + part) * 8 + 2 * e));
                v[i][2 * e] = x.x, v[i][2 * e + 1] = x.y;
                mx = fmaxf(mx, fmaxf(fabsf(x.x), fabsf(x.y)));
            }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        pow2_scale(mx, sc, inv);
#pragma unroll
        for (int i = 0; i < HD / 32; i++) {
            uint32_t t[4][3];
#pragma unroll
            for (int e = 0; e < 4; e++) split3(v[i][2 * e] * sc, v[i][2 * e + 1] * sc, t[e]);
            unsigned char *to = smem + (4 * i + part) * (kRows * 16) + r * 16;
#pragma unroll
            for (int k = 0; k < 3; k++) *reinterpret_cast<uint4 *>(to + k * L::kQPlane) = make_uint4(t[0][k], t[1][k], t[2][k], t[3][k]);
        }
        if (part == 0) factor_row[r] = inv * (1.0f / sqrtf((float)HD));
        fence_async_smem();
    }
    exact = __syncthreads_or(exact);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    if (exact) {
        exact_rows<HD, GROUP>(p, kc, vc, seq, kvh, row0 + warp * 8, n_rows);
    } else if (warp >= 12) {
        move_registers<true, kIssueRegs, kLaunchRegs>();
        if (warp == kMmaWarp) {
            constexpr uint32_t idesc_s = (1u << 4) | ((uint32_t)(kKeys >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);  // fp16 × fp16 → fp32, K-major, M = 128, N = 64
            constexpr uint32_t idesc_o = (1u << 4) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);     // N = head_dim
            bool ok = true;
            auto await = [&](uint32_t bar, uint32_t parity) {
                ok = ok && mbar_wait(bar, parity, abort_flag, p.status);
                ok = __all_sync(0xffffffffu, ok);
                tc_fence_after();
                return ok;
            };
            const uint32_t base = smem_u32(smem);
            // A score: the exact product of the first terms, and beside it the others but those of 2^-24 and less (q1·k2, q2·k1, q2·k2).
            auto scores = [&](uint32_t j) {
                const uint32_t b = j & 1u, ph = (j >> 1) & 1u;
                if (!await(s_empty + 8 * b, ph ^ 1u) || !await(k_full + 8 * b, ph)) return;
                const uint32_t d = tmem_base + L::kS + b * 128;
                const uint64_t q = smem_desc(base, kRows * 16, 128), k = smem_desc(base + L::kOffK + b * 3 * L::kKPlane, kKeys * 16, 128);
                constexpr uint32_t q_plane = L::kQPlane >> 4, k_plane = L::kKPlane >> 4, q_step = (2 * kRows * 16) >> 4, k_step = (2 * kKeys * 16) >> 4;
                const uint32_t q_lo = (uint32_t)q, q_hi = (uint32_t)(q >> 32), k_lo = (uint32_t)k, k_hi = (uint32_t)(k >> 32);
                if (elect_one()) {
                    mma_steps<0, KS>([&](auto ic) {
                        constexpr uint32_t i = decltype(ic)::value;
                        constexpr int add = i != 0;
                        auto mma = [&](auto accc, uint32_t to, uint32_t qt, uint32_t kt) {
                            umma_f16_ss<decltype(accc)::value>(to, q_lo + i * q_step + qt * q_plane, q_hi, k_lo + i * k_step + kt * k_plane, k_hi, idesc_s);
                        };
                        constexpr std::integral_constant<int, add> fresh{};
                        constexpr std::integral_constant<int, 1> more{};
                        mma(fresh, d, 0, 0);
                        mma(fresh, d + 64, 0, 1);
                        mma(more, d + 64, 1, 0);
                        mma(more, d + 64, 1, 1);
                        mma(more, d + 64, 0, 2);
                        mma(more, d + 64, 2, 0);
                    });
                    umma_commit(s_full + 8 * b);
                    umma_commit(k_empty + 8 * b);
                }
                __syncwarp();
            };
            scores(0);
            for (uint32_t j = 0; j < n_tiles && ok; j++) {
                if (j + 1 < n_tiles) scores(j + 1);
                if (!ok) break;
                const uint32_t b = j & 1u;
                if (!await(v_full, j & 1u) || !await(o_empty, (j & 1u) ^ 1u) || !await(p_full + 8 * b, (j >> 1) & 1u)) break;
                const uint64_t v = smem_desc(base + L::kOffV, HD * 16, 128);
                constexpr uint64_t v_plane = L::kVPlane >> 4, v_step = (2 * HD * 16) >> 4;
                const uint32_t d = tmem_base + L::kO, hi = tmem_base + L::kP + b * 64, lo = hi + 32;
                if (elect_one()) {
                    mma_steps<0, 4>([&](auto kc) {
                        constexpr uint32_t i = decltype(kc)::value;
                        umma_f16_ts<(i != 0)>(d, lo + 8 * i, v + i * v_step + v_plane, idesc_o);
                        umma_f16_ts<1>(d, lo + 8 * i, v + i * v_step, idesc_o);
                        umma_f16_ts<1>(d, hi + 8 * i, v + i * v_step + v_plane, idesc_o);
                    });
                    mma_steps<0, 4>([&](auto kc) {
                        constexpr uint32_t i = decltype(kc)::value;
                        umma_f16_ts<1>(d, hi + 8 * i, v + i * v_step, idesc_o);
                    });
                    umma_commit(o_full);
                    umma_commit(v_empty);
                    umma_commit(p_empty + 8 * b);
                    mbar_arrive(o_full);
                }
                __syncwarp();
            }
        } else if ((warp == kLoadK || warp == kLoadV) && lane == 0) {
            const bool is_k = warp == kLoadK;
            const unsigned char *src = p.planes + (size_t)blockIdx.y * p.all_tiles * L::kTile + (is_k ? 0u : 3 * L::kKPlane);
            const uint32_t bytes = is_k ? 3 * L::kKPlane : 2 * L::kVPlane;
            for (uint32_t j = 0; j < n_tiles; j++) {
                const uint32_t b = is_k ? j & 1u : 0u, ph = is_k ? (j >> 1) & 1u : j & 1u, full = is_k ? k_full + 8 * b : v_full;
                if (!mbar_wait(is_k ? k_empty + 8 * b : v_empty, ph ^ 1u, abort_flag, p.status)) break;
                mbar_arrive_expect_tx(full, bytes);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 smem_u32(smem + (is_k ? L::kOffK + b * 3 * L::kKPlane : L::kOffV))),
                             "l"(src + (size_t)j * L::kTile), "r"(bytes), "r"(full)
                             : "memory");
            }
        }
    } else if (warp < 8) {
        // soft-max: this thread's row, half of its positions
        move_registers<true, kSoftRegs, kLaunchRegs>();
        const uint32_t quarter = warp & 3u, r = quarter * 32 + lane, lanes = quarter << 21, half = warp >> 2, col0 = half * (kKeys / 2);
        uint32_t row = row0 + r;
        row = row < n_rows ? row : n_rows - 1;
        const uint32_t qpos = p.pos0 + row / GROUP;
        const float row_factor = factor_row[r];
        float m = -FLT_MAX, l = 0.f;
        bool ok = true;
        float ki_next = __ldcg(stats).y;
        for (uint32_t j = 0; j < n_tiles; j++) {
            const uint32_t b = j & 1u, ph = (j >> 1) & 1u, key0 = j * kKeys + col0;
            const float f = row_factor * ki_next;
            if (j + 1 < n_tiles) ki_next = __ldcg(stats + j + 1).y;
            // (A warp that gives up goes on to meet the other half at the barrier of every tile, which has no bound.)
            ok = ok && mbar_wait(s_full + 8 * b, ph, abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const uint32_t at = tmem_base + lanes + L::kS + b * 128 + col0;
            const bool edge = j * kKeys + kKeys - 1 > p.pos0 + row0 / GROUP;  // some row of the tile may not see all keys
            const uint32_t seen = !edge ? kKeys : qpos < key0 ? 0u : qpos - key0 + 1;  // keys of this half that this row sees (or more)
            float mx4[4] = {-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
            if (ok) {
                uint32_t a[32], c[32];
                tmem_ld32_issue(at, a);
                tmem_ld32_issue(at + 64, c);
                tmem_ld_wait();
#pragma unroll
                for (uint32_t i = 0; i < 32; i += 2) {
                    float2 s = unpair(add2(pair_bits(a[i], a[i + 1]), pair_bits(c[i], c[i + 1])));
                    if (edge) s.x = i < seen ? s.x : -FLT_MAX, s.y = i + 1 < seen ? s.y : -FLT_MAX;
                    mx4[i & 2] = fmaxf(mx4[i & 2], s.x);
                    mx4[(i & 2) + 1] = fmaxf(mx4[(i & 2) + 1], s.y);
                }
            }
            // The largest score itself, in all its bits: sixteen of them, rounded up, are 2^-7 of a score too much, and with scores in the thousands nothing of a
            // probability is left in fp16.  One word per half and row has to do (there is no room for those of two tiles), so the warps of both halves meet twice.
            const float most = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            most_row[half * kRows + r] = most;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
            const float mx = fmaxf(most, most_row[(half ^ 1u) * kRows + r]);
            asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
            const float mn = mx < -3e38f ? m : fmaxf(m, mx * f);  // (no position of the tile that the row sees)
            const float alpha = expf(m - mn);
            m = mn;
            // the probabilities of two tiles before have been used, and alpha of that tile read
            ok = ok && mbar_wait(p_empty + 8 * b, ph ^ 1u, abort_flag, p.status) && mbar_wait(a_empty + 8 * b, ph ^ 1u, abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) continue;
            tc_fence_after();
            if (half == 0) alpha_row[b * kRows + r] = alpha;
            // What the addition, the scaling and the subtraction round off enters by its first power.  Step by step over sixteen
            // keys, two to an instruction: a key after the other is a chain of some 25 dependent operations each, and this warp has its scheduler
            // to itself (13000 clocks a tile).
            const uint64_t f2 = pair(f, f), minus_f2 = pair(-f, -f), mn2 = pair(mn, mn), minus_mn2 = pair(-mn, -mn), minus_one = pair(-1.f, -1.f),
                           prob = pair(kProbScale, kProbScale);
            uint64_t sum2 = 0;
#pragma unroll
            for (uint32_t c0 = 0; c0 < kKeys / 2; c0 += 16) {
                uint32_t a[16], c[16];
                tmem_ld16_issue(at + c0, a);
                tmem_ld16_issue(at + 64 + c0, c);
                tmem_ld_wait();
                if (c0 + 16 == kKeys / 2) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(s_empty + 8 * b);
                }
                uint64_t small[8], v[8], e[8];
#pragma unroll
                for (uint32_t i = 0; i < 8; i++) {
                    const uint64_t x = pair_bits(a[2 * i], a[2 * i + 1]), y = pair_bits(c[2 * i], c[2 * i + 1]), sum = add2(x, y);
                    small[i] = fma2(fma2(x, minus_one, sum), minus_one, y);
                    v[i] = mul2(sum, f2);
                    small[i] = fma2(small[i], f2, fma2(sum, f2, mul2(sum, minus_f2)));
                }
#pragma unroll
                for (uint32_t i = 0; i < 8; i++) {
                    e[i] = add2(v[i], minus_mn2);
                    small[i] = add2(small[i], fma2(add2(e[i], mn2), minus_one, v[i]));
                }
                float2 w[8];
#pragma unroll
                for (uint32_t i = 0; i < 8; i++) {
                    const float2 d = unpair(e[i]);
                    w[i] = make_float2(expf(d.x), expf(d.y));
                }
                uint32_t hi[8], lo[8];
#pragma unroll
                for (uint32_t i = 0; i < 8; i++) {
                    const uint64_t w2 = pair(w[i].x, w[i].y);
                    e[i] = mul2(fma2(w2, small[i], w2), prob);
                    float2 x = unpair(e[i]);
                    if (edge) {
                        x.x = c0 + 2 * i < seen ? x.x : 0.f, x.y = c0 + 2 * i + 1 < seen ? x.y : 0.f;
                        e[i] = pair(x.x, x.y);
                    }
                    sum2 = add2(sum2, e[i]);
                    const __half2 h = __floats2half2_rn(x.x, x.y);
                    const float2 back = __half22float2(h);
                    const float2 rest = unpair(fma2(pair(back.x, back.y), minus_one, e[i]));
                    hi[i] = h2(h);
                    lo[i] = h2(__floats2half2_rn(rest.x, rest.y));
                }
                const uint32_t to = tmem_base + lanes + L::kP + b * 64 + (col0 + c0) / 2;
                tmem_st8(to, make_uint4(hi[0], hi[1], hi[2], hi[3]), make_uint4(hi[4], hi[5], hi[6], hi[7]));
                tmem_st8(to + 32, make_uint4(lo[0], lo[1], lo[2], lo[3]), make_uint4(lo[4], lo[5], lo[6], lo[7]));
            }
            const float2 sums = unpair(sum2);
            const float sum = sums.x + sums.y;
            l = fmaf(l, alpha, sum);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + 8 * b);
        }
        // (over the largest scores of this row and half, which the other half's warp has read)
        sum_row[half * kRows + r] = l;
        __syncwarp();
        if (lane == 0) mbar_arrive(l_full);
    } else {
        // output sums: this thread's row
        move_registers<true, kSumRegs, kLaunchRegs>();
        const uint32_t r = (warp & 3u) * 32 + lane, lanes = (warp & 3u) << 21;
        uint64_t o[HD / 2];
#pragma unroll
        for (int i = 0; i < HD / 2; i++) o[i] = 0;
        bool ok = true;
        float vi_next = __ldcg(stats).w;
        for (uint32_t j = 0; j < n_tiles; j++) {
            const float vi = vi_next;
            if (j + 1 < n_tiles) vi_next = __ldcg(stats + j + 1).w;
            ok = mbar_wait(o_full, j & 1u, abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const float alpha = alpha_row[(j & 1u) * kRows + r];
            __syncwarp();
            if (lane == 0) mbar_arrive(a_empty + 8 * (j & 1u));
            const uint64_t alpha2 = pair(alpha, alpha), vi2 = pair(vi, vi), lost = pair(kTruncation, kTruncation);
#pragma unroll
            for (uint32_t c0 = 0; c0 < HD; c0 += 32) {
                uint32_t v[32];
                tmem_ld32_issue(tmem_base + lanes + L::kO + c0, v);
                tmem_ld_wait();
                if (c0 + 32 == HD) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(o_empty);
                }
#pragma unroll
                for (uint32_t i = 0; i < 32; i += 2) {
                    const uint64_t x = pair_bits(v[i], v[i + 1]);
                    o[(c0 + i) / 2] = fma2(o[(c0 + i) / 2], alpha2, mul2(fma2(x, lost, x), vi2));
                }
            }
        }
        if (ok) ok = mbar_wait(l_full, 0, abort_flag, p.status);
        const uint32_t row = row0 + r;
        if (ok && row < n_rows) {
            const float inv = 1.0f / (sum_row[r] + sum_row[kRows + r]);
            float *op = p.out + ((size_t)seq * p.n_tokens + row / GROUP) * p.out_stride + (size_t)(kvh * GROUP + row % GROUP) * HD;
#pragma unroll
            for (uint32_t i = 0; i < HD; i += 2) {
                const float2 x = unpair(o[i / 2]);
                *reinterpret_cast<float2 *>(op + i) = make_float2(x.x * inv, x.y * inv);
            }
        }
    }

    // common exit: nothing of this CTA may still be in flight when its TMEM and shared memory go
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (*abort_flag) {
        // gave up: let MMAs that were already issued drain before the resources are freed
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) {
        }
        __syncthreads();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int HD, int GROUP>
cudaError_t launch_variant(PrefillParams p, uint32_t n_seq, void *scratch, size_t scratch_bytes, bool pdl, cudaStream_t s, uint64_t *launches) {
    auto kern = attn_prefill_kernel<HD, GROUP>;
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
            if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Layout<HD>::kSmem);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    // As many pairs at a time as the scratch holds the operands of: all of them, but for long contexts and batches.
    const size_t per_pair = (size_t)p.all_tiles * (sizeof(float4) + Layout<HD>::kTile);
    const uint32_t pairs = p.n_kv_heads * n_seq;
    size_t fit = (scratch_bytes - 128) / per_pair;
    if (fit == 0) return cudaErrorInvalidValue;
    if (fit > pairs) fit = pairs;
    if (fit > 65535) fit = 65535;
    const uint32_t tiles = (p.n_tokens * GROUP + kRows - 1) / kRows;
    p.stats = static_cast<float4 *>(scratch);
    p.planes = static_cast<unsigned char *>(scratch) + ((fit * p.all_tiles * sizeof(float4) + 127) & ~(size_t)127);
    for (p.pair0 = 0; p.pair0 < pairs; p.pair0 += (uint32_t)fit) {
        const uint32_t n = pairs - p.pair0 < fit ? pairs - p.pair0 : (uint32_t)fit;
        e = launch_kernel(attn_prefill_operands_kernel<HD>, dim3(p.all_tiles, n), dim3(256), 0, s, pdl || p.pair0 > 0, p);
        if (e == cudaSuccess) e = launch_kernel(kern, dim3(tiles, n), dim3(kThreads), Layout<HD>::kSmem, s, true, p);
        if (e != cudaSuccess) return e;
        *launches += 2;
    }
    return cudaSuccess;
}

}  // namespace

// Whether the tiled kernel is the faster one.  Its time, in us: start, conversion and first tile 12 (head_dim 64) or 18, then 1.6 or 2.1 per K / V tile of the longest CTA and wave of
// CTAs; one query per CTA (attn_decode_gqa_kernel): 6, and per query of 4096 columns 0.1 and 1.04 ns per key.  Both per layer, measured, this kernel against that: 1.1B shape 66 tokens
// 14, 10, 100 15.4, 14.4, 130 15.7, 17.0, 300 21.5, 46; 8B shape 50 22, 12, 100 23.1, 21.7, 130 24.4, 27.4, 300 30, 78; 70B shape 66 23, 19, 100 25, 28, 300 37, 113.
bool attn_prefill_preferred(uint32_t hd, uint32_t n_heads, uint32_t n_kv_heads, uint32_t n_tokens, uint32_t n_seq, uint32_t pos0, int sm_count) {
    if (!attn_gqa_supported(hd, n_heads, n_kv_heads)) return false;
    const uint32_t group = n_heads / n_kv_heads;
    const uint64_t ctas = (uint64_t)((n_tokens * group + kRows - 1) / kRows) * n_kv_heads * n_seq;
    const uint64_t waves = (ctas + sm_count - 1) / sm_count, tiles = (pos0 + n_tokens + kKeys - 1) / kKeys;
    const double keys = pos0 + 0.5 * n_tokens, size = hd / 128.0;
    const double tiled = 6.0 + 12.0 * size + (double)waves * tiles * (1.1 + size) + 0.028 * size * tiles * n_kv_heads * n_seq;
    const double single = 6.0 + (double)n_seq * n_tokens * (0.1 + 1.04e-3 * keys) * ((double)n_heads * hd / 4096);
    return tiled < single;
}

size_t attn_prefill_scratch_bytes(uint32_t hd, uint32_t positions) {
    return (size_t)((positions + kKeys - 1) / kKeys) * (sizeof(float4) + (size_t)kKeys * hd * 10) + 128;
}

cudaError_t launch_attn_prefill(const AttnPrefill &a, cudaStream_t s, uint64_t *launches) {
    if (a.n_tokens == 0 || a.n_seq == 0) return cudaSuccess;
    if (!attn_gqa_supported(a.hd, a.n_heads, a.n_kv_heads) || a.q_stride % 2 || a.out_stride % 2 || a.kv_stride % 4 || !a.scratch || !a.status) return cudaErrorInvalidValue;
    if (a.scratch_bytes < attn_prefill_scratch_bytes(a.hd, a.pos0 + a.n_tokens)) return cudaErrorInvalidValue;
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
    p.all_tiles = (a.pos0 + a.n_tokens - 1) / kKeys + 1;
    p.status = a.status;
    const uint32_t g = a.n_heads / a.n_kv_heads;
    cudaError_t e = cudaErrorInvalidValue;
#define YULE_PREFILL_CASE(G, H) if (g == G && a.hd == H) e = launch_variant<H, G>(p, a.n_seq, a.scratch, a.scratch_bytes, a.pdl, s, launches)
    YULE_PREFILL_CASE(1, 64); YULE_PREFILL_CASE(2, 64); YULE_PREFILL_CASE(4, 64); YULE_PREFILL_CASE(8, 64);
    YULE_PREFILL_CASE(1, 128); YULE_PREFILL_CASE(2, 128); YULE_PREFILL_CASE(4, 128); YULE_PREFILL_CASE(8, 128);
#undef YULE_PREFILL_CASE
    return e;
}

}  // namespace yule
