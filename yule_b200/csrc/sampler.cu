// sampler.cu — Yule's token sampler on the device (yule-infer/src/sampler.rs:17-136): repetition penalty,
// temperature, softmax, top-k, min-p, top-p, renormalisation and the inverse-CDF pick, in one kernel, so that a
// sampled decode loop moves neither the vocabulary-sized logits nor the pick across the bus.
//
// One cluster of eight CTAs, each of which keeps an eighth of the vocabulary (consecutive indices) in its shared memory from
// the single read of the logits to the pick; every step of the reference is a phase between cluster barriers, at which
// the CTAs read one another's partial sums and histograms (distributed shared memory; each phase has its own words, so
// that one barrier per phase is enough).  Eight SMs because a phase is then about as long as a barrier: one CTA with the
// probabilities in global memory took 477 us per pick from 128256 logits, as long as eight layers of a model of that size.
// What the reference does with sorts is done with radix selection over the bit patterns of the (non-negative)
// probabilities:
//   top-k   the threshold `sorted[k]` of the descending order (sampler.rs:58-70) is the value of rank k: four
//           passes over 8-bit digits with a 256-bin count histogram (equal digits within a warp are counted together:
//           nearly all probabilities of a large vocabulary share a few exponents);
//   top-p   the shortest descending prefix whose mass reaches top_p (sampler.rs:83-118): the same descent with
//           per-bin sums, accumulated as 2^-44 fixed point in 64-bit integers so that the result does not
//           depend on the order in which threads add; equal probabilities at the boundary are taken in index
//           order (the reference's unstable sort leaves that order open).
// The random number is an argument (the reference draws it from the OS CSPRNG, sampler.rs:212-220): the host
// supplies it, which also makes a sampled run reproducible.
// Differences from the CPU code are confined to the order of floating-point additions (tree instead of
// sequential sums) and the device's expf; they can move a pick only when the random value falls within
// rounding distance of a boundary of the cumulative distribution.

#include <cfloat>

#include <cooperative_groups.h>

#include "internal.h"

namespace yule {

namespace {

namespace cg = cooperative_groups;

constexpr int kSampThreads = 1024;
constexpr uint32_t kSampCtas = 8;
constexpr size_t kSampMaxSmem = 200 * 1024;  // slices that need more live in global memory
constexpr float kFixScale = 17592186044416.0f;  // 2^44
constexpr uint32_t kFew = 256;  // candidates that one CTA finishes alone

__device__ __forceinline__ float block_reduce_max(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[threadIdx.x & 31];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float block_reduce_sum(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[threadIdx.x & 31];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Inclusive scan of one value per thread over the CTA (warp scans, then the warp totals).
__device__ __forceinline__ uint32_t block_scan_inclusive_u32(uint32_t v, uint32_t *red, uint32_t *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    __syncthreads();
    if (lane == 31) red[wid] = v;
    __syncthreads();
    uint32_t w = red[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
    }
    const uint32_t before = __shfl_sync(0xffffffffu, w, wid > 0 ? wid - 1 : 0);
    *total = __shfl_sync(0xffffffffu, w, 31);
    return v + (wid > 0 ? before : 0u);
}

// The logit of token i after the repetition penalty (once per earlier occurrence, sampler.rs:26-38) and the
// temperature (sampler.rs:41-46).
__device__ __forceinline__ float adjusted_logit(const float *logits, const uint32_t *counts, uint32_t i, float penalty,
                                                bool penalise, float inv_t, bool scale) {
    float l = logits[i];
    if (penalise)
        for (uint32_t c = counts[i]; c > 0; c--) l = l > 0.0f ? l / penalty : l * penalty;
    if (scale) l *= inv_t;
    return l;
}

// What the CTAs of the cluster show one another: every phase writes words of its own.
struct SampShared {
    float mx, sum, total;
    uint32_t ties, first;
    float best;
    uint32_t best_idx;
    uint32_t kcnt[4][256];            // top-k histograms
    unsigned long long psum[4][256];  // top-p histograms
    uint32_t pcnt[4][256];
    uint32_t n_cand;
    uint2 cand[kFew];  // (bits of the probability, token)
};

// What is left of a call once few candidates are: `c` of them, at most kFew, lie on the CTAs of the cluster in any order, all others have
// lower probabilities and at least top_k + 1 are here.  A thread each: exact top-k threshold, min-p, top-p (all by counting and by fixed-point sums over the
// candidates, the same sets as the descents over the vocabulary give) and the pick in index order.  The pick is warp 0's.
__device__ uint32_t finish_few(cg::cluster_group &cluster, SampShared &sh, uint32_t n, const SampleSettings &set, float inv_sum, float rnd) {
    static_assert(kFew <= 256, "its lists lie where the histograms were");
    uint32_t *bits = sh.kcnt[0], *token = sh.kcnt[1], *kept = sh.kcnt[2], *token_in_order = sh.kcnt[3];  // (nobody reads these any more)
    unsigned long long *mass = sh.psum[0];
    float *in_order = reinterpret_cast<float *>(sh.pcnt[0]);
    __shared__ uint32_t s_threshold, s_boundary;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    uint32_t c = 0;
    for (uint32_t o = 0; o < kSampCtas; o++) {
        const SampShared *from = cluster.map_shared_rank(&sh, o);
        const uint32_t m = from->n_cand;
        if (tid >= c && tid < c + m) {
            const uint2 e = from->cand[tid - c];
            bits[tid] = e.x;
            token[tid] = e.y;
        }
        c += m;
    }
    if (tid == 0) s_threshold = s_boundary = 0;
    __syncthreads();
    const bool mine = tid < c;
    const uint32_t b = mine ? bits[tid] : 0u, i = mine ? token[tid] : 0u;
    uint32_t place = 0;
    if (mine) {
        uint32_t above = 0, equal = 0;
        for (uint32_t j = 0; j < c; j++) {
            above += bits[j] > b;
            equal += bits[j] == b;
            place += token[j] < i;
        }
        if (above <= set.top_k && set.top_k < above + equal) s_threshold = b;  // (all that write it write the same)
    }
    __syncthreads();
    const float q = __uint_as_float(b);
    bool keep = mine && b != 0u && b >= s_threshold && (!(set.min_p > 0.0f) || q >= inv_sum * set.min_p);
    if (set.top_p < 1.0f) {
        const unsigned long long want = (unsigned long long)(set.top_p * kFixScale), f = (unsigned long long)(q * kFixScale);
        if (mine) {
            kept[tid] = keep ? b : 0u;
            mass[tid] = keep ? f : 0ull;
        }
        __syncthreads();
        unsigned long long above = 0;
        uint32_t ties = 0, before = 0;
        if (keep) {
            for (uint32_t j = 0; j < c; j++) {
                if (kept[j] > b) above += mass[j];
                if (kept[j] == b) {
                    ties++;
                    before += token[j] < i;
                }
            }
            if (above + ties * f >= want) atomicMax(&s_boundary, b);  // the mass reaches top_p with these
        }
        __syncthreads();
        if (keep && s_boundary) {
            if (b == s_boundary) {
                const unsigned long long need = want > above ? want - above : 0;
                uint32_t m = f ? (uint32_t)((need + f - 1) / f) : 1u;
                m = m < 1 ? 1u : m > ties ? ties : m;
                keep = before < m;
            } else {
                keep = b > s_boundary;
            }
        }
    }
    if (mine) {
        in_order[place] = keep ? q : 0.f;
        token_in_order[place] = i;
    }
    __syncthreads();
    if (tid >= 32) return 0;
    float total = 0.f;
    for (uint32_t j = lane; j < c; j += 32) total += in_order[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const float inv_total = 1.0f / total;
    float carry = 0.f;
    if (rnd <= 0.f) return 0;  // the first token reaches it
    for (uint32_t base = 0; base < c; base += 32) {
        const uint32_t j = base + lane;
        const float own = j < c ? in_order[j] : 0.f;
        float v = own * inv_total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float w = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= (uint32_t)o) v += w;
        }
        const uint32_t hit = __ballot_sync(0xffffffffu, carry + v >= rnd && own > 0.f);
        if (hit) return token_in_order[base + __ffs(hit) - 1];
        carry += __shfl_sync(0xffffffffu, v, 31);
    }
    return n - 1;
}

struct SampleParams {
    const float *logits;
    uint32_t n, slice;         // slice: vocabulary entries per CTA
    SampleSettings set;
    const SampleSettings *device_set;  // overrides `set` when present (replayed from a graph)
    const uint32_t *previous;  // tokens seen so far (prompt and picks)
    uint32_t n_previous;
    float r;                   // uniform random value in [0, 1)
    const float *r_values;     // device_set: value g of the stream, g = loop[0]
    uint32_t *loop;            // device_set: [0] picks made so far, [1] tokens before the first pick; [0] moves on
    float *probs;              // global memory for slices that do not fit shared memory, else null
    uint32_t *counts;
    uint32_t *out_token;       // the pick
    uint32_t *append_to;       // when set: the pick is also stored at append_to[n_previous] (the running token list)
    uint32_t *feed_state;      // when set: the pick is also stored at feed_state[0] (the runner's next input token)
};

__global__ void __cluster_dims__(kSampCtas, 1, 1) __launch_bounds__(kSampThreads) sample_kernel(const SampleParams p) {
    extern __shared__ float dyn[];
    __shared__ SampShared sh;
    __shared__ float red[32];
    __shared__ uint32_t redu[32];
    __shared__ unsigned long long tsum[256];
    __shared__ uint32_t tcnt[256];
    __shared__ uint32_t s_prefix, s_rank, s_take, s_have, s_first, s_upto;
    __shared__ unsigned long long s_carry;
    yule_pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t lo = rank * p.slice < p.n ? rank * p.slice : p.n, hi = lo + p.slice < p.n ? lo + p.slice : p.n, n = hi - lo;
    float *probs = p.probs ? p.probs + lo : dyn;
    uint32_t *counts = p.probs ? p.counts + lo : reinterpret_cast<uint32_t *>(dyn + p.slice);
    for (uint32_t i = tid; i < 1024; i += kSampThreads) {
        (&sh.kcnt[0][0])[i] = 0;
        (&sh.psum[0][0])[i] = 0;
        (&sh.pcnt[0][0])[i] = 0;
    }
    if (tid == 0) {
        s_first = 0xFFFFFFFFu;
        sh.n_cand = 0;
    }
    yule_pdl_wait();
    const SampleSettings set = p.device_set ? *p.device_set : p.set;
    const uint32_t n_previous = p.device_set ? p.loop[1] + p.loop[0] : p.n_previous;
    const float rnd = p.device_set ? p.r_values[p.loop[0]] : p.r;
    const bool penalise = set.repetition_penalty != 1.0f && n_previous > 0;
    const bool scale = set.temperature > 0.0f && set.temperature != 1.0f;
    const float inv_t = scale ? 1.0f / set.temperature : 1.0f;
    const float *logits = p.logits + lo;

    auto leave = [&](uint32_t pick) {
        if (rank == 0 && tid == 0) {
            *p.out_token = pick;
            if (p.append_to) p.append_to[n_previous] = pick;
            if (p.feed_state) p.feed_state[0] = pick;
            if (p.device_set) {
                p.feed_state[1] = n_previous;  // the position of the token just picked
                p.loop[0] += 1;
            }
        }
        cluster.sync();  // nobody leaves while its words may still be read; loop[0] moves on after everyone has read it (see above)
    };

    // occurrences of every token among the previous ones
    if (penalise) {
        for (uint32_t i = tid; i < n; i += kSampThreads) counts[i] = 0;
        __syncthreads();
        for (uint32_t j = tid; j < n_previous; j += kSampThreads) {
            const uint32_t t = p.previous[j];
            if (t >= lo && t < hi) atomicAdd(&counts[t - lo], 1u);
        }
        __syncthreads();
    }
    auto adjusted = [&](uint32_t i) { return adjusted_logit(logits, counts, i, set.repetition_penalty, penalise, inv_t, scale); };
    // softmax (sampler.rs:49-55)
    float mx = -FLT_MAX;
    for (uint32_t i = tid; i < n; i += kSampThreads) {
        const float l = adjusted(i);
        probs[i] = l;
        mx = fmaxf(mx, l);
    }
    mx = block_reduce_max(mx, red);
    if (tid == 0) sh.mx = mx;
    cluster.sync();
    for (uint32_t c = 0; c < kSampCtas; c++) mx = fmaxf(mx, cluster.map_shared_rank(&sh, c)->mx);
    float sum = 0.f;
    for (uint32_t i = tid; i < n; i += kSampThreads) {
        const float e = expf(probs[i] - mx);
        probs[i] = e;
        sum += e;
    }
    sum = block_reduce_sum(sum, red);
    if (tid == 0) sh.sum = sum;
    cluster.sync();
    sum = 0.f;
    for (uint32_t c = 0; c < kSampCtas; c++) sum += cluster.map_shared_rank(&sh, c)->sum;
    const float inv_sum = 1.0f / sum;
    for (uint32_t i = tid; i < n; i += kSampThreads) probs[i] *= inv_sum;
    __syncthreads();

    // top-k (sampler.rs:58-70): keep probs >= the value of rank k in descending order
    bool few = false;
    if (set.top_k > 0 && set.top_k < p.n) {
        // What bounds a call is its phases, each a barrier of the cluster, remote reads and a pass over the slice.  Where few tokens are left (few share the first sixteen
        // bits of a vocabulary's fortieth largest) the descent ends and one CTA finishes over them, with six barriers instead of thirteen: 128256 logits with the
        // default settings 55 -> 31 us in the token loop.  Not with a sum that is not finite, nor where min-p may leave nothing.
        const bool may = set.top_k < kFew && inv_sum <= FLT_MAX && !(set.min_p > 1.0f);
        if (tid == 0) {
            s_prefix = 0;
            s_rank = set.top_k;
        }
        __syncthreads();
        for (int pass = 0; pass < 4 && !few; pass++) {
            const int shift = 24 - 8 * pass;
            const uint32_t prefix = s_prefix, mask = pass == 0 ? 0u : 0xFFFFFFFFu << (shift + 8);
            for (uint32_t base = 0; base < n; base += kSampThreads) {
                const uint32_t i = base + tid, b = i < n ? __float_as_uint(probs[i]) : 0u;
                const uint32_t d = (i < n && (b & mask) == prefix) ? (b >> shift) & 255u : 256u;
                const uint32_t same = __match_any_sync(0xffffffffu, d);
                if (d < 256u && lane == (uint32_t)__ffs(same) - 1) atomicAdd(&sh.kcnt[pass][d], (uint32_t)__popc(same));
            }
            cluster.sync();
            if (tid < 256) {
                uint32_t v = 0;
                for (uint32_t c = 0; c < kSampCtas; c++) v += cluster.map_shared_rank(&sh, c)->kcnt[pass][tid];
                tcnt[tid] = v;
            }
            __syncthreads();
            if (wid == 0) {
                // lane i looks at bins 255 − 8i … 248 − 8i; the bin in which the rank falls
                uint32_t mine = 0;
                for (int q = 0; q < 8; q++) mine += tcnt[255 - 8 * lane - q];
                uint32_t incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= (uint32_t)o) incl += v;
                }
                const uint32_t want = s_rank;
                const uint32_t who = __ballot_sync(0xffffffffu, want < incl);
                const uint32_t sel = who ? __ffs(who) - 1 : 31;
                if (lane == sel) {
                    uint32_t rest = want - (incl - mine), d = 255 - 8 * lane;
                    for (int q = 0; q < 7 && rest >= tcnt[d]; q++) rest -= tcnt[d--];
                    s_rank = rest;
                    s_prefix = prefix | (d << shift);
                    s_upto = set.top_k - rest + tcnt[d];  // tokens of this bin and above it
                }
            }
            __syncthreads();
            few = may && s_upto <= kFew;
        }
        if (few) {
            const uint32_t from = s_prefix;
            for (uint32_t i = tid; i < n; i += kSampThreads) {
                const uint32_t b = __float_as_uint(probs[i]);
                if (b >= from) sh.cand[atomicAdd(&sh.n_cand, 1u)] = make_uint2(b, lo + i);
            }
            cluster.sync();
            leave(rank == 0 ? finish_few(cluster, sh, p.n, set, inv_sum, rnd) : 0u);
            return;
        }
        const float threshold = __uint_as_float(s_prefix);
        for (uint32_t i = tid; i < n; i += kSampThreads)
            if (!(probs[i] >= threshold)) probs[i] = 0.f;
        __syncthreads();
    }
    // min-p (sampler.rs:73-80): the largest probability is that of the largest logit, exp(0) / sum, and survives top-k
    if (set.min_p > 0.0f) {
        const float thr = inv_sum * set.min_p;
        for (uint32_t i = tid; i < n; i += kSampThreads)
            if (!(probs[i] >= thr)) probs[i] = 0.f;
        __syncthreads();
    }
    // top-p (sampler.rs:83-118)
    if (set.top_p < 1.0f) {
        const unsigned long long want = (unsigned long long)(set.top_p * kFixScale);
        if (tid == 0) {
            s_prefix = 0;
            s_carry = 0;
            s_take = s_have = 0xFFFFFFFFu;  // ties to keep at the boundary value; all of them unless the descent says otherwise
        }
        __syncthreads();
        bool all_in = false;
        for (int pass = 0; pass < 4 && !all_in; pass++) {
            const int shift = 24 - 8 * pass;
            const uint32_t prefix = s_prefix, mask = pass == 0 ? 0u : 0xFFFFFFFFu << (shift + 8);
            for (uint32_t i = tid; i < n; i += kSampThreads) {
                const float q = probs[i];
                const uint32_t b = __float_as_uint(q);
                if (q != 0.f && (b & mask) == prefix) {  // zeros carry no mass: they cannot be where it reaches top_p
                    atomicAdd(&sh.psum[pass][(b >> shift) & 255u], (unsigned long long)(q * kFixScale));
                    atomicAdd(&sh.pcnt[pass][(b >> shift) & 255u], 1u);
                }
            }
            cluster.sync();
            if (tid < 256) {
                unsigned long long v = 0;
                uint32_t k = 0;
                for (uint32_t c = 0; c < kSampCtas; c++) {
                    const SampShared *o = cluster.map_shared_rank(&sh, c);
                    v += o->psum[pass][tid];
                    k += o->pcnt[pass][tid];
                }
                tsum[tid] = v;
                tcnt[tid] = k;
            }
            __syncthreads();
            if (wid == 0) {
                unsigned long long mine = 0;
                for (int q = 0; q < 8; q++) mine += tsum[255 - 8 * lane - q];
                unsigned long long incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= (uint32_t)o) incl += v;
                }
                unsigned long long carry = s_carry + (incl - mine);
                int found = -1;
                for (int q = 0; q < 8 && found < 0; q++) {
                    const uint32_t d = 255 - 8 * lane - q;
                    if (tcnt[d] > 0 && carry + tsum[d] >= want)
                        found = (int)d;
                    else
                        carry += tsum[d];
                }
                const uint32_t who = __ballot_sync(0xffffffffu, found >= 0);
                if (!who) {
                    if (lane == 0) s_rank = 0xFFFFFFFFu;  // the mass never reaches top_p: every token stays (the reference never breaks)
                } else if (lane == (uint32_t)__ffs(who) - 1) {
                    const uint32_t d = (uint32_t)found;
                    s_rank = 0;
                    s_carry = carry;
                    s_prefix = prefix | (d << shift);
                    if (pass == 3) {
                        // tcnt[d] tokens share the boundary value v: the first m of them (index order) complete the nucleus
                        const unsigned long long v = tsum[d] / tcnt[d];
                        const unsigned long long need = want > carry ? want - carry : 0;
                        uint32_t m = v ? (uint32_t)((need + v - 1) / v) : 1u;
                        if (m < 1) m = 1;
                        if (m > tcnt[d]) m = tcnt[d];
                        s_take = m;
                        s_have = tcnt[d];
                    }
                }
            }
            __syncthreads();
            all_in = s_rank == 0xFFFFFFFFu;
        }
        if (!all_in) {
            const uint32_t vb = s_prefix, take = s_take;
            const bool split = take < s_have;  // the same in every CTA
            uint32_t seen = 0;                 // boundary-valued tokens before this chunk
            if (split) {
                uint32_t c = 0;
                for (uint32_t i = tid; i < n; i += kSampThreads) c += __float_as_uint(probs[i]) == vb ? 1u : 0u;
                uint32_t total;
                block_scan_inclusive_u32(c, redu, &total);
                if (tid == 0) sh.ties = total;
                cluster.sync();
                for (uint32_t o = 0; o < rank; o++) seen += cluster.map_shared_rank(&sh, o)->ties;
            }
            for (uint32_t base = 0; base < n; base += kSampThreads) {
                const uint32_t i = base + tid, b = i < n ? __float_as_uint(probs[i]) : 0u;
                bool keep = b >= vb;
                if (split) {
                    const uint32_t is_tie = (i < n && b == vb) ? 1u : 0u;
                    uint32_t total;
                    const uint32_t incl = block_scan_inclusive_u32(is_tie, redu, &total);
                    keep = b > vb || (is_tie && seen + incl <= take);
                    seen += total;
                    __syncthreads();
                }
                if (i < n && !keep) probs[i] = 0.f;
            }
            __syncthreads();
        }
    }
    // renormalise (sampler.rs:121-130).  Warp w owns the w-th run of consecutive entries of the slice from here on.
    const uint32_t seg = (n + 31) / 32, s0 = wid * seg < n ? wid * seg : n, s1 = s0 + seg < n ? s0 + seg : n;
    float wsum = 0.f;
    for (uint32_t i = s0 + lane; i < s1; i += 32) wsum += probs[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xffffffffu, wsum, o);
    if (lane == 0) red[wid] = wsum;
    __syncthreads();
    float before = 0.f, mine = 0.f;  // of this CTA: the warps before this one, all of them
    for (uint32_t w = 0; w < 32; w++) {
        if (w == wid) before = mine;
        mine += red[w];
    }
    if (tid == 0) sh.total = mine;
    cluster.sync();
    float total = 0.f, earlier = 0.f;
    for (uint32_t c = 0; c < kSampCtas; c++) {
        if (c == rank) earlier = total;
        total += cluster.map_shared_rank(&sh, c)->total;
    }
    uint32_t pick;
    if (!(total > 0.0f)) {
        // nothing left: argmax of the adjusted logits, ties to the highest index (sampler.rs:123-125, :150-163)
        float best = -FLT_MAX;
        uint32_t idx = 0;
        bool any = false;
        for (uint32_t i = tid; i < n; i += kSampThreads) {
            const float l = adjusted(i);
            if (!any || l >= best) {
                best = l;
                idx = i;
                any = true;
            }
        }
        const float bmax = block_reduce_max(any ? best : -FLT_MAX, red);
        __syncthreads();
        if (tid == 0) s_first = 0;
        __syncthreads();
        if (any && best == bmax) atomicMax(&s_first, idx);
        __syncthreads();
        if (tid == 0) {
            sh.best = n ? bmax : -FLT_MAX;
            sh.best_idx = lo + s_first;
        }
        cluster.sync();
        float top = -FLT_MAX;
        pick = 0;
        for (uint32_t c = 0; c < kSampCtas; c++) {
            const SampShared *o = cluster.map_shared_rank(&sh, c);
            if (c * p.slice < p.n && o->best >= top) {
                top = o->best;
                pick = o->best_idx;
            }
        }
    } else {
        // inverse CDF in index order (sampler.rs:166-183): the first token whose running sum reaches r, else the last.  A token
        // without mass does not move the reference's sum, so it is never the one (but for r = 0, which the first token reaches):
        // here the sums of a warp's start and of the end of the warp before may differ by a rounding, and r may fall between.
        const float inv_total = 1.0f / total;
        float carry = (earlier + before) * inv_total;
        if (carry + wsum * inv_total * 1.001f >= rnd) {  // (warps that cannot hold the crossing do not look)
            for (uint32_t base = s0; base < s1; base += 32) {
                const uint32_t i = base + lane;
                const float own = i < s1 ? probs[i] : 0.f;
                float q = own * inv_total;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float v = __shfl_up_sync(0xffffffffu, q, o);
                    if (lane >= (uint32_t)o) q += v;
                }
                const uint32_t hit = __ballot_sync(0xffffffffu, i < s1 && carry + q >= rnd && (own > 0.f || rnd <= 0.f));
                if (hit) {
                    if (lane == 0) atomicMin(&s_first, base + __ffs(hit) - 1);
                    break;
                }
                carry += __shfl_sync(0xffffffffu, q, 31);
            }
        }
        __syncthreads();
        if (tid == 0) sh.first = s_first == 0xFFFFFFFFu ? 0xFFFFFFFFu : lo + s_first;
        cluster.sync();
        pick = p.n - 1;
        for (uint32_t c = 0; c < kSampCtas; c++) {
            const uint32_t f = cluster.map_shared_rank(&sh, c)->first;
            if (f != 0xFFFFFFFFu) {
                pick = f;
                break;
            }
        }
    }
    leave(pick);
}

}  // namespace

cudaError_t launch_sample(const SampleArgs &a, cudaStream_t s, uint64_t *launches) {
    if (a.n == 0) return cudaErrorInvalidValue;
    SampleParams p = {};
    p.logits = a.logits;
    p.n = a.n;
    p.slice = (a.n + kSampCtas - 1) / kSampCtas;
    p.set = a.set;
    p.device_set = a.device_set;
    p.previous = a.previous;
    p.n_previous = a.n_previous;
    p.r = a.r;
    p.r_values = a.r_values;
    p.loop = a.loop;
    p.out_token = a.out_token;
    p.append_to = a.append_to;
    p.feed_state = a.feed_state;
    size_t smem = (size_t)p.slice * 8;
    if (smem > kSampMaxSmem) {
        p.probs = a.scratch;
        p.counts = reinterpret_cast<uint32_t *>(a.scratch + a.n);
        smem = 0;
    }
    static bool attr_done[64] = {};  // the opt-in for large dynamic shared memory belongs to the device
    static std::mutex mu;
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !attr_done[dev]) {
            e = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSampMaxSmem);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    *launches += 1;
    return launch_kernel(sample_kernel, dim3(kSampCtas), dim3(kSampThreads), smem, s, a.pdl, p);
}

}  // namespace yule
