// attn_cluster.cu — decode attention of one query per sequence, a thread-block cluster per (KV head, sequence).
//
// What it computes is the per-head loop of yule-infer/src/model_runner.rs:672-758 for all query heads of a KV head, with the
// rotation of q and of the new K row and the append of the new K / V rows folded in (gpu_runner.rs:422-499), as
// attn_decode_gqa_kernel does (attn_gqa.cuh: sliding window, soft-cap, fused mode have the meaning given there).
//
// What bounds it: at the contexts of a chat a layer's K and V rows are a few hundred KB, and the time is a chain of
// latencies.  So everything that does not depend on the launch before goes out ahead of `griddepcontrol.wait` (the position, the
// rotation table, the first tiles of K and V), the positions are dealt over the CTAs of a cluster, and the CTAs' sums meet in
// each other's shared memory behind one cluster barrier; the split kernel's partial sums went through global memory, a fence, a
// ticket and two more passes of loads.  At long contexts it is a stream: tiles of 32 positions through a ring of asynchronous
// copies, running maximum and sum per head.
//
// Measured, us by which the launch moves the end of a token step on, against the split kernel this replaced there: 1.1B shape (32 heads of 64
// on 4) at 50 positions 7.8 -> 3.9, at 100 7.8 -> 4.1, at 1930 15.0 -> 8.9; 8B shape (32 of 128 on 8) at 50 9.4 -> 4.5, at 130 9.6 -> 5.6.  Not for the many
// queries of a prompt: per position it takes more instructions than the splits (runner.cu has the line).
//
// Every warp has four rows of a tile to itself, from the copy to the weighted sum, with a running maximum of its own, so the
// stream has no CTA barrier; 16000 positions of the 8B shape take 35 us (3.7 TB/s), 42 with three barriers a tile.
//
// Each CTA pushes its sums for output element e to the CTA that owns e, so nobody reads another CTA's memory after the
// barrier and every CTA may leave when it is done.

#include <cfloat>
#include <mutex>

#include "internal.h"

namespace yule {

namespace {

#include "attn_gqa.cuh"
#include "tp_pairs.cuh"

constexpr uint32_t kTile = 32;        // positions per tile: eight warps of four
constexpr uint32_t kMaxRanks = kAttnMaxRanks;  // CTAs of a cluster
// Tiles per CTA from which another cluster joins in.  us per token and layer, heads of 64, two against four: 1.1B shape at 1930 positions 10.3, 12.0, at
// 430 9.9, 9.7.  Heads of 128, two, three, four (8B shape with a narrow feed-forward, whole layer): at 300 positions 31.2, 30.6, 30.7, at 500 31.6, 32.4, 32.7, at 1500
// 33.3, 34.4, 35.5, at 4000 the same: three is right up to some 400 positions, two would be beyond.
constexpr uint32_t cluster_tiles(uint32_t hd) { return hd == 64 ? 2u : 3u; }
constexpr int kWarps = kThreads / 32;
template <int HD>
constexpr uint32_t kMaxTileStages = HD == 64 ? 6 : 3;  // 96 KB: two CTAs to an SM

template <int HD>
constexpr uint32_t kStageFloats = 2 * kTile * HD;  // K rows, then V rows
// shared memory behind the tile ring, in floats: queries, new K and V row, weights, factors, maxima and sums of the warps, mailbox
template <int GROUP, int HD>
constexpr uint32_t kFixedFloats = GROUP * HD + 2 * HD + kWarps * 4 * GROUP + kWarps * 8 + kWarps * 16 + 16 + GROUP * HD + 2 * GROUP * kMaxRanks;

__device__ __forceinline__ uint32_t smem_at(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t rank, float v) {
    asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %0, %1;\n\tst.shared::cluster.f32 [a], %2;\n\t}" ::"r"(addr), "r"(rank), "f"(v) : "memory");
}

// GROUP floats from an address aligned to all of them
template <int GROUP>
__device__ __forceinline__ void load_group(const float *from, float (&to)[GROUP]) {
    if constexpr (GROUP % 4 == 0) {
#pragma unroll
        for (int h = 0; h < GROUP; h += 4) *reinterpret_cast<float4 *>(to + h) = *reinterpret_cast<const float4 *>(from + h);
    } else {
#pragma unroll
        for (int h = 0; h < GROUP; h++) to[h] = from[h];
    }
}

template <int GROUP, int HD, bool TP>
__global__ void __launch_bounds__(kThreads, 2) attn_cluster_kernel(const __grid_constant__ AttnParams p, const uint32_t stages) {
    constexpr int J = HD / 32;                             // 16-byte steps per lane and row
    constexpr int GH = GROUP * J > 16 ? 16 / J : GROUP;    // query heads scored together (their values are registers)
    constexpr int HD4 = HD / 4;
    constexpr uint32_t kOut = GROUP * HD;
    extern __shared__ __align__(16) float sm[];
    yule_pdl_launch_dependents();
    uint32_t rank, ranks;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(ranks));
    const uint32_t kvh = blockIdx.y, z = blockIdx.z, head0 = kvh * GROUP, tid = threadIdx.x;
    const uint32_t cluster = blockIdx.x >> (31 - __clz(ranks));
    const int lane = tid & 31, wid = tid >> 5, qtr = lane >> 3, l8 = lane & 7;
    if (!p.settled) yule_pdl_wait();

    float *tiles = sm;
    float *qs = tiles + (size_t)stages * kStageFloats<HD>;  // GROUP x HD rotated queries
    float *kcur = qs + kOut, *vcur = kcur + HD;             // the current token's rotated K row and its V row
    float *weights = vcur + HD;                             // [warp][position of four][GROUP]
    float *factor = weights + kWarps * 4 * GROUP;           // [warp][head]: what the sums so far are multiplied by
    float *wml = factor + kWarps * 8;                       // [warp][head] (maximum, sum)
    float *cta_ml = wml + kWarps * 16;                      // [head] (maximum, sum)
    float *mail = cta_ml + 16;                              // [rank][share of the outputs]
    float *stats = mail + kOut;                             // [rank][head] (maximum, sum)

    const uint32_t pos = p.pos_ptr ? p.pos_ptr[p.pos_per_query ? z : 0] : p.seq_len - 1 + z;
    const uint32_t seq = pos + 1;
    float *const k_cache = p.k_cache + (size_t)z * p.kv_batch_stride + (size_t)kvh * HD;
    float *const v_cache = p.v_cache + (size_t)z * p.kv_batch_stride + (size_t)kvh * HD;
    const bool fused = p.k_new != nullptr;
    const uint32_t first_visible = (p.window && pos >= p.window) ? pos - p.window : 0;
    const uint32_t begin = p.softcap != 0.f ? 0u : first_visible;  // (attn_gqa_unit: why masked positions are visited under a soft-cap)
    // clusters at work at this length; the others leave (all their CTAs alike)
    const uint32_t span = seq - begin, per_cluster = ranks * p.min_chunk;
    uint32_t eff = (span + per_cluster - 1) / per_cluster;
    eff = eff < p.n_splits ? eff : p.n_splits;
    if (cluster >= eff) return;
    if (ranks > 1) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");  // waited for before the first remote store
    const uint32_t parts = eff * ranks, chunk = (span + parts - 1) / parts, part = cluster * ranks + rank;
    const uint32_t lo = begin + part * chunk < seq ? begin + part * chunk : seq;
    const uint32_t hi = lo + chunk < seq ? lo + chunk : seq;
    const uint32_t n_tiles = (hi - lo + kTile - 1) / kTile;

    // This warp's four rows of tile i into its slot; the current token's row is not in the cache yet.  One group of copies per call,
    // empty past the end.
    const uint32_t c4 = lane % HD4 * 4, r0 = wid * 4 + lane / HD4, row0_smem = smem_at(tiles + r0 * HD + c4);
    size_t off = (size_t)(lo + r0) * p.kv_stride + c4;  // of this lane's first element of the next tile
    uint32_t t = lo + r0, fetch_slot = 0;
    auto fetch = [&]() {
        if (t < hi) {
            const uint32_t to = row0_smem + fetch_slot * (kStageFloats<HD> * 4);
#pragma unroll
            for (uint32_t k = 0; k < 4; k += 32 / HD4) {
                if (t + k < hi && !(fused && t + k == pos)) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + k * HD * 4), "l"(k_cache + off + (size_t)k * p.kv_stride) : "memory");
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + (kTile + k) * HD * 4), "l"(v_cache + off + (size_t)k * p.kv_stride) : "memory");
                }
            }
        }
        off += (size_t)kTile * p.kv_stride;
        t += kTile;
        if (++fetch_slot == stages) fetch_slot = 0;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (uint32_t i = 0; i + 1 < stages || i == 0; i++) fetch();  // stages - 1 tiles ahead (one stage: the only tile)

    // RoPE as in apply_rope (model_runner.rs:277-293): products and sums rounded separately.
    constexpr int QIT = (GROUP * (HD / 2) + kThreads - 1) / kThreads;
    float rot_c[QIT], rot_s[QIT];
#pragma unroll
    for (int it = 0; it < QIT; it++) {
        const uint32_t idx = tid + it * kThreads;
        rot_c[it] = 1.f, rot_s[it] = 0.f;
        if (p.cos_table && idx < GROUP * (HD / 2)) {
            rot_c[it] = p.cos_table[(size_t)pos * (HD / 2) + idx % (HD / 2)];
            rot_s[it] = p.sin_table[(size_t)pos * (HD / 2) + idx % (HD / 2)];
        }
    }
    if (p.settled) yule_pdl_wait();  // from here on the outputs of the launch before are read
    const float *q_in = p.q + (size_t)z * p.q_stride + (size_t)head0 * HD;
    const float *k_new = fused ? p.k_new + (size_t)z * p.kv_stride + (size_t)kvh * HD : nullptr;
    const float *v_new = fused ? p.v_new + (size_t)z * p.kv_stride + (size_t)kvh * HD : nullptr;
    const bool owner = fused && pos >= lo && pos < hi;  // of the current position
    float v_row = 0.f;
    if (owner && tid < HD) v_row = v_new[tid];
#pragma unroll
    for (int it = 0; it < QIT; it++) {
        const uint32_t idx = tid + it * kThreads;
        if (idx >= GROUP * (HD / 2)) break;
        const uint32_t i = idx % (HD / 2);
        float q0 = q_in[2 * idx], q1 = q_in[2 * idx + 1], k0 = 0.f, k1 = 0.f;
        const bool with_k = owner && idx < HD / 2;
        if (with_k) k0 = k_new[2 * i], k1 = k_new[2 * i + 1];
        if (p.cos_table) {
            const float c = rot_c[it], s = rot_s[it];
            const float r0 = __fsub_rn(__fmul_rn(q0, c), __fmul_rn(q1, s)), r1 = __fadd_rn(__fmul_rn(q0, s), __fmul_rn(q1, c));
            const float r2 = __fsub_rn(__fmul_rn(k0, c), __fmul_rn(k1, s)), r3 = __fadd_rn(__fmul_rn(k0, s), __fmul_rn(k1, c));
            q0 = r0, q1 = r1, k0 = r2, k1 = r3;
        }
        qs[2 * idx] = q0;
        qs[2 * idx + 1] = q1;
        if (with_k) {
            kcur[2 * i] = k0;
            kcur[2 * i + 1] = k1;
            k_cache[(size_t)pos * p.kv_stride + 2 * i] = k0;
            k_cache[(size_t)pos * p.kv_stride + 2 * i + 1] = k1;
        }
    }
    if (owner && tid < HD) {
        vcur[tid] = v_row;
        v_cache[(size_t)pos * p.kv_stride + tid] = v_row;
    }

    __syncthreads();  // queries and new rows are there; from here to the end of the stream every warp is on its own

    const float scale = 1.0f / sqrtf((float)HD);
    float4 acc[GROUP];
#pragma unroll
    for (int h = 0; h < GROUP; h++) acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    float m_run = -FLT_MAX, l_run = 0.f;  // lane (qtr, l8): maximum of head l8, its sum over every fourth position
    uint32_t slot = 0;
    for (uint32_t i = 0; i < n_tiles; i++) {
        // this warp's rows of tile i are here (those of later tiles may be on their way), and all its lanes are done with tile i - 1
        if (stages < 3) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else if (stages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (stages == 5) asm volatile("cp.async.wait_group 3;" ::: "memory");
        else asm volatile("cp.async.wait_group 4;" ::: "memory");
        __syncwarp();
        if (stages > 1) fetch();
        const uint32_t t0 = lo + i * kTile + wid * 4;
        if (t0 >= hi) break;
        const uint32_t live = hi - t0;  // of the warp's four positions
        const float *kt = tiles + (size_t)slot * kStageFloats<HD> + wid * 4 * HD, *vt = kt + kTile * HD;
        if (++slot == stages) slot = 0;
        // scores: eight lanes per position, 16 bytes each per step; lane l8 of a position keeps head l8
        const uint32_t tq = t0 + qtr;
        const float *krow = (fused && tq == pos) ? kcur : kt + qtr * HD;
        float4 kv[J];
#pragma unroll
        for (int j = 0; j < J; j++) kv[j] = *reinterpret_cast<const float4 *>(krow + j * 32 + l8 * 4);
        float sc = 0.f;
#pragma unroll
        for (int h0 = 0; h0 < GROUP; h0 += GH) {
            float d[GH];
#pragma unroll
            for (int h = 0; h < GH; h++) {
                float a0 = 0.f, a1 = 0.f;
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const float4 q = *reinterpret_cast<const float4 *>(qs + (h0 + h) * HD + j * 32 + l8 * 4);
                    a0 = fmaf(q.x, kv[j].x, a0);
                    a1 = fmaf(q.y, kv[j].y, a1);
                    a0 = fmaf(q.z, kv[j].z, a0);
                    a1 = fmaf(q.w, kv[j].w, a1);
                }
                d[h] = a0 + a1;
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < GH; h++) d[h] += __shfl_xor_sync(0xffffffffu, d[h], o);
#pragma unroll
            for (int h = 0; h < GH; h++) sc = l8 == h0 + h ? d[h] : sc;
        }
        sc *= scale;
        if (p.softcap != 0.f) sc = tq < first_visible ? -p.softcap : p.softcap * tanhf(sc / p.softcap);
        // running soft-max of the warp
        const bool valid = qtr < live;
        float mx = valid ? sc : -FLT_MAX;
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        mx = fmaxf(mx, m_run);
        const float e = valid ? expf(sc - mx) : 0.f, f = expf(m_run - mx);
        l_run = fmaf(l_run, f, e);
        m_run = mx;
        float *w = weights + wid * 4 * GROUP;
        if (l8 < GROUP) {
            w[qtr * GROUP + l8] = e;
            if (qtr == 0) factor[wid * 8 + l8] = f;
        }
        const bool rescale = __any_sync(0xffffffffu, l8 < GROUP && f != 1.f);
        __syncwarp();
        if (rescale) {
#pragma unroll
            for (int h = 0; h < GROUP; h++) {
                const float fh = factor[wid * 8 + h];
                acc[h].x *= fh, acc[h].y *= fh, acc[h].z *= fh, acc[h].w *= fh;
            }
        }
        // sums of e · V for all heads from one read of V
#pragma unroll
        for (uint32_t k = 0; k < 4; k += 32 / HD4) {
            const uint32_t rv = k + lane / HD4;
            if (rv < live) {
                const float4 v = *reinterpret_cast<const float4 *>(((fused && t0 + rv == pos) ? vcur : vt + rv * HD) + c4);
                float ew[GROUP];
                load_group<GROUP>(w + rv * GROUP, ew);
#pragma unroll
                for (int h = 0; h < GROUP; h++) {
                    const float eh = ew[h];
                    acc[h].x = fmaf(eh, v.x, acc[h].x);
                    acc[h].y = fmaf(eh, v.y, acc[h].y);
                    acc[h].z = fmaf(eh, v.z, acc[h].z);
                    acc[h].w = fmaf(eh, v.w, acc[h].w);
                }
            }
        }
    }
    // the warps meet, in the ring: nobody still reads it, and every copy that was started has been waited for
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 8);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 16);
    if (qtr == 0) {
        wml[(wid * 8 + l8) * 2] = m_run;
        wml[(wid * 8 + l8) * 2 + 1] = l_run;
    }
    if (HD4 < 32) {
#pragma unroll
        for (int h = 0; h < GROUP; h++) {
            acc[h].x += __shfl_xor_sync(0xffffffffu, acc[h].x, 16);
            acc[h].y += __shfl_xor_sync(0xffffffffu, acc[h].y, 16);
            acc[h].z += __shfl_xor_sync(0xffffffffu, acc[h].z, 16);
            acc[h].w += __shfl_xor_sync(0xffffffffu, acc[h].w, 16);
        }
    }
    __syncthreads();
    // thread (head, warp): the weight of the warp's sums, and the CTA's maximum and sum of the head
    if (tid < 8 * kWarps) {
        const uint32_t h = tid / kWarps, w = tid % kWarps;
        const float2 ml = *reinterpret_cast<const float2 *>(wml + (w * 8 + h) * 2);
        float M = ml.x;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        const float ww = ml.y == 0.f ? 0.f : expf(ml.x - M);  // (a warp without positions; a NaN stays one)
        float L = ml.y * ww;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        factor[h * kWarps + w] = ww;
        if (w == 0) {
            cta_ml[2 * h] = M;
            cta_ml[2 * h + 1] = L;
        }
    }
    float *partial = tiles;  // [warp][GROUP][HD] = 8 · GROUP · HD floats <= one stage (64 · HD)
    if (lane < HD4) {
#pragma unroll
        for (int h = 0; h < GROUP; h++) *reinterpret_cast<float4 *>(partial + (wid * GROUP + h) * HD + c4) = acc[h];
    }
    __syncthreads();
    const uint32_t share_log2 = 31 - __clz(kOut) - (31 - __clz(ranks)), share = 1u << share_log2;  // outputs per CTA
    if (ranks > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // every CTA of the cluster has started
#pragma unroll
    for (uint32_t k = 0; k < (kOut + kThreads - 1) / kThreads; k++) {
        const uint32_t idx = tid + k * kThreads;
        if (idx < kOut) {
            float ww[kWarps], o = 0.f;
            load_group<kWarps>(factor + idx / HD * kWarps, ww);
#pragma unroll
            for (int w = 0; w < kWarps; w++) o = fmaf(ww[w], partial[w * kOut + idx], o);
            if (ranks > 1) st_cluster(smem_at(mail + rank * share + (idx & (share - 1))), idx >> share_log2, o);
            else mail[idx] = o;
        }
    }
    if (tid < 2 * GROUP * ranks) {
        const uint32_t to = tid / (2 * GROUP), e = tid % (2 * GROUP);
        if (ranks > 1) st_cluster(smem_at(stats + rank * 2 * GROUP + e), to, cta_ml[e]);
        else stats[e] = cta_ml[e];
    }
    if (ranks > 1) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else {
        __syncthreads();
    }
    float *out = p.out + (size_t)z * p.out_stride;
    auto store = [&](uint32_t idx, float v) {
        out[(size_t)head0 * HD + idx] = v;
        if (TP && p.tp.push) tp_push_value(p.tp, (size_t)head0 * HD + idx, v);
    };
    // several clusters: their sums and statistics go through global memory, element by element to the last one there
    float *acc_of = p.scratch + (size_t)z * p.n_heads * p.n_splits * (HD + 2);  // [head][cluster][HD]
    float2 *stat_of = reinterpret_cast<float2 *>(acc_of + (size_t)p.n_heads * p.n_splits * HD);  // [head][cluster]
    for (uint32_t i = tid; i < share; i += kThreads) {
        const uint32_t idx = rank * share + i, h = idx / HD;
        float M = -FLT_MAX;
        for (uint32_t c = 0; c < ranks; c++) M = fmaxf(M, stats[(c * GROUP + h) * 2]);
        float L = 0.f, O = 0.f;
        for (uint32_t c = 0; c < ranks; c++) {  // in the order of the positions
            const float l = stats[(c * GROUP + h) * 2 + 1], w = l > 0.f ? expf(stats[(c * GROUP + h) * 2] - M) : 0.f;
            L = fmaf(l, w, L);
            O = fmaf(mail[c * share + i], w, O);
        }
        if (eff == 1) {
            store(idx, O * (1.0f / L));
        } else {
            const size_t at = (size_t)(head0 + h) * p.n_splits + cluster;
            acc_of[at * HD + idx % HD] = O;
            // every CTA writes the statistics of the heads it merges; CTAs that share a head write the same values
            if (idx % HD == 0 || i == 0) stat_of[at] = make_float2(M, L);
        }
    }
    if (eff == 1) return;
    __shared__ uint32_t s_last;
    __threadfence();
    __syncthreads();
    uint32_t *ticket = p.tickets + ((size_t)z * p.n_kv_heads + kvh) * kMaxRanks + rank;
    if (tid == 0) s_last = atomicAdd(ticket, 1u) == eff - 1 ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t i = tid; i < share; i += kThreads) {
        const uint32_t idx = rank * share + i;
        const size_t at = (size_t)(head0 + idx / HD) * p.n_splits;
        float M = -FLT_MAX, L = 0.f, O = 0.f;
        for (uint32_t c0 = 0; c0 < eff; c0 += 4) {  // four loads in flight; running maximum, in the order of the positions
            float2 st[4];
            float o[4];
#pragma unroll
            for (uint32_t c = 0; c < 4; c++) {
                const bool there = c0 + c < eff;
                st[c] = there ? __ldcg(stat_of + at + c0 + c) : make_float2(-FLT_MAX, 0.f);
                o[c] = there ? __ldcg(acc_of + (at + c0 + c) * HD + idx % HD) : 0.f;
            }
            float m4 = M;
#pragma unroll
            for (uint32_t c = 0; c < 4; c++) m4 = fmaxf(m4, st[c].x);
            const float back = expf(M - m4);
            L *= back, O *= back, M = m4;
#pragma unroll
            for (uint32_t c = 0; c < 4; c++) {
                const float w = st[c].y > 0.f ? expf(st[c].x - M) : 0.f;
                L = fmaf(st[c].y, w, L);
                O = fmaf(o[c], w, O);
            }
        }
        store(idx, O * (1.0f / L));
    }
    if (tid == 0) *ticket = 0;  // ready for the next launch on this stream
}

template <int GROUP, int HD>
cudaError_t launch_cluster_variant(const AttnParams &p, uint32_t ranks, uint32_t stages, uint32_t n_seq, bool pdl, cudaStream_t s) {
    auto kern = p.tp.push ? attn_cluster_kernel<GROUP, HD, true> : attn_cluster_kernel<GROUP, HD, false>;
    const size_t smem = ((size_t)stages * kStageFloats<HD> + kFixedFloats<GROUP, HD>) * sizeof(float);
    // the opt-in for large dynamic shared memory belongs to the device and is asked for once
    static bool attr_done[2][64] = {};
    static std::mutex mu;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        bool *done = dev >= 0 && dev < 64 ? &attr_done[p.tp.push ? 1 : 0][dev] : nullptr;
        if (!done || !*done) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)((kMaxTileStages<HD> * kStageFloats<HD> + kFixedFloats<GROUP, HD>) * sizeof(float)));
            if (e != cudaSuccess) return e;
            if (done) *done = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ranks * p.n_splits, p.n_kv_heads, n_seq);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, p, stages);
}

}  // namespace

// CTAs of a cluster, and clusters per (KV head, query): up to 256 CTAs in all, as many as two to an SM find room for whatever
// the GPC (288 of them, in clusters of four, ran in two waves: 4096 positions of the 8B shape 22 us instead of 15).
//   A launch of known length takes clusters of eight (8B shape, 250 positions 5.1 us, clusters of four 6.2).  In a chain of dependent
// launches eight CTAs of one GPC become free later than four: per token 1.1B shape at 100 positions 0.3 us a layer for four, 8B 0.7;
// sixteen cost 1.1 us more than four.
void attn_cluster_shape(uint32_t units, uint32_t hd, uint32_t max_seq_len, bool known_length, int sm_count, uint32_t *ranks, uint32_t *clusters) {
    uint32_t c = 1;
    const uint32_t most = known_length ? kMaxRanks : 4;
    while (c < most && units * c * 2 <= (uint32_t)sm_count && c * 8 < max_seq_len) c *= 2;
    uint32_t n = 256 / (units * c ? units * c : 1);
    const uint32_t per = c * cluster_tiles(hd) * kTile, by_len = (max_seq_len + per - 1) / per;
    n = n < by_len ? n : by_len;
    *ranks = c;
    *clusters = n < 1 ? 1 : n > 16 ? 16 : n;
}

cudaError_t launch_attn_cluster(const AttnDecode &a, int sm_count, cudaStream_t s, uint64_t *launches) {
    if (!attn_gqa_supported(a.hd, a.n_heads, a.n_kv_heads) || a.kv_stride % 4) return cudaErrorInvalidValue;
    // several queries: consecutive positions of one cache, which they only read, or each with a position, a cache and new rows of its own
    if (a.n_tokens > 1 && (a.k_new || a.pos_ptr) && !a.pos_per_query) return cudaErrorInvalidValue;
    if (a.n_tokens > 1 && a.k_new && !a.kv_batch_stride) return cudaErrorInvalidValue;
    AttnParams p = {};
    p.q = a.q;
    p.k_new = a.k_new;
    p.v_new = a.v_new;
    p.k_cache = a.k_cache;
    p.v_cache = a.v_cache;
    p.cos_table = a.cos_table;
    p.sin_table = a.sin_table;
    p.pos_ptr = a.pos_ptr;
    p.seq_len = a.seq_len;
    p.out = a.out;
    p.hd = a.hd;
    p.n_heads = a.n_heads;
    p.n_kv_heads = a.n_kv_heads;
    p.kv_stride = a.kv_stride;
    p.window = a.window;
    p.softcap = a.softcap;
    p.pos_per_query = a.pos_per_query ? 1u : 0u;
    p.kv_batch_stride = a.kv_batch_stride;
    p.q_stride = a.q_stride;
    p.out_stride = a.out_stride;
    p.tp = a.tp;
    p.settled = a.settled ? 1u : 0u;
    const uint32_t g = a.n_heads / a.n_kv_heads, units = a.n_kv_heads * a.n_tokens;
    uint32_t ranks, clusters;
    attn_cluster_shape(units, a.hd, a.max_seq_len, !a.pos_ptr, sm_count, &ranks, &clusters);
    if (clusters > 1 && (!a.scratch || !a.tickets || a.n_splits < clusters)) clusters = a.scratch && a.tickets && a.n_splits ? a.n_splits : 1;
    p.n_splits = clusters;
    p.min_chunk = cluster_tiles(a.hd) * kTile;
    p.scratch = a.scratch;
    p.tickets = a.tickets;
    const uint32_t parts = ranks * clusters, most = (a.max_seq_len + parts - 1) / parts;  // positions of a CTA where all clusters work
    uint32_t stages = (most + kTile - 1) / kTile;
    stages = stages < cluster_tiles(a.hd) ? cluster_tiles(a.hd) : stages;
    if (stages * kTile > a.max_seq_len) stages = (a.max_seq_len + kTile - 1) / kTile;
    const uint32_t limit = a.hd == 64 ? kMaxTileStages<64> : kMaxTileStages<128>;
    stages = stages > limit ? limit : stages;
    *launches += 1;
#define YULE_GQA_CASE(G, H) if (g == G && a.hd == H) return launch_cluster_variant<G, H>(p, ranks, stages, a.n_tokens, a.pdl, s)
    YULE_GQA_CASE(1, 64); YULE_GQA_CASE(2, 64); YULE_GQA_CASE(4, 64); YULE_GQA_CASE(8, 64);
    YULE_GQA_CASE(1, 128); YULE_GQA_CASE(2, 128); YULE_GQA_CASE(4, 128); YULE_GQA_CASE(8, 128);
#undef YULE_GQA_CASE
    return cudaErrorInvalidValue;
}

}  // namespace yule
