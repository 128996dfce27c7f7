// qmv_q4k_mma.cu — Q4_K and Q5_K fused dequantise + matvec over two to four activation vectors per pass, weights streamed
// through registers (one vector: qmv_digits.cu; Q4_K where the activation image fits beside a ring: qmv_kquant_batch.cu).
//
// Exactness.  The contract is yule-core/src/dequant.rs:929-972:
//     sum += (d*sc_s) * Σ_l q_l x_l − (dmin*mn_s) * Σ_l x_l        per 32-column sub-block s.
// Operands are fed to the tensor core without rounding:
//   A (weights)  q·sc_s as fp16 — an integer ≤ 15·63 = 945, exact.  Built from the packed nibbles
//                as (1024+q)·sc − 1024·sc in one fp16 FMA (exact: the product fits in the FMA's
//                internal precision and the result is an integer < 2048).
//   B (x)        x·2^e split into hi = fp16(x·2^e) and lo = fp16(x·2^e − hi): two columns of the
//                8-wide B tile, summed after the MMA.  2^e normalises max|x| to [2^13, 2^14) so
//                neither overflow nor fp16 subnormals cost precision (error ≤ 2^-22 relative).
//   accumulate   fp32 in the MMA; d, dmin and 2^-e are applied in fp32 afterwards.
//   mins         one extra MMA per super-block: A = mn_s, B = Σ_l x_l of each sub-block (hi/lo).
// What differs from the CPU code is only the order of the fp32 additions.
//
// Mapping.  A CTA of 8 warps owns ROWS (16 or 8) consecutive rows; warp w takes super-blocks
// w, w+8, … of those rows.  Lane (g = lane/4, t = lane%4) holds rows g and g+8 and the 64-column
// group t of the super-block: 32 bytes of qs per row plus the 16-byte header — all 16-byte
// loads, issued for the warp's first super-block before anything else, the next super-block's
// while the current one is being multiplied.  The k index of the MMA is a free permutation
// (A and B agree on it), so nibbles go straight from the loaded words into fragments.
// Cross-warp sums go through 2 KB of shared memory in a fixed order (deterministic).
//
// The residual is added in the epilogue.  Programmatic dependent launch: weights do not depend on the previous kernel, so
// their loads are issued before `griddepcontrol.wait`; only the activation read waits.

#include <cstdlib>

#include <cuda_fp16.h>

#include "internal.h"

namespace yule {

namespace {

#include "q4k_mma_common.cuh"


struct Q4kMmaParams {
    const uint8_t *w;       // raw blocks
    float *out;             // [batch][out_stride]
    uint32_t n_rows, out_stride, n_tiles;
    const float *x;         // [batch][x_stride]
    uint32_t x_stride, n_cols, batch;
    const float *residual;  // same layout as out, or null
};

__device__ __forceinline__ void group_barrier(int group) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kWarps * 32) : "memory");
}

// Walks one warp's units in order: tile index k (of its group), super-block slot j; the row pointers are recomputed only
// when the tile changes.
template <int ROWS, bool Q5>
struct UnitCursor {
    static constexpr int NR = ROWS / 8;
    uint32_t k, j;
    const uint4 *rowp[NR];

    __device__ __forceinline__ void locate(const Q4kMmaParams &p, uint32_t first_tile, uint32_t tile_stride, uint32_t bpr,
                                           int g) {
        const uint32_t tile = first_tile + k * tile_stride;
#pragma unroll
        for (int r = 0; r < NR; r++) {
            uint32_t row = tile * ROWS + g + 8 * r;
            row = row < p.n_rows ? row : p.n_rows - 1;  // clamp: the load stays in bounds, the result is dropped
            rowp[r] = reinterpret_cast<const uint4 *>(p.w + (size_t)row * bpr * (Q5 ? 176 : 144));
        }
    }
    __device__ __forceinline__ void advance(const Q4kMmaParams &p, uint32_t first_tile, uint32_t tile_stride, uint32_t bpr,
                                            int g, uint32_t nbw) {
        if (++j == nbw) {
            j = 0;
            k++;
            locate(p, first_tile, tile_stride, bpr, g);
        }
    }
};

// Persistent kernel, one CTA per SM: CTA c owns tiles c, c+G, c+2G, … (G = gridDim.x), dealt
// alternately to its two 8-warp groups, so every SM gets the same number of tiles (±1) and at any
// moment the grid streams one contiguous region of the tensor.  Within a tile, warp w of the
// group multiplies super-blocks w, w+8, …; a warp's (tile, super-block) units form one
// sequence that is prefetched DEPTH units ahead.  The activations are staged once per CTA.
template <int ROWS, int DEPTH, bool Q5>
__global__ void __launch_bounds__(kThreadsCta, 1)
qmv_q4k_mma_kernel(const __grid_constant__ Q4kMmaParams p) {
    constexpr int NR = ROWS / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    yule_pdl_launch_dependents();

    const int lane = threadIdx.x & 31;
    const int group = threadIdx.x >> 8, wid = (threadIdx.x >> 5) & (kWarps - 1);
    const int g = lane >> 2, t = lane & 3;
    const uint32_t bpr = p.n_cols / 256;
    const uint32_t nbw = bpr > (uint32_t)wid ? (bpr - wid + kWarps - 1) / kWarps : 0;  // super-blocks per tile for this warp
    const uint32_t G = gridDim.x;
    // tiles of this CTA: blockIdx.x + i*G; group takes i = group, group + 2, …
    const uint32_t first_tile = blockIdx.x + group * G, tile_stride = kGroups * G;
    const uint32_t my_tiles = p.n_tiles > first_tile ? (p.n_tiles - first_tile + tile_stride - 1) / tile_stride : 0;
    constexpr uint32_t tiles_per_round = kRoundSlots;

    const SmemLayout sm = carve(smem_raw, p.n_cols, p.batch);
    float *partial = sm.partial + (size_t)group * kRoundSlots * kWarps * 4 * 16;

    UnitCursor<ROWS, Q5> ld_cur;
    ld_cur.k = ld_cur.j = 0;
    const uint32_t total_units = my_tiles * nbw;
    uint32_t issued = 0;
    BlockLoads buf[DEPTH][NR];
    if (total_units) {
        ld_cur.locate(p, first_tile, tile_stride, bpr, g);
#pragma unroll
        for (int i = 0; i < DEPTH; i++) {
            if (issued < total_units) {
                issue_loads<NR, Q5>(buf[i], ld_cur.rowp, wid + kWarps * ld_cur.j, t);
                issued++;
                if (issued < total_units) ld_cur.advance(p, first_tile, tile_stride, bpr, g, nbw);
            }
        }
    }

    yule_pdl_wait();  // own weight loads are in flight; the activations come from the kernel before
    stage_activations<false>(sm, p.x, p.x_stride, p.n_cols, p.batch, nullptr, 0.f);
    // B column n = g: vector n/2, part n%2.  Lanes whose vector does not exist read vector 0;
    // their output columns are never looked at.
    const uint32_t vec = (uint32_t)(g >> 1) < p.batch ? (g >> 1) : 0;
    const uint4 *xb_lane = sm.xb + (size_t)vec * (p.n_cols / 4) + (g & 1) * 4 + t;
    const uint32_t *sb_lane = sm.sb + (size_t)vec * (p.n_cols / 32) + (g & 1) * 4 + t;

    // Cross-warp sums of the tiles [k0, k0+kn) of this group, then the epilogue.  Every warp of
    // the group calls this once per round.
    auto finish_round = [&](uint32_t k0, uint32_t kn) {
        group_barrier(group);
        const uint32_t n_warps_used = bpr < (uint32_t)kWarps ? bpr : kWarps;
        const uint32_t tid = threadIdx.x & (kWarps * 32 - 1);
        for (uint32_t idx = tid; idx < kn * 64; idx += kWarps * 32) {
            const uint32_t kk = idx >> 6, v = (idx >> 4) & 3, rr = idx & 15;
            if (v >= p.batch || rr >= ROWS) continue;
            const uint32_t row = (first_tile + (k0 + kk) * tile_stride) * ROWS + rr;
            if (row >= p.n_rows) continue;
            float sum = 0.f;  // fixed order over the warps: deterministic
            for (uint32_t w2 = 0; w2 < n_warps_used; w2++) sum += partial[((kk * kWarps + w2) * 4 + v) * 16 + rr];
            sum *= sm.inv_scale[v];
            const size_t o = (size_t)v * p.out_stride + row;
            p.out[o] = p.residual ? sum + p.residual[o] : sum;
        }
        group_barrier(group);
    };

    if (nbw == 0) {
        // more warps than super-blocks per row: this warp only helps with the reductions
        for (uint32_t k0 = 0; k0 < my_tiles; k0 += tiles_per_round)
            finish_round(k0, (my_tiles - k0) < tiles_per_round ? (my_tiles - k0) : tiles_per_round);
    } else {

    float acc[NR][2];
#pragma unroll
    for (int r = 0; r < NR; r++) acc[r][0] = acc[r][1] = 0.f;
    uint32_t k0 = 0, kn = my_tiles < tiles_per_round ? my_tiles : tiles_per_round;
    uint32_t in_slot = 0, slot = 0;  // super-blocks done in the current tile; slots done in the round
    // unit n lives in buf[n % DEPTH]; the loop is unrolled by DEPTH so the ring index is static
    for (uint32_t base = 0; base < total_units; base += DEPTH) {
#pragma unroll
        for (int i = 0; i < DEPTH; i++) {
            if (base + i < total_units) {
                consume_block<NR, Q5>(buf[i], wid + kWarps * in_slot, t, xb_lane, sb_lane, acc);
                if (issued < total_units) {
                    issue_loads<NR, Q5>(buf[i], ld_cur.rowp, wid + kWarps * ld_cur.j, t);
                    issued++;
                    if (issued < total_units) ld_cur.advance(p, first_tile, tile_stride, bpr, g, nbw);
                }
                if (++in_slot == nbw) {
                    // lane (g, t) holds, for vector t, rows g (and g+8): hi-column + lo-column sums
#pragma unroll
                    for (int r = 0; r < NR; r++) {
                        partial[((slot * kWarps + wid) * 4 + t) * 16 + g + 8 * r] = acc[r][0] + acc[r][1];
                        acc[r][0] = acc[r][1] = 0.f;
                    }
                    in_slot = 0;
                    if (++slot == kn) {
                        finish_round(k0, kn);
                        k0 += kn;
                        kn = (my_tiles - k0) < tiles_per_round ? (my_tiles - k0) : tiles_per_round;
                        slot = 0;
                    }
                }
            }
        }
    }
    }  // nbw != 0

}

template <int ROWS, int DEPTH, bool Q5>
cudaError_t launch_variant(const Q4kMmaParams &p, int sm_count, size_t smem, bool pdl, cudaStream_t s) {
    auto kern = qmv_q4k_mma_kernel<ROWS, DEPTH, Q5>;
    // per instantiation: the opt-in for large dynamic shared memory
    // (the attribute belongs to the device, not the process: one flag per device ordinal)
    static bool attr_done[64] = {};
    static std::mutex mu;
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !attr_done[dev]) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    // one CTA per SM; fewer when there are not enough tiles to give every group one
    uint32_t grid = (uint32_t)sm_count;
    const uint32_t want = (p.n_tiles + kGroups - 1) / kGroups;
    if (grid > want) grid = want;
    return launch_kernel(kern, dim3(grid), dim3(kThreadsCta), smem, s, pdl, p);
}

}  // namespace

bool q4k_mma_supported(uint32_t n_cols, uint32_t batch) {
    return n_cols % 256 == 0 && batch >= 1 && batch <= 4 && smem_bytes(n_cols, batch) <= 200 * 1024;
}

cudaError_t launch_q4k_mma(const Q4kBatch &f, int sm_count, cudaStream_t s, uint64_t *launches) {
    if (f.rows == 0) return cudaSuccess;
    Q4kMmaParams p = {};
    // Tile height.  16-row tiles use the whole MMA and half the instructions per byte of 8-row tiles; they win
    // as soon as they keep about 60 % of the warp groups busy (measured: 4096 rows, 256 tiles for 296 groups,
    // 10-25 % faster with 16; 2048 rows, 128 tiles, faster with 8).
    const uint32_t n_groups = (uint32_t)kGroups * (uint32_t)sm_count;
    const int tile_rows = ((f.rows / 16) * 10 >= n_groups * 6) ? 16 : 8;
    p.w = f.w;
    p.out = f.out;
    p.n_rows = f.rows;
    p.out_stride = f.out_stride;
    p.n_tiles = (f.rows + tile_rows - 1) / tile_rows;
    p.x = f.x;
    p.x_stride = f.x_stride;
    p.n_cols = f.n_cols;
    p.batch = f.batch;
    p.residual = f.residual;
    const size_t smem = smem_bytes(f.n_cols, f.batch);
    cudaError_t e;
    if (f.q5)
        e = tile_rows == 8 ? launch_variant<8, 4, true>(p, sm_count, smem, f.pdl, s) : launch_variant<16, 2, true>(p, sm_count, smem, f.pdl, s);
    else
        e = tile_rows == 8 ? launch_variant<8, 4, false>(p, sm_count, smem, f.pdl, s) : launch_variant<16, 2, false>(p, sm_count, smem, f.pdl, s);
    if (e != cudaSuccess) return e;
    *launches += 1;
    return cudaSuccess;
}

}  // namespace yule
