// q6k_planar.cu — the row-planar device copy of a Q6_K tensor.
//
// A Q6_K super-block is 210 bytes (ql[128] qh[64] scales[16] d[2]) and only 2-byte aligned in the GGUF stream, which rules
// out both wide loads and bulk copies (16-byte granular).  The device keeps, next to the raw tensor, the same bytes
// regrouped row by row: every block's ql of the row, then every block's qh, then the scales, then the d values (padded to
// a multiple of 16 bytes).  Any run of blocks that starts at a multiple of eight is then four 16-byte-aligned contiguous
// pieces.  Same values, 210 bytes per block plus at most 14 bytes per row; built once per tensor.

#include "internal.h"

namespace yule {

namespace {

__host__ __device__ inline uint32_t d_section_bytes(uint32_t bpr) { return (bpr * 2 + 15) & ~15u; }
__host__ __device__ inline size_t row_record_bytes(uint32_t bpr) { return (size_t)bpr * 208 + d_section_bytes(bpr); }

__global__ void repack_q6k_rows_kernel(const uint8_t *__restrict__ raw, uint8_t *__restrict__ planar, uint64_t n_rows, uint32_t bpr) {
    const size_t rec = row_record_bytes(bpr);
    const uint32_t dsec = d_section_bytes(bpr);
    const uint64_t per_row = (uint64_t)bpr * 104 + dsec / 2;  // 16-bit pieces of a row record (blocks are 2-byte aligned)
    const uint64_t total = n_rows * per_row;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t row = i / per_row;
        const uint32_t o = (uint32_t)(i - row * per_row) * 2;  // byte offset inside the record
        const uint8_t *src_row = raw + row * bpr * 210;
        unsigned short v = 0;
        if (o < bpr * 128) {
            v = *reinterpret_cast<const unsigned short *>(src_row + (size_t)(o / 128) * 210 + (o % 128));
        } else if (o < bpr * 192) {
            const uint32_t q = o - bpr * 128;
            v = *reinterpret_cast<const unsigned short *>(src_row + (size_t)(q / 64) * 210 + 128 + (q % 64));
        } else if (o < bpr * 208) {
            const uint32_t q = o - bpr * 192;
            v = *reinterpret_cast<const unsigned short *>(src_row + (size_t)(q / 16) * 210 + 192 + (q % 16));
        } else {
            const uint32_t q = (o - bpr * 208) / 2;  // block index; the tail of the section is padding
            if (q < bpr) v = *reinterpret_cast<const unsigned short *>(src_row + (size_t)q * 210 + 208);
        }
        *reinterpret_cast<unsigned short *>(planar + row * rec + o) = v;
    }
}

}  // namespace

size_t q6k_planar_bytes(uint64_t n_rows, uint32_t n_cols) { return (size_t)n_rows * row_record_bytes(n_cols / 256) + 256; }
size_t q6k_planar_row_bytes(uint32_t n_cols) { return row_record_bytes(n_cols / 256); }

cudaError_t launch_q6k_repack(const uint8_t *raw, uint8_t *planar, uint64_t n_rows, uint32_t n_cols, cudaStream_t s,
                              uint64_t *launches) {
    if (n_rows == 0) return cudaSuccess;
    repack_q6k_rows_kernel<<<148 * 8, 256, 0, s>>>(raw, planar, n_rows, n_cols / 256);
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace yule
