// readback.cu — small results to the host.
//
// A host that drives the layers itself reads a vector back after every few launches, and what that costs is not the transfer (22 KB
// over PCIe are 0.5 us) but its dressing: a copy on a copy engine, which has to be told by the launch queue, and a wait for the
// whole stream.  Up to kReadBackBytes a kernel on the same stream stores the bytes into host memory itself, behind a matvec as its
// dependent launch, and writes an epoch behind them that the host polls.  What bounds it is the trip over PCIe that a system-wide fence waits for: with two
// fences per CTA, and a second driver query for the destination, pinned memory was slower than the copy engine on every call behind anything but a matvec.
//   us, copy engine, two fences, one: idle stream, 16 KB pinned 12.5, 13.8, 11.6, pageable 15.7, 14.6, 12.3; 512 KB pinned 21.6, 25.4, 21.0, 1 MB 30.7, 35.2, 30.8
// (beyond it, the copy engine).  5632x2048 matvec and its result 22.0, 18.4, 16.5; 4096x14336 by four rows 33.7, 33.2, 28.9; RMSNorm of 5632 values and its
// result 19.1, 17.8, 15.8.  What a trip costs depends on the host: on another one the 5632x2048 matvec took 21.7 and, with two fences, 21.2.

#include <atomic>
#include <chrono>
#include <cstring>

#include <cuda.h>

#include "internal.h"

namespace yule {

namespace {

constexpr uint32_t kThreads = 256;
constexpr size_t kFlagOffset = kReadBackBytes;  // the epoch lies behind the landing area, in a line of its own

// n bytes (both addresses multiples of 16); the last CTA to have stored its share writes the epoch.
__global__ void __launch_bounds__(kThreads) read_back_kernel(const unsigned char *src, unsigned char *dst, uint32_t n, uint32_t *ticket, uint32_t *flag, uint32_t epoch) {
    yule_pdl_launch_dependents();
    yule_pdl_wait();
    const uint32_t first = blockIdx.x * kThreads + threadIdx.x, step = gridDim.x * kThreads;
    for (uint32_t i = first; i < n / 16; i += step) reinterpret_cast<uint4 *>(dst)[i] = __ldcg(reinterpret_cast<const uint4 *>(src) + i);
    if (first < (n & 15u)) dst[(n & ~15u) + first] = __ldcg(src + (n & ~15u) + first);
    __syncthreads();
    if (threadIdx.x == 0) {
        // The CTAs meet on the device; one fence of the last of them, which a trip to the host takes, then orders all their stores before the epoch.
        bool last = true;
        if (gridDim.x > 1) {
            __threadfence();
            last = atomicAdd(ticket, 1u) == gridDim.x - 1;
            if (last) *ticket = 0;  // for the next launch on this stream
        }
        if (last) {
            __threadfence_system();
            *reinterpret_cast<volatile uint32_t *>(flag) = epoch;
        }
    }
}

__global__ void set_words_kernel(uint32_t *at, uint32_t a, uint32_t b) {
    at[0] = a;
    at[1] = b;
}

// Whether the n bytes at `data` are host memory that is not managed, by one driver query.  `view`: the device's view of them where a kernel may store there, all
// n inside one allocation or registration that the device may write (stores to memory registered read-only, or past a registration, would fault), else null.
bool host_destination(void *data, size_t n, unsigned char **view) {
    typedef CUresult (*QueryFn)(unsigned int, CUpointer_attribute *, void **, CUdeviceptr);
    static const QueryFn query = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &fn, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            fn = nullptr;
        }
        return reinterpret_cast<QueryFn>(fn);
    }();
    unsigned int type = 0, managed = 0, access = 0;
    CUdeviceptr device = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute which[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
                                   CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE, CU_POINTER_ATTRIBUTE_ACCESS_FLAGS};
    void *values[] = {&type, &managed, &device, &start, &size, &access};
    const CUdeviceptr at = reinterpret_cast<CUdeviceptr>(data);
    *view = nullptr;
    if (!query || query(6, which, values, at) != CUDA_SUCCESS || managed || (type != 0 && type != CU_MEMORYTYPE_HOST)) return false;
    // (type 0: pageable memory, of which CUDA knows nothing; the range is in host addresses)
    if (type != 0 && device && access == CU_POINTER_ATTRIBUTE_ACCESS_FLAG_READWRITE && at >= start && n <= size && at - start <= size - n)
        *view = reinterpret_cast<unsigned char *>(device);
    return true;
}

}  // namespace

cudaError_t read_back_create(yule_cuda_ctx *ctx) {
    cudaError_t e = cudaHostAlloc((void **)&ctx->rb_host, kReadBackBytes + 128, cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&ctx->rb_device, ctx->rb_host, 0);
    if (e == cudaSuccess) e = cudaMalloc((void **)&ctx->rb_ticket, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(ctx->rb_ticket, 0, sizeof(uint32_t));
    if (e == cudaSuccess) memset(ctx->rb_host + kFlagOffset, 0, 128);
    return e;
}
void read_back_destroy(yule_cuda_ctx *ctx) {
    if (ctx->rb_host) cudaFreeHost(ctx->rb_host);
    if (ctx->rb_ticket) cudaFree(ctx->rb_ticket);
}

// The stream's work so far is over and its bytes are in `data` when this returns.  Calls of several threads take turns: landing area,
// ticket and epoch are one set.
cudaError_t read_back(yule_cuda_ctx *ctx, const void *src, void *data, size_t n, bool pdl) {
    unsigned char *view = nullptr;
    if (n == 0 || n > kReadBackBytes || ctx->capturing || (reinterpret_cast<uintptr_t>(src) & 15) || !host_destination(data, n, &view)) {
        cudaError_t e = n ? cudaMemcpyAsync(data, src, n, cudaMemcpyDeviceToHost, ctx->stream) : cudaSuccess;
        return e == cudaSuccess ? cudaStreamSynchronize(ctx->stream) : e;
    }
    std::lock_guard<std::mutex> lock(ctx->rb_mu);
    unsigned char *direct = (reinterpret_cast<uintptr_t>(data) & 15) == 0 ? view : nullptr;
    const uint32_t epoch = ++ctx->rb_epoch, grid = (uint32_t)(n < 64 * 4096 ? (n + 4095) / 4096 : 64);
    volatile uint32_t *flag = reinterpret_cast<volatile uint32_t *>(ctx->rb_host + kFlagOffset);
    cudaError_t e = launch_kernel(read_back_kernel, dim3(grid), dim3(kThreads), 0, ctx->stream, pdl, (const unsigned char *)src, direct ? direct : ctx->rb_device,
                                  (uint32_t)n, ctx->rb_ticket, reinterpret_cast<uint32_t *>(ctx->rb_device + kFlagOffset), epoch);
    if (e != cudaSuccess) return e;
    // Poll for as long as a short chain of launches takes; whoever waits for more waits for the stream, which also brings its errors.
    const auto t0 = std::chrono::steady_clock::now();
    for (uint32_t it = 1; *flag != epoch; it++) {
        if ((it & 63u) == 0 && std::chrono::steady_clock::now() - t0 > std::chrono::microseconds(500)) {
            e = cudaStreamSynchronize(ctx->stream);
            if (e != cudaSuccess) return e;
            if (*flag != epoch) return cudaErrorUnknown;  // (the stream is over, so the store has been made)
            break;
        }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    if (!direct) memcpy(data, ctx->rb_host, n);
    return cudaSuccess;
}

cudaError_t launch_set_words(uint32_t *at, uint32_t a, uint32_t b, cudaStream_t s) {
    set_words_kernel<<<1, 1, 0, s>>>(at, a, b);
    return cudaGetLastError();
}

}  // namespace yule
