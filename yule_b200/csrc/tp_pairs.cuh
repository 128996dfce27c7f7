// tp_pairs.cuh — the two ends of a gathered vector's (value, epoch) pairs under tensor parallelism (TpFuse in
// internal.h).  Include inside namespace yule { namespace { … } }.
#pragma once

// Kept out of line: the tensor-parallel path must not cost the single-GPU kernels registers.
__device__ __noinline__ void tp_push_value(const TpFuse &tp, size_t o, float v) {
    const uint2 pair = make_uint2(__float_as_uint(v), *tp.tick * tp.epochs_per_tick + tp.push_index + 1u);
    for (uint32_t pp = 0; pp < tp.world; pp++)  // one 8-byte store each
        asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(tp.pair_out[pp] + o), "r"(pair.x), "r"(pair.y) : "memory");
}
// Eight consecutive elements of a gathered vector from its (value, epoch) pairs: polls until all eight
// carry `epoch`.  Bounded, and bounded once per failure: the first wait that runs out of `budget` cycles
// writes the status word, and every wait that starts (or polls) after that returns at once, so a lost peer
// costs one budget per kernel in flight, not one per wait.  The values returned after a give-up are
// whatever the buffer held; the host reads the status word and discards the step.
__device__ __forceinline__ void tp_load8(const uint2 *pairs, uint32_t epoch, int *status, long long budget, float (&a)[8]) {
    long long t0 = 0;
    for (uint32_t it = 0;; it++) {
        uint4 q[4];
        // one 16-byte load per two pairs: value and epoch of a pair must come from the same access
#pragma unroll
        for (int i = 0; i < 4; i++)
            asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(q[i].x), "=r"(q[i].y), "=r"(q[i].z), "=r"(q[i].w)
                         : "l"(pairs + 2 * i)
                         : "memory");
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 4; i++) ok = ok && q[i].y == epoch && q[i].w == epoch;
        if (!ok) {
            if (it == 0) t0 = clock64();
            if (it != 0 && (it & 63u) != 63u) continue;
            if (*reinterpret_cast<volatile int *>(status) == 0) {
                if (clock64() - t0 < budget) continue;
                atomicCAS(status, 0, kStatusPeerTimeout);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            a[2 * i] = __uint_as_float(q[i].x);
            a[2 * i + 1] = __uint_as_float(q[i].z);
        }
        return;
    }
}
