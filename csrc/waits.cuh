// Bounded waits on shared-memory barriers, with a flag per translation unit.
#pragma once
#include "common.cuh"

namespace dlp {

static __device__ int g_gemm_wait_expired;      // a bounded wait ran into its limit (dlp_gemm_wait_expired)

// After the limit the flag is set and every later wait gives up after a short try, so the kernel runs to its end, frees its tensor memory
// and returns (with wrong results).
template <bool CLUSTER = false>
__device__ __forceinline__ void mbar_wait_b(uint64_t* bar, uint32_t parity) {
    for (unsigned spins = 0; !(CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)); ++spins) {
        if ((spins & 1023u) == 1023u && *reinterpret_cast<volatile int*>(&g_gemm_wait_expired) != 0) return;
        if (spins > (1u << 22)) { atomicExch(&g_gemm_wait_expired, 1); return; }
    }
}
static inline int gemm_wait_flag(int* out) {      // this translation unit's flag (current device)
    int v = 0;
    DLP_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_gemm_wait_expired, sizeof(int)));
    *out |= v;
    return 0;
}
__device__ __forceinline__ void gemm_wait_aftermath() {
    if (threadIdx.x == 0 && *reinterpret_cast<volatile int*>(&g_gemm_wait_expired) != 0)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);       // a wait gave up: copies in flight land before the block goes away
}

}  // namespace dlp
