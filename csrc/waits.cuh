// Bounded waits on shared-memory barriers.  A wait that lasts longer than the limit (2 s unless dlp_set_wait_limit says otherwise; counted from its
// own first tries, so kernels that start ahead of their predecessor's end wait for that first) raises a status and returns, and every later wait
// gives up after a short try: the kernel runs to its end, frees its tensor memory and returns, with wrong results.  The status is a word of this
// translation unit on the device and one in host memory (dlp_wait_watch) that costs the host a load; dlp_wait_status clears both.
#pragma once
#include "common.cuh"

namespace dlp {

constexpr long long WAIT_CLOCKS = 2000000000ll;        // of an SM in a second, at most (a limit is no shorter than it says)
static __device__ int g_wait_expired;                 // a wait of this unit's kernels ran out
static __device__ int* g_wait_host;                   // the host's word, once somebody watches it
static __device__ long long g_wait_limit = WAIT_CLOCKS * 2;

struct WaitUnit { int (*set)(int* host_word, long long limit); int (*get)(int* out); int (*clear)(); };      // on the current device
bool wait_register(const WaitUnit& u);                // (waits.cu)
static int wait_unit_set(int* host_word, long long limit) {
    DLP_CHECK_CUDA(cudaMemcpyToSymbol(g_wait_host, &host_word, sizeof(host_word)));
    DLP_CHECK_CUDA(cudaMemcpyToSymbol(g_wait_limit, &limit, sizeof(limit)));
    return 0;
}
static int wait_unit_get(int* out) {
    int v = 0;
    DLP_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_wait_expired, sizeof(int)));
    *out |= v;
    return 0;
}
static int wait_unit_clear() {
    const int zero = 0;
    DLP_CHECK_CUDA(cudaMemcpyToSymbol(g_wait_expired, &zero, sizeof(int)));
    return 0;
}
static const bool g_wait_registered = wait_register({wait_unit_set, wait_unit_get, wait_unit_clear});

__device__ __forceinline__ bool wait_gives_up(long long& since) {
    const long long now = clock64();                   // (of this SM: it does not step back)
    if (since == 0) since = now;
    if (*reinterpret_cast<volatile int*>(&g_wait_expired) != 0) return true;
    if (now - since <= *reinterpret_cast<volatile long long*>(&g_wait_limit)) return false;
    atomicExch(&g_wait_expired, 1);
    if (int* host = *reinterpret_cast<int* volatile*>(&g_wait_host)) {
        *reinterpret_cast<volatile int*>(host) = 1;
        __threadfence_system();
    }
    return true;
}
template <bool CLUSTER = false>
__device__ __forceinline__ void mbar_wait_b(uint64_t* bar, uint32_t parity) {
    long long since = 0;
    for (unsigned tries = 1; !(CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)); ++tries)
        if ((tries & 63u) == 0 && wait_gives_up(since)) return;
}
__device__ __forceinline__ void gemm_wait_aftermath() {
    if (threadIdx.x == 0 && *reinterpret_cast<volatile int*>(&g_wait_expired) != 0)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);       // a wait gave up: copies in flight land before the block goes away
}

}  // namespace dlp
