// The status of bounded waits (waits.cuh): one word in host memory for all kernels and devices of the process.
#include "waits.cuh"

#include <mutex>
#include <set>
#include <vector>

#include "../include/dlp_b200.h"

namespace dlp {

static std::vector<WaitUnit>& wait_units() { static std::vector<WaitUnit> units; return units; }
bool wait_register(const WaitUnit& u) { wait_units().push_back(u); return true; }

static std::mutex g_mu;
static std::set<int> g_watched;                       // devices whose kernels know the word
static int* g_word = nullptr;                         // pinned, mapped
static long long g_limit = WAIT_CLOCKS * 2;

static int each_unit(int (*f)(const WaitUnit&, void*), void* arg) {
    for (const WaitUnit& u : wait_units())
        if (int rc = f(u, arg)) return rc;
    return 0;
}
static int set_unit(const WaitUnit& u, void*) { return u.set(g_word, g_limit); }
static int get_unit(const WaitUnit& u, void* out) { return u.get((int*)out); }
static int clear_unit(const WaitUnit& u, void*) { return u.clear(); }

static int watch_device() {                           // (g_mu held)
    int dev = 0;
    DLP_CHECK_CUDA(cudaGetDevice(&dev));
    if (g_word == nullptr) {
        int* w = nullptr;
        DLP_CHECK_CUDA(cudaHostAlloc((void**)&w, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
        *w = 0;
        g_word = w;
    }
    if (g_watched.count(dev)) return 0;
    if (int rc = each_unit(set_unit, nullptr)) return rc;
    g_watched.insert(dev);
    return 0;
}

// One wait that nothing ends, for trying what a caller sees of it
__global__ void wait_probe_kernel() {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        mbar_wait_b(&bar, 0);
    }
}

}  // namespace dlp

using namespace dlp;

extern "C" {

int dlp_wait_watch(const volatile int32_t** word) {
    DLP_REQUIRE(word, "dlp_wait_watch: null argument");
    std::lock_guard<std::mutex> lock(g_mu);
    if (int rc = watch_device()) return rc;
    *word = g_word;
    return 0;
}

int dlp_set_wait_limit(double seconds) {
    DLP_REQUIRE(seconds > 0 && seconds <= 3600, "dlp_set_wait_limit: %g seconds", seconds);
    std::lock_guard<std::mutex> lock(g_mu);
    if (int rc = watch_device()) return rc;
    g_limit = (long long)(seconds * WAIT_CLOCKS);
    return each_unit(set_unit, nullptr);
}

int dlp_gemm_wait_expired(int* out) {
    DLP_REQUIRE(out, "dlp_gemm_wait_expired: null argument");
    *out = 0;
    return each_unit(get_unit, out);
}

int dlp_wait_status(int* out) {
    DLP_REQUIRE(out, "dlp_wait_status: null argument");
    *out = 0;
    DLP_CHECK_CUDA(cudaDeviceSynchronize());
    std::lock_guard<std::mutex> lock(g_mu);
    int dev = 0;
    DLP_CHECK_CUDA(cudaGetDevice(&dev));
    if (g_watched.count(dev)) *out = *(volatile int*)g_word;
    else if (int rc = each_unit(get_unit, out)) return rc;
    if (*out == 0) return 0;
    if (int rc = each_unit(clear_unit, nullptr)) return rc;
    for (int other : g_watched) {                     // (which device it was, the word does not say)
        if (other == dev) continue;
        DLP_CHECK_CUDA(cudaSetDevice(other));
        const cudaError_t e = cudaDeviceSynchronize();
        const int rc = e == cudaSuccess ? each_unit(clear_unit, nullptr) : -1;
        DLP_CHECK_CUDA(cudaSetDevice(dev));
        if (rc) return rc;
    }
    if (g_word) *(volatile int*)g_word = 0;
    return 0;
}

int dlp_wait_probe(void* stream) {
    wait_probe_kernel<<<1, 32, 0, (cudaStream_t)stream>>>();
    DLP_LAUNCH_CHECK();
    return 0;
}

}  // extern "C"
