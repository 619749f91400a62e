// Device-side status word of the tensor-core kernels and the host-side hooks around it.
//
// Every barrier wait in the tcgen05 kernels has a cycle budget.  A CTA whose wait runs out
// raises the status word of its device, drains (no further data is touched), frees its TMEM
// and exits; CTAs that start afterwards see the word and drain at once, so a kernel that gave
// up never leaves work half done silently: the word stays set until the host clears it.
#include "tc_kernels.cuh"

#include "tc_plan.cuh"

#include <atomic>

namespace natten {

__device__ int g_tc_status = 0;

namespace {
std::mutex g_status_mutex;
int* g_status_addr[64] = {nullptr};
std::atomic<int*> g_status_host[64] = {};    // pinned, mapped: a kernel that gives up writes it itself
std::atomic<long long> g_wait_budget{tc::kWaitBudgetCycles};
std::atomic<int> g_inject{0};
} // namespace

namespace tcplan {

static cudaError_t current_device(int& dev)
{
    const cudaError_t err = cudaGetDevice(&dev);
    return err == cudaSuccess && (dev < 0 || dev >= 64) ? cudaErrorInvalidDevice : err;
}

cudaError_t status_ptr(int*& p)
{
    int dev = 0;
    cudaError_t err = current_device(dev);
    if (err != cudaSuccess) return err;
    std::lock_guard<std::mutex> lock(g_status_mutex);
    if (!g_status_addr[dev]) {
        void* word = nullptr;
        err = cudaGetSymbolAddress(&word, g_tc_status);
        if (err != cudaSuccess) return err;
        g_status_addr[dev] = static_cast<int*>(word);
    }
    p = g_status_addr[dev];
    return cudaSuccess;
}

cudaError_t status_host_ptr(int*& p)
{
    int dev = 0;
    cudaError_t err = current_device(dev);
    if (err != cudaSuccess) return err;
    p = g_status_host[dev].load(std::memory_order_acquire);
    if (p) return cudaSuccess;
    std::lock_guard<std::mutex> lock(g_status_mutex);
    p = g_status_host[dev].load(std::memory_order_acquire);
    if (!p) {
        void* word = nullptr;
        // the process's first call may be made while its stream is captured; allocating is no part of the graph
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        err = cudaThreadExchangeStreamCaptureMode(&mode);
        if (err != cudaSuccess) return err;
        err = cudaHostAlloc(&word, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (err != cudaSuccess) return err;
        p = static_cast<int*>(word);
        *p = 0;
        g_status_host[dev].store(p, std::memory_order_release);
    }
    return cudaSuccess;
}

long long debug_wait_budget() { return g_wait_budget.load(); }
int debug_inject() { return g_inject.load(); }

} // namespace tcplan

int tc_device_status()
{
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int)) != cudaSuccess) return -1;
    return v;
}

int tc_clear_status()
{
    const int zero = 0;
    int dev = 0;
    if (cudaDeviceSynchronize() == cudaSuccess && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64)
        if (int* w = g_status_host[dev].load(std::memory_order_acquire)) *static_cast<volatile int*>(w) = 0;
    return (int)cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int));
}

int tc_status_async(int* host_word, cudaStream_t s)
{
    if (!host_word) return (int)cudaErrorInvalidValue;
    int* p = nullptr;
    const cudaError_t err = tcplan::status_ptr(p);
    if (err != cudaSuccess) return (int)err;
    return (int)cudaMemcpyAsync(host_word, p, sizeof(int), cudaMemcpyDeviceToHost, s);
}

int tc_host_status(int device)
{
    if (device < 0 || device >= 64) return 0;
    int* w = g_status_host[device].load(std::memory_order_acquire);
    return w ? *static_cast<volatile int*>(w) : 0;
}

void tc_debug_wait(long long budget_cycles, int inject)
{
    g_wait_budget.store(budget_cycles > 0 ? budget_cycles : tc::kWaitBudgetCycles);
    g_inject.store(inject);
}

int tc_debug_inject() { return tcplan::debug_inject(); }

} // namespace natten
