// gbReduceSumNoAlloc: the deterministic float64 sum of FvmFieldReduceSum for
// callers that cannot allocate device memory.
//
// Some callers cannot call cudaMalloc at the point where they need a
// reduction: hosts that hand out all device memory from their own pool and
// forbid other allocations, and plugins that must keep their device footprint
// fixed after setup.  The mesh/field entry points allocate their
// scratch (reduction partials, gradients) on first use; this entry point
// allocates nothing.  Its scratch -- a float64 partial sum per block and the
// calls' arrival counters -- lives in the file-scope array below, which every
// GPU that loads the library holds until the process exits.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

#include "gb_device.cuh"
#include "gb_internal.h"

namespace gb {
namespace {

// Partial sums: at most this many blocks of kNoAllocBlockItems inputs.
constexpr int kNoAllocPartials = 4096;                           // 32 KiB per GPU
constexpr int64_t kNoAllocBlockItems = (int64_t)kBlock * 8;      // inputs per block
constexpr int64_t kNoAllocMaxItems = (int64_t)kNoAllocPartials * kNoAllocBlockItems;   // 8,388,608
constexpr int kMaxDevices = 64;

// Arrival counters of the calls, taken in turn, after the partial sums.  What
// the blocks of a call add to its counter comes to zero (modulo 2^32), so a
// counter is at zero again once every call that used it has ended, even if
// calls overlapped on it (more than 64 in flight, or a captured call, which
// keeps its counter, replayed beside another): an overlap can spoil the
// results of the calls that overlap, never those of later ones.
constexpr int kCounters = 64;
static __device__ __align__(256) double g_noalloc_partials[kNoAllocPartials + kCounters];

constexpr int kSumThreads = 512;
constexpr int kSumMaxBlocks = 592;        // 444 resident at once (34 registers, three per SM), then the rest

__device__ __forceinline__ double sum_block(double x) {
    __shared__ double w[kSumThreads / 32];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) w[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < 32) {
        t = lane < kSumThreads / 32 ? w[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    }
    __syncthreads();
    return t;   // valid in thread 0
}

// The whole sum in one launch: each block sums its contiguous share (16-byte
// loads between the ragged ends), the last one to arrive sums the partials in
// block order.  The order of every addition depends on n and the alignment of
// v alone.  Bound by latency at these sizes: calls on 5 M values (20 MB) take
// 10.1 us one after another; as two launches with 4-byte loads they took 13.9.
__global__ void __launch_bounds__(kSumThreads) k_sum(int64_t n, const float* __restrict__ v, double* partials,
                                                     unsigned int* arrived, double* result) {
    __shared__ bool last;
    const int64_t head = min(n, (int64_t)((16 - (reinterpret_cast<uintptr_t>(v) & 15)) & 15) / 4);
    const int64_t n4 = (n - head) / 4;
    const float4* v4 = reinterpret_cast<const float4*>(v + head);
    const int64_t lo = n4 * blockIdx.x / gridDim.x, hi = n4 * (blockIdx.x + 1) / gridDim.x;
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
#pragma unroll 4
    for (int64_t i = lo + threadIdx.x; i < hi; i += kSumThreads) {
        const float4 x = __ldg(&v4[i]);
        a += (double)x.x;
        b += (double)x.y;
        c += (double)x.z;
        d += (double)x.w;
    }
    if (blockIdx.x == 0) {
        const int64_t tail = head + 4 * n4;
        if (threadIdx.x < head) a += (double)v[threadIdx.x];
        if (tail + threadIdx.x < n) b += (double)v[tail + threadIdx.x];
    }
    const double bs = sum_block((a + b) + (c + d));
    if (gridDim.x == 1) {
        if (threadIdx.x == 0) *result = bs;
        return;
    }
    if (threadIdx.x == 0) {
        // block 0 adds 1 - gridDim.x, the others 1: zero only when all have arrived
        const unsigned int add = blockIdx.x == 0 ? 1u - gridDim.x : 1u;
        partials[blockIdx.x] = bs;
        __threadfence();
        last = atomicAdd(arrived, add) + add == 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double s = 0.0;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kSumThreads) s += __ldcg(&partials[k]);
    const double t = sum_block(s);
    if (threadIdx.x == 0) *result = t;
}

// Device address of g_noalloc_partials, resolved once per device.  In host
// code the array's name is only a host-side stand-in for the symbol, so the
// kernels are given this address.  The cached address belongs to the
// device's current context: after cudaDeviceReset the module may load at
// another address, so a caller that resets a device must not use this entry
// point on it again in the same process.
std::mutex g_mu;
std::atomic<unsigned int> g_turn{0};
double* g_ptr[kMaxDevices] = {nullptr};

bool scratch_for_current_device(double** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_error(std::string("gbReduceSumNoAlloc: cudaGetDevice: ") + cudaGetErrorString(e));
        return false;
    }
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("gbReduceSumNoAlloc: device ordinal out of range");
        return false;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (e != cudaSuccess || !p) {
            set_error(std::string("gbReduceSumNoAlloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            return false;
        }
        g_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_ptr[dev];
    return true;
}

// Whether p is device (or managed) memory this context can write: a host
// pointer given here would be written through by the kernel.
bool device_pointer(const void* p) {
    cudaPointerAttributes a{};
    const cudaError_t e = cudaPointerGetAttributes(&a, p);
    if (e != cudaSuccess) {
        cudaGetLastError();   // the error is not sticky; clear it so later calls do not see it
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

}  // namespace
}  // namespace gb

using namespace gb;

extern "C" int gbReduceSumNoAlloc(const float* values, uint64_t n, double* result, void* stream) {
    clear_error();
    if (!values || !result || !device_pointer(values) || !device_pointer(result)) {
        set_error("gbReduceSumNoAlloc: values and result must be device (or managed) memory");
        return 1;
    }
    if (n > (uint64_t)kNoAllocMaxItems) {
        set_error("gbReduceSumNoAlloc: " + std::to_string(n) + " values exceed the maximum of " +
                  std::to_string(kNoAllocMaxItems) + " (" + std::to_string(kNoAllocPartials) +
                  " partial sums of " + std::to_string(kNoAllocBlockItems) + " values)");
        return 1;
    }
    double* partials = nullptr;
    if (!scratch_for_current_device(&partials)) return 1;
    cudaStream_t s = (cudaStream_t)stream;
    // a block per 2048 values, up to four per SM
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(kSumMaxBlocks, ((int64_t)n + kNoAllocBlockItems - 1) / kNoAllocBlockItems));
    k_sum<<<blocks, kSumThreads, 0, s>>>(
        (int64_t)n, values, partials, reinterpret_cast<unsigned int*>(partials + kNoAllocPartials + g_turn++ % kCounters),
        result);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("gbReduceSumNoAlloc: ") + cudaGetErrorString(e));
        return 1;
    }
    return 0;
}
