// csrc/hp_overset_gpu.cu over a fake of the runtime calls that it makes on the
// host, no GPU: call number `fail_at` fails, and the fake notes what was still
// unfinished when the library function returned, and what the calls left
// behind in the device's default memory pool.  Built as a library for
// test_overset_exits.py.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cub/device/device_scan.cuh>
#include <map>

namespace fake {
int fail_at, call, pending, live, threshold_sets;
uint64_t threshold;
bool freed_since_sync;   // memory freed on the stream that no wait has given back yet
cudaError_t step() { return ++call == fail_at ? cudaErrorMemoryAllocation : cudaSuccess; }
cudaError_t malloc_async(void** p, size_t n, cudaStream_t) {
    cudaError_t e = step();
    if (e != cudaSuccess) return e;
    *p = std::malloc(n);
    live++;
    return e;
}
cudaError_t free_async(void* p, cudaStream_t) {
    std::free(p);
    live--;
    freed_since_sync = true;
    return cudaSuccess;
}
cudaError_t memcpy_async(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) {
    cudaError_t e = step();
    if (e == cudaSuccess) pending++;
    return e;
}
cudaError_t memset_async(void*, int, size_t, cudaStream_t) {
    cudaError_t e = step();
    if (e == cudaSuccess) pending++;
    return e;
}
cudaError_t sync(cudaStream_t) {
    freed_since_sync = false;
    if (pending == 0) return cudaSuccess;   // nothing to wait for, nothing to report
    pending = 0;
    return step();
}
cudaError_t create(cudaStream_t* st, unsigned) {
    cudaError_t e = step();
    if (e == cudaSuccess) *st = (cudaStream_t)0x10;
    return e;
}
cudaError_t destroy(cudaStream_t) { return cudaSuccess; }
cudaError_t last_error() { return step(); }
cudaError_t device(int* d) { *d = 0; return step(); }
cudaError_t pool(cudaMemPool_t* p, int) { *p = (cudaMemPool_t)0x20; return step(); }
cudaError_t pool_get(cudaMemPool_t, cudaMemPoolAttr, void* v) { *(uint64_t*)v = threshold; return step(); }
cudaError_t pool_set(cudaMemPool_t, cudaMemPoolAttr, void* v) {
    threshold = *(uint64_t*)v;
    threshold_sets++;
    return step();
}
struct DeviceScan {
    template <class T>
    static cudaError_t ExclusiveSum(void* tmp, size_t& bytes, const T*, T*, int, cudaStream_t) {
        cudaError_t e = step();
        if (tmp == nullptr) bytes = 1000;
        else if (e == cudaSuccess) pending++;
        return e;
    }
};
}  // namespace fake

#define cub fake
#define cudaMallocAsync(p, n, s) fake::malloc_async((void**)(p), n, s)
#define cudaFreeAsync fake::free_async
#define cudaMemcpyAsync fake::memcpy_async
#define cudaMemsetAsync fake::memset_async
#define cudaStreamSynchronize fake::sync
#define cudaStreamCreateWithFlags fake::create
#define cudaStreamDestroy fake::destroy
#define cudaGetLastError fake::last_error
#define cudaGetDevice fake::device
#define cudaDeviceGetDefaultMemPool fake::pool
#define cudaMemPoolGetAttribute fake::pool_get
#define cudaMemPoolSetAttribute fake::pool_set
#include "../multiphase-code_b200/csrc/hp_overset_gpu.cu"

extern "C" void fake_reset(int fail_at) {
    fake::fail_at = fail_at;
    fake::call = fake::pending = fake::live = fake::threshold_sets = 0;
    fake::threshold = 0;
    fake::freed_since_sync = false;
}
// calls made, operations unfinished, buffers not freed, pool settings changed,
// freed memory that no wait has let the pool give back
extern "C" void fake_report(int out[5]) {
    out[0] = fake::call; out[1] = fake::pending; out[2] = fake::live; out[3] = fake::threshold_sets;
    out[4] = fake::freed_since_sync;
}
