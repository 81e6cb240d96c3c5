// util.cuh -- device-wide primitives used by setup and planning: exclusive scans
// and a stable LSD radix sort (64-bit keys, 32-bit values).
#pragma once

#include "hmg_internal.cuh"
#include "../../include/hmg.h"

namespace hmg {

// The library's own stream-ordered pool on the current device (null if it cannot be
// created: the device's default pool then serves).  While handles live it keeps up to
// POOL_KEEP freed bytes mapped; the last handle's destruction gives them back.  The
// default pool, which other code may share and whose settings stay untouched, unmaps
// everything free at every synchronisation: about 0.2 ms to map and 0.2 ms to unmap a
// small block, 6.3 ms a GB each way (measured on a B200), in a setup that synchronises
// some twenty times.  Thread-safe.  A cudaDeviceReset ends the pool with its context: the
// next use makes another, and handles of the old context (their generation) no longer count.
static constexpr unsigned long long POOL_KEEP = 1ull << 30;
cudaMemPool_t device_pool();
unsigned pool_retain(int device);  // the current device; returns the pool's generation (0: no pool)
void pool_release(int device, unsigned generation);

// Stream-ordered device allocation helpers.
template <typename T>
hmg_status dalloc(T** p, size_t count, cudaStream_t s)
{
    *p = nullptr;
    if (count == 0) count = 1;
    const cudaMemPool_t pool = device_pool();
    cudaError_t e = pool ? cudaMallocFromPoolAsync((void**)p, count * sizeof(T), pool, s)
                         : cudaMallocAsync((void**)p, count * sizeof(T), s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("device allocation of %zu bytes failed: %s", count * sizeof(T),
                  cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? HMG_ERR_NOMEM : HMG_ERR_CUDA;
    }
    return HMG_OK;
}

template <typename T>
void dfree(T*& p, cudaStream_t s)
{
    if (p) cudaFreeAsync((void*)p, s);
    p = nullptr;
}

// out[i] = sum_{k<i} in[k]; optionally *total_dev = sum of all (device pointer).
// T = int or long long.  in and out may alias.
template <typename T>
hmg_status scan_exclusive(const T* in, T* out, long long n, T* total_dev, cudaStream_t s);

// Stable LSD radix sort, 8-bit digits, in place (uses n-sized temporaries).
hmg_status radix_sort_pairs(uint64_t* keys, uint32_t* vals, int n, int key_bits,
                            cudaStream_t s);

}  // namespace hmg
