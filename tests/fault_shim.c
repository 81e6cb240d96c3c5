/* Fakes of the CUDA runtime's allocating and copying calls for tests/test_gpu_failures.py:
 * linked into a copy of the library with -Wl,--wrap=..., they answer with an error, without
 * calling CUDA, when the armed count runs out.  Everything fails on the host. */
#include <cuda_runtime_api.h>

enum { MALLOC, POOL, COPY, CALLS };
static int left[CALLS] = {-1, -1, -1};
static int seen[CALLS];

/* the call number `after` (0: the next) of kind `which` fails, once; < 0: none does */
void hmg_test_fail(int which, int after)
{
    left[which] = after;
    seen[which] = 0;
}

/* calls of the kind since it was armed */
int hmg_test_seen(int which) { return seen[which]; }

static int hit(int which)
{
    seen[which]++;
    return left[which] >= 0 && left[which]-- == 0;
}

cudaError_t __real_cudaMalloc(void** p, size_t n);
cudaError_t __wrap_cudaMalloc(void** p, size_t n)
{
    return hit(MALLOC) ? cudaErrorMemoryAllocation : __real_cudaMalloc(p, n);
}

cudaError_t __real_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s);
cudaError_t __wrap_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s)
{
    return hit(POOL) ? cudaErrorMemoryAllocation : __real_cudaMallocFromPoolAsync(p, n, pool, s);
}

cudaError_t __real_cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st);
cudaError_t __wrap_cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st)
{
    return hit(COPY) ? cudaErrorUnknown : __real_cudaMemcpyAsync(d, s, n, k, st);
}
