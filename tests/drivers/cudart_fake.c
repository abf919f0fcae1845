/* Fakes of the CUDA runtime's calls for tests of failing calls, preloaded into a
   child process: each passes on to the runtime, counts, and on request returns an
   error in the place of one call, which then does not happen (or, of free memory,
   another number). */
#include <cuda_runtime_api.h>
#include <dlfcn.h>

enum { INSTANTIATE, GRAPH_LAUNCH, COOPERATIVE, ALLOCATION, KINDS };
static long long calls[KINDS], failAt[KINDS];
static size_t failBytes;

/* The nth call of a kind from now on fails (0: none); of allocations, the nth of
   exactly `bytes` bytes.  Counts from zero again. */
void fake_arm(int kind, long long nth, size_t bytes)
{
    calls[kind] = 0;
    failAt[kind] = nth;
    if (kind == ALLOCATION) failBytes = bytes;
}
long long fake_count(int kind) { return calls[kind]; }

static size_t freeBytes;  /* what cudaMemGetInfo reports as free; 0: the truth */
void fake_free(size_t bytes) { freeBytes = bytes; }

static int fails(int kind) { return ++calls[kind] == failAt[kind]; }
static void* real(const char* name) { return dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name); }

cudaError_t cudaGraphInstantiate(cudaGraphExec_t* exec, cudaGraph_t graph, unsigned long long flags)
{
    if (fails(INSTANTIATE)) return cudaErrorMemoryAllocation;
    return ((cudaError_t(*)(cudaGraphExec_t*, cudaGraph_t, unsigned long long))real("cudaGraphInstantiate"))(exec, graph, flags);
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t exec, cudaStream_t s)
{
    if (fails(GRAPH_LAUNCH)) return cudaErrorMemoryAllocation;
    return ((cudaError_t(*)(cudaGraphExec_t, cudaStream_t))real("cudaGraphLaunch"))(exec, s);
}
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t s)
{
    if (bytes == failBytes && fails(ALLOCATION)) return cudaErrorMemoryAllocation;
    return ((cudaError_t(*)(void**, size_t, cudaStream_t))real("cudaMallocAsync"))(p, bytes, s);
}
cudaError_t cudaMemGetInfo(size_t* unused, size_t* total)
{
    const cudaError_t e = ((cudaError_t(*)(size_t*, size_t*))real("cudaMemGetInfo"))(unused, total);
    if (e == cudaSuccess && freeBytes) *unused = freeBytes;
    return e;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* kernel, void** args)
{
    for (unsigned k = 0; k < cfg->numAttrs; ++k)
        if (cfg->attrs[k].id == cudaLaunchAttributeCooperative && cfg->attrs[k].val.cooperative && fails(COOPERATIVE))
            return cudaErrorCooperativeLaunchTooLarge;
    return ((cudaError_t(*)(const cudaLaunchConfig_t*, const void*, void**))real("cudaLaunchKernelExC"))(cfg, kernel, args);
}
