// Host-side stand-ins for the CUDA runtime and for the parts of the library that
// pg_split_merge calls: linked with its object file alone, so no GPU is touched.
// Every call is appended to a log; call number `fail` returns an error.
#include <math.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

// device names in functions of the header that are not used here
static inline size_t __cvta_generic_to_shared(const void *) { return 0; }
static inline long long clock64() { return 0; }
static inline void atomicOr(uint32_t *, uint32_t) {}

#include "pg_internal.cuh"

namespace {
std::string g_log;
int g_calls, g_fail, g_queries;

cudaError_t call(const char *fmt, ...) {
    char line[128];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(line, sizeof line, fmt, ap);
    va_end(ap);
    const bool fails = g_calls++ == g_fail;
    g_log += std::string(line) + (fails ? " failed\n" : "\n");
    return fails ? cudaErrorUnknown : cudaSuccess;
}
long id(const void *p) { return (long)(uintptr_t)p; }
int launch_error;
}  // namespace

extern "C" {
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t s) {
    launch_error = call("launch %ld", id(s));
    return (cudaError_t)launch_error;
}
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, struct CUstream_st *s) {
    g_grid = g, g_block = b, g_smem = m, g_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *m, void *s) {
    *g = g_grid, *b = g_block, *m = g_smem, *(cudaStream_t *)s = g_stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaUnregisterFatBinary(void **) {}
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { *a = *b = 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return call("device sync"); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return call("record %ld %ld", id(e), id(s)); }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return call("attribute"); }
cudaError_t cudaGetLastError() { const int e = launch_error; launch_error = 0; return (cudaError_t)e; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) { return call("launch %ld", id(c->stream)); }
cudaError_t cudaMalloc(void **, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
    ++g_queries;
    *n = 4;
    return call("occupancy");
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *, unsigned, int) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return call("sync %ld", id(s)); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { return call("wait %ld %ld", id(s), id(e)); }
}

namespace pg {
int set_error(pg_ctx *, int status, const std::string &) { return status; }
int check_cuda(pg_ctx *, cudaError_t e, const char *) { return e == cudaSuccess ? PG_OK : PG_ERR_CUDA; }
void guide_mark_stale(pg_ctx *) {}
int order_regions(pg_ctx *, const uint32_t *, uint32_t, uint32_t, uint32_t *, uint32_t, uint32_t *, cudaStream_t s) {
    return call("launch %ld", id(s)) == cudaSuccess ? PG_OK : PG_ERR_CUDA;
}
}  // namespace pg

// `calls` split/merge passes of one context on stream 1 (side streams 10, 11; fork event
// 20, joins 30, 31), CUDA call `fail` of the last of them failing.  The last
// call's log; *queries: occupancy queries of all calls.
extern "C" int split_merge_calls(int calls, int fail, uint32_t cluster_size, uint32_t regions, char *log, int cap, int *queries) {
    alignas(16) static uint32_t words[64];
    pg_ctx ctx;
    ctx.sm_count = 152;
    ctx.max_regions = regions;
    ctx.d_counters = ctx.d_order = ctx.d_late = words;
    ctx.d_states = reinterpret_cast<pg_region_state *>(words);
    ctx.d_extras = reinterpret_cast<pg_region_extra *>(words);
    for (int i = 0; i < 2; ++i) {
        ctx.sm_aux[i] = (cudaStream_t)(uintptr_t)(10 + i);
        ctx.sm_join[i] = (cudaEvent_t)(uintptr_t)(30 + i);
    }
    ctx.sm_fork = (cudaEvent_t)(uintptr_t)20;
    pg_default_split_merge_config(&ctx.sm);
    ctx.sm.cluster_size = cluster_size;
    int st = PG_OK;
    g_queries = 0;
    for (int i = 0; i < calls; ++i) {
        g_log.clear();
        g_calls = 0;
        g_fail = i + 1 == calls ? fail : -1;
        st = pg_split_merge(&ctx, reinterpret_cast<float *>(words), reinterpret_cast<float *>(words), words, regions,
                            (void *)(uintptr_t)1);
    }
    snprintf(log, (size_t)cap, "%s", g_log.c_str());
    *queries = g_queries;
    return st;
}
