// fake_cuda.cpp — a CUDA runtime and the kernels' launchers for tests of the host code without a GPU: device
// memory is host memory, kernels do nothing, and what concerns the order of work is written to a log.  The
// n-th allocation or path-kernel launch from now on can be made to fail.
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "sr_bvh_build.h"
#include "sr_kernels.h"
#include "sr_wavefront.h"

static std::string g_log;
static size_t g_next = 1;
static int g_fail_malloc = 0, g_fail_launch = 0;

static void note(const char* format, ...) {
    char line[128];
    va_list a;
    va_start(a, format);
    vsnprintf(line, sizeof(line), format, a);
    va_end(a);
    g_log += line;
    g_log += '\n';
}

extern "C" {
const char* fake_log() { return g_log.c_str(); }
void fake_reset(int malloc_to_fail, int launch_to_fail) {
    g_log.clear();
    g_fail_malloc = malloc_to_fail, g_fail_launch = launch_to_fail;
}

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return note("sync device"), cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    note("malloc");
    if (g_fail_malloc && --g_fail_malloc == 0) return cudaErrorMemoryAllocation;
    return *p = calloc(1, n + 64), cudaSuccess;
}
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return memset(d, v, n), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)g_next++, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return note("sync %zu", (size_t)s), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    return note("wait %zu %zu", (size_t)s, (size_t)e), cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)g_next++, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)g_next++, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return note("record %zu %zu", (size_t)s, (size_t)e), cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { return note("launch %zu graph", (size_t)s), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}

namespace sr {

cudaError_t wave_paths(const WaveLaunch&, uint32_t, int sms, cudaStream_t st) {
    note("launch %zu paths %d", (size_t)st, sms);
    return g_fail_launch && --g_fail_launch == 0 ? cudaErrorLaunchFailure : cudaSuccess;
}
uint64_t wave_paths_pixels(bool, int sms) { return (uint64_t)sms * 2048; }
cudaError_t wave_init(const WaveLaunch&, cudaStream_t st, uint32_t) { return note("launch %zu init", (size_t)st), cudaSuccess; }
cudaError_t wave_bounce(const WaveLaunch&, int, cudaStream_t, const cudaStream_t*, const cudaEvent_t*) { return cudaSuccess; }
cudaError_t wave_tail(const WaveLaunch&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t wave_build_graph(const WaveLaunch&, cudaStream_t, const cudaStream_t*, const cudaEvent_t*, cudaGraphExec_t*) {
    return cudaSuccess;
}
cudaError_t wave_build_graph_batch(const WaveLaunch*, int, cudaStream_t, const cudaStream_t*, const cudaEvent_t*,
                                   cudaGraphExec_t*) {
    return cudaSuccess;
}
void wave_occupancy(bool, bool, int* a, int* b, int* c) { *a = *b = *c = 4; }
int wave_trace_occupancy(bool, bool, int) { return 4; }
void wave_grid_sizes(WaveLaunch&, int, const WaveTune*) {}
void wave_adj_grid_sizes(WaveLaunch&, int) {}
cudaError_t wave_adj_density(const AdjPass*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_adjoint_checkpoint(const WaveLaunch&, const float*, const uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_trace_persistent(const DevScene&, bool, const float*, uint32_t, Rec*, uint32_t*, int32_t*, int32_t*,
                                    float*, float*, uint32_t*, int, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_trace(const DevScene&, const float*, uint32_t, int32_t*, int32_t*, float*, float*, uint32_t*, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_render(const DevScene&, const DevView&, const DevParams&, const DevAovs&, unsigned long long*, uint32_t*,
                          cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_sky_table(const DevScene&, float4*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_adjoint(const DevScene&, const DevView&, const DevParams&, const DevAovs&, const float*, int, int, float*,
                           int, float*, float*, float*, uint32_t*, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_texels_from_rgb(const float*, float4*, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_compose(const DevAovs&, uint32_t, uint32_t, const ComposeConsts&, const float2*, const float*,
                           const float*, bool, uint8_t*, float4*, cudaStream_t, float*) {
    return cudaSuccess;
}
cudaError_t launch_compose_static(int, const DevAovs&, uint32_t, uint32_t, const ComposeConsts&, float, float, float,
                                  uint8_t*, cudaStream_t, size_t*, bool*) {
    return cudaSuccess;
}
size_t compose_static_capacity() { return 0; }
cudaError_t launch_aov_image(const DevAovs&, uint32_t, int32_t, float, const uint8_t*, uint32_t, float, float, uint8_t*,
                             cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_overlay(const OverlayLineOp*, uint32_t, const OverlayGlyphOp*, uint32_t, const uint8_t*, const uint32_t*,
                           const float*, uint32_t, uint32_t, int32_t*, uint8_t*, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t build_bvh_device(const std::vector<host::Box>&, float, float, int, cudaStream_t, host::BvhHost&) {
    return cudaErrorNotSupported;
}
cudaError_t build_bvh_device_arrays(const float*, int, float, float, int, cudaStream_t, float*, int32_t*, int32_t*, uint32_t*,
                                    bool*) {
    return cudaErrorNotSupported;
}

}  // namespace sr
