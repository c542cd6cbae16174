// A CUDA runtime without a GPU, for tests of the host code: memory is host
// memory, copies and memsets run at once, kernels are only counted.  One launch
// can be made to fail, and cooperative launches of more than a given number of
// CTAs are refused, as they are where fewer SMs are free to the caller.
#include <cstdlib>
#include <cstring>
#include <cuda_runtime_api.h>

static int g_launches = 0, g_fail_at = -1;
static unsigned g_coop_max = 0, g_coop_grid = 0;
static cudaError_t g_last = cudaSuccess;

static cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) g_last = e;
  return e;
}
static cudaError_t launch() { return set(g_launches++ == g_fail_at ? cudaErrorInvalidConfiguration : cudaSuccess); }

extern "C" {
#define API __attribute__((visibility("default")))

// launches from now on; launch number fail_at fails (-1: none); cooperative
// launches of more than coop_max CTAs are refused (0: none)
API void fake_reset(int fail_at, unsigned coop_max) {
  g_launches = 0;
  g_fail_at = fail_at;
  g_coop_max = coop_max;
  g_coop_grid = 0;
  g_last = cudaSuccess;
}
API int fake_launches() { return g_launches; }
API unsigned fake_coop_grid() { return g_coop_grid; }  // CTAs of the largest cooperative launch that was taken

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) {
  for (unsigned i = 0; i < c->numAttrs; ++i)
    if (c->attrs[i].id == cudaLaunchAttributeCooperative && c->attrs[i].val.cooperative) {
      if (g_coop_max && c->gridDim.x > g_coop_max) return set(cudaErrorCooperativeLaunchTooLarge);
      if (c->gridDim.x > g_coop_grid) g_coop_grid = c->gridDim.x;
    }
  return launch();
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

cudaError_t cudaMalloc(void** p, size_t n) { return (*p = calloc(1, n)) ? cudaSuccess : set(cudaErrorMemoryAllocation); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 1; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 1; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

// no graphs: a call that repeats runs directly
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorStreamCaptureUnsupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
