// Around the runtime's launch calls (ld --wrap): one launch can be dropped, as
// a mistake in the host code might, and the call goes on without it.
#include <cuda_runtime_api.h>

static int g_launches = 0, g_drop = -1;

extern "C" {
cudaError_t __real_cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t);
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**);

__attribute__((visibility("default"))) void shim_drop(int launch) {  // launch number from now on; -1: none
  g_launches = 0;
  g_drop = launch;
}
cudaError_t __wrap_cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t m, cudaStream_t s) {
  return g_launches++ == g_drop ? cudaSuccess : __real_cudaLaunchKernel(f, g, b, a, m, s);
}
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  return g_launches++ == g_drop ? cudaSuccess : __real_cudaLaunchKernelExC(c, f, a);
}
}
