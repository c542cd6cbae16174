// ggms_direct.cu -- the one-launch path's launch, instantiated per value type.
#define GGMS_TU tu_direct
#include "ggms_direct.cuh"

namespace ggms {

template <typename T>
int launch_direct(Context* ctx, const DirectArgs<T>& a, unsigned ctas, cudaStream_t s) {
  using K = typename KeyOf<T>::K;
  static std::atomic<int> ready[MAX_DEVICES];  // per device: the kernels' attributes are set
  constexpr size_t sort_smem = sizeof(SortSmem<K>) + direct_cap<K>() * sizeof(K);
  if (!ready[ctx->device]) {
    GGMS_CU(cudaFuncSetAttribute(direct_select<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)direct_smem<K>()));
    GGMS_CU(cudaFuncSetAttribute(direct_sort<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_smem));
    ready[ctx->device] = 1;
  }
  ++ctx->launches;
  if (a.n <= direct_cap<K>()) {
    direct_sort<T><<<1, DR_NT, sort_smem, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? GGMS_OK : GGMS_E_CUDA;
  }
  unsigned grid = std::min<unsigned>(ctas, (unsigned)ctx->sms);
  GGMS_CU(launch_coop(direct_select<T>, grid, DR_NT, direct_smem<K>(), s, a));
  return GGMS_OK;
}

template int launch_direct<float>(Context*, const DirectArgs<float>&, unsigned, cudaStream_t);
template int launch_direct<double>(Context*, const DirectArgs<double>&, unsigned, cudaStream_t);
template int launch_direct<uint32_t>(Context*, const DirectArgs<uint32_t>&, unsigned, cudaStream_t);
template int launch_direct<int32_t>(Context*, const DirectArgs<int32_t>&, unsigned, cudaStream_t);

}  // namespace ggms

#ifdef GGMS_SETUP_TRACE
extern "C" GGMS_API int ggms_trace_read_direct(unsigned long long* out) {
  return cudaMemcpyFromSymbol(out, ggms_trace_buf, sizeof(ggms_trace_buf)) == cudaSuccess ? 0 : 4;
}
extern "C" GGMS_API int ggms_trace_read_cta_direct(unsigned long long* out) {
  return cudaMemcpyFromSymbol(out, ggms_trace_cta, sizeof(ggms_trace_cta)) == cudaSuccess ? 0 : 4;
}
#endif
