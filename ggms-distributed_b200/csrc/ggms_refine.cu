// ggms_refine.cu -- the refinement levels' launch, instantiated per value type.
#define GGMS_TU tu_refine
#include "ggms_refine.cuh"

namespace ggms {

template <typename T>
int launch_refine(Context* ctx, const RefineArgs<T>& a, cudaStream_t s) {
  static std::atomic<int> per_sm_of[MAX_DEVICES];  // per device: its attribute set, its resident CTAs per SM
  std::atomic<int>& per_sm = per_sm_of[ctx->device];
  if (!per_sm) {
    GGMS_CU(cudaFuncSetAttribute(refine_levels<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SMALL_SELECT_SMEM));
    int o = 0;
    GGMS_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, refine_levels<T>, RF_NT, SMALL_SELECT_SMEM));
    if (o < 1) return GGMS_E_CUDA;
    per_sm = std::min(o, 2);
  }
  ++ctx->launches;
  unsigned grid = (unsigned)(ctx->sms * per_sm);
  GGMS_CU(launch_coop(refine_levels<T>, grid, RF_NT, SMALL_SELECT_SMEM, s, a));
  return GGMS_OK;
}

template int launch_refine<float>(Context*, const RefineArgs<float>&, cudaStream_t);
template int launch_refine<double>(Context*, const RefineArgs<double>&, cudaStream_t);
template int launch_refine<uint32_t>(Context*, const RefineArgs<uint32_t>&, cudaStream_t);
template int launch_refine<int32_t>(Context*, const RefineArgs<int32_t>&, cudaStream_t);

}  // namespace ggms
