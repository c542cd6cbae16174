// ggms_batch.cu -- the batched path's launches, instantiated per value type.
#define GGMS_TU tu_batch
#include "ggms_batch.cuh"

namespace ggms {

namespace {

template <typename T, uint32_t ROW>
int launch_rows(Context* ctx, const BatchArgs<T>& a, cudaStream_t s) {
  static std::atomic<int> resident[MAX_DEVICES];  // per device: attribute set, resident CTAs per SM
  std::atomic<int>& per_sm = resident[ctx->device];
  constexpr size_t smem = RW_NT / 32 * sizeof(RowSmem<typename KeyOf<T>::K, ROW>);
  if (!per_sm) {
    GGMS_CU(cudaFuncSetAttribute(rows_select<T, ROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int o = 0;
    GGMS_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, rows_select<T, ROW>, RW_NT, smem));
    if (o < 1) return GGMS_E_CUDA;
    per_sm = o;
  }
  ++ctx->launches;
  GGMS_CU(launch_pdl(rows_select<T, ROW>, (unsigned)(ctx->sms * per_sm), RW_NT, smem, s, a));
  return GGMS_OK;
}

}  // namespace

template <typename T>
int launch_batch(Context* ctx, const BatchArgs<T>& a, cudaStream_t s) {
  static std::atomic<int> ready[MAX_DEVICES];  // per device: the attribute is set
  using K = typename KeyOf<T>::K;
  constexpr size_t smem = sizeof(DirectSmem<K>), sort_smem = sizeof(SortSmem<K>) + direct_cap<K>() * sizeof(K);
  if (!ready[ctx->device]) {
    GGMS_CU(cudaFuncSetAttribute(batch_teams<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    GGMS_CU(cudaFuncSetAttribute(batch_singles<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    GGMS_CU(cudaFuncSetAttribute(batch_sorts<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_smem));
    ready[ctx->device] = 1;
  }
  ctx->launches += 4;
  batch_init<T><<<std::min<unsigned>(cdiv(std::max(a.nseg, a.r.nk), 256), (unsigned)ctx->sms * 8), 256, 0, s>>>(
      a, (uint32_t)ctx->sms);
  GGMS_CU(cudaGetLastError());
  if (const int r = launch_rows<T, BT_ROW0>(ctx, a, s)) return r;
  if (const int r = launch_rows<T, BT_ROW0 * 2>(ctx, a, s)) return r;
  batch_sorts<T><<<(unsigned)ctx->sms, DR_NT, sort_smem, s>>>(a);
  GGMS_CU(cudaGetLastError());
  // fewer than ctx->sms segments are longer than a share: one round with that many CTAs
  unsigned grid = std::min<unsigned>((unsigned)ctx->sms, TEAM_MAX_CTAS);
  for (uint32_t round = 0; round * grid < (uint32_t)ctx->sms; ++round) {
    if (round) ++ctx->launches;
    GGMS_CU(launch_coop(batch_teams<T>, grid, DR_NT, smem, s, a, round));
  }
  // a single's segment has more than direct_cap keys
  const unsigned most = (unsigned)std::min<uint64_t>(a.nseg, a.n / direct_cap<K>());
  if (most) batch_singles<T><<<most, DR_NT, smem, s>>>(a);
  GGMS_CU(cudaGetLastError());
  return GGMS_OK;
}

template int launch_batch<float>(Context*, const BatchArgs<float>&, cudaStream_t);
template int launch_batch<uint32_t>(Context*, const BatchArgs<uint32_t>&, cudaStream_t);

}  // namespace ggms
