// ggms_engine.cuh -- host orchestration of one call: the single-vector path
// (run_single), the batched segmented path (run_segmented), the autotuner and
// the entry-point bodies.
//
// One call = one stream-ordered sequence of kernels over a cached workspace:
// no host round trip between the passes, no allocation on the steady path,
// one H2D of the ks and one D2H of the answers when those live in host memory.
// (The reference does ~12 cudaMalloc/cudaFree and ~10 blocking copies per
// call: DistributedSMOS/bucketMultiselect.cu:583-606, 625-638, 805-845.)
//
// Each translation unit that includes this header defines GGMS_TU first and
// instantiates the templates for its own value types: the kernels (and the
// once-per-kernel attribute flags next to their launches) then belong to that
// unit alone, and the units compile in parallel.
#pragma once
#include "ggms_host.cuh"
#include "ggms_kernels.cuh"
#include "ggms_refine.cuh"
#include "ggms_direct.cuh"
#include "ggms_batch.cuh"
#include "ggms_learned.cuh"
#include "ggms_window.cuh"

GGMS_BEGIN

template <typename K>
struct Workspace {
  Counters* C;
  uint32_t* krank;
  uint32_t* kseg;
  uint32_t* kbin;
  K* kkey;
  K* samp_raw;
  K* samp_sorted;
  Assigner<K>* asg;       // [0] sampled, [1] learned (the PL models)
  Grid<K>* grid;          // [0] sampled, [1] learned (what the passes evaluate)
  LearnState* learn;
  Windows<K>* win;        // PASS 1 windows
  uint32_t* hist0;
  uint32_t* aflag0;
  uint32_t* kcnt0;        // per level-0 bucket: ks it holds (right after aflag0: one memset clears both)
  uint32_t* cmap0;
  uint32_t* crow;         // per-CTA bucket counts of PASS 1 -> per-CTA cursors of PASS 2
  uint32_t* ic;           // coarse mode: inclusive counts of the NGRP groups
  uint32_t* aflagc;       // coarse mode: groups holding a k
  Seg<K>* segs[2];
  uint32_t* cursor[2];
  TileRef* tiles[2];
  uint32_t* rows[2];
  uint32_t* aflag[2];
  uint32_t* khead[2];     // per segment: head of its k list (small segments)
  uint32_t* knext;        // per k: next k in its segment's list
  uint32_t* smalls;       // ids of the small segments the current level created
  uint32_t* tinies;       // ids of the tiny segments the current level created
  uint32_t* bigs[2];      // per pool: the segments a level refines, by row
  uint32_t* lists;        // batched path: segments by class [BT_CLASSES][nlist]
  uint32_t* scratch;      // ... per CTA: a team's global histogram and cursors
  K* points;
  K* cand[2];
  size_t bytes;
};


template <typename K>
static Workspace<K> layout(const Plan& p, uint8_t* base) {
  Bump b;
  Workspace<K> w;
  static_assert(sizeof(Counters) <= ARENA_BAR, "the barrier word follows the counters");
  size_t o_C = b.take(sizeof(Counters));
  b.take(ARENA_BAR_BYTES);
  size_t o_krank = b.take(4ull * p.nk);
  size_t o_kseg = b.take(4ull * p.nk);
  size_t o_kbin = b.take(4ull * p.nk);
  size_t o_kkey = b.take(sizeof(K) * p.nk);
  size_t o_sr = b.take(sizeof(K) * p.S);
  size_t o_ss = b.take(sizeof(K) * p.S);
  size_t o_asg = b.take(sizeof(Assigner<K>) * 2);
  size_t o_grid = b.take(sizeof(Grid<K>) * 2);
  size_t o_learn = b.take(sizeof(LearnState));
  size_t o_win = b.take(sizeof(Windows<K>));
  size_t o_h0 = b.take(4ull * p.B);
  size_t o_a0 = b.take(4ull * (p.B / 32) + 4ull * p.B);
  size_t o_c0 = b.take(4ull * p.B);
  size_t o_crow = b.take(4ull * p.B * (p.ncta ? p.ncta : 2));  // (0: the other paths' buckets of one key)
  size_t o_ic = b.take(4ull * NGRP);
  size_t o_afc = b.take(4ull * (NGRP / 32));
  size_t o_segs[2], o_cur[2], o_tiles[2], o_rows[2], o_af[2], o_cand[2], o_kh[2];
  size_t o_knext = b.take(4ull * p.nk);
  size_t o_smalls = b.take(4ull * p.cap_seg);
  size_t o_tinies = b.take(4ull * p.cap_seg);
  size_t o_bigs[2];
  for (int i = 0; i < 2; ++i) o_bigs[i] = b.take(4ull * p.cap_rows);
  size_t o_lists = b.take(4ull * BT_CLASSES * p.nlist);
  size_t o_scratch = b.take(p.nlist ? 4ull * BT_SCRATCH * p.sms : 0);
  for (int i = 0; i < 2; ++i) {
    o_kh[i] = b.take(4ull * p.cap_seg);
    o_segs[i] = b.take(sizeof(Seg<K>) * p.cap_seg);
    o_cur[i] = b.take(4ull * p.cap_seg);
    o_tiles[i] = b.take(sizeof(TileRef) * p.cap_tiles);
    o_rows[i] = b.take(4ull * NBIN * p.cap_rows);
    o_af[i] = b.take(4ull * NBIN_WORDS * p.cap_rows);
  }
  size_t o_pts = b.take(sizeof(K) * p.nk);
  for (int i = 0; i < 2; ++i) o_cand[i] = b.take(sizeof(K) * p.n);
  w.bytes = b.take(0) + 256;
  if (!base) return w;
  w.C = (Counters*)(base + o_C);
  w.krank = (uint32_t*)(base + o_krank);
  w.kseg = (uint32_t*)(base + o_kseg);
  w.kbin = (uint32_t*)(base + o_kbin);
  w.kkey = (K*)(base + o_kkey);
  w.samp_raw = (K*)(base + o_sr);
  w.samp_sorted = (K*)(base + o_ss);
  w.asg = (Assigner<K>*)(base + o_asg);
  w.grid = (Grid<K>*)(base + o_grid);
  w.learn = (LearnState*)(base + o_learn);
  w.win = (Windows<K>*)(base + o_win);
  w.hist0 = (uint32_t*)(base + o_h0);
  w.aflag0 = (uint32_t*)(base + o_a0);
  w.kcnt0 = w.aflag0 + p.B / 32;
  w.cmap0 = (uint32_t*)(base + o_c0);
  w.crow = (uint32_t*)(base + o_crow);
  w.ic = (uint32_t*)(base + o_ic);
  w.aflagc = (uint32_t*)(base + o_afc);
  for (int i = 0; i < 2; ++i) {
    w.segs[i] = (Seg<K>*)(base + o_segs[i]);
    w.cursor[i] = (uint32_t*)(base + o_cur[i]);
    w.tiles[i] = (TileRef*)(base + o_tiles[i]);
    w.rows[i] = (uint32_t*)(base + o_rows[i]);
    w.aflag[i] = (uint32_t*)(base + o_af[i]);
    w.cand[i] = (K*)(base + o_cand[i]);
    w.khead[i] = (uint32_t*)(base + o_kh[i]);
  }
  w.knext = (uint32_t*)(base + o_knext);
  w.smalls = (uint32_t*)(base + o_smalls);
  w.tinies = (uint32_t*)(base + o_tinies);
  for (int i = 0; i < 2; ++i) w.bigs[i] = (uint32_t*)(base + o_bigs[i]);
  w.lists = (uint32_t*)(base + o_lists);
  w.scratch = (uint32_t*)(base + o_scratch);
  w.points = (K*)(base + o_pts);
  return w;
}


// The arguments of refine_levels over a workspace: the levels from 1 on, then
// the answers to `out` (device or pinned memory).
template <typename T>
static RefineArgs<T> refine_args(const Workspace<typename KeyOf<T>::K>& w, const Context* c, uint64_t n, uint32_t nk, Caps caps,
                                 T* out, Counters* report) {
  RefineArgs<T> a;
  a.C = w.C;
  a.bar = (uint32_t*)(c->arena + ARENA_BAR);
  a.left = a.bar + ARENA_BAR_BYTES / 4 - 1;
  a.limit = barrier_limit(c, n, nk);
  for (int i = 0; i < 2; ++i) {
    a.cand[i] = w.cand[i];
    a.segs[i] = w.segs[i];
    a.tiles[i] = w.tiles[i];
    a.rows[i] = w.rows[i];
    a.aflag[i] = w.aflag[i];
    a.bigs[i] = w.bigs[i];
    a.cursor[i] = w.cursor[i];
    a.khead[i] = w.khead[i];
  }
  a.knext = w.knext;
  a.smalls = w.smalls;
  a.tinies = w.tinies;
  a.krank = w.krank;
  a.kseg = w.kseg;
  a.kbin = w.kbin;
  a.points = w.points;
  a.kkey = w.kkey;
  a.nk = nk;
  a.caps = caps;
  a.caps.tiny_keys = RF_TINY / sizeof(typename KeyOf<T>::K);  // of the levels' children
  a.out = out;
  a.report = report;
  return a;
}

// ------------------------------------------------------------------ kernel configs

template <typename T>
static size_t l0_count_smem(uint32_t B, int nt, int unroll, uint32_t nst) {
  const size_t base = GRID_SMEM + (size_t)B * 4u + wq_bytes((uint32_t)nt, sizeof(typename KeyOf<T>::K));
  return unroll < 0 ? ((base + 127) & ~(size_t)127) + ring_bytes(unroll, nst) : base;
}
template <typename T>
static size_t l0_coarse_smem(int nt, int unroll, uint32_t nst) {
  const size_t ch = (size_t)nt * coarse_du(unroll < 0 ? 0 : unroll) * (16 / sizeof(T));
  const size_t base = GRID_SMEM + ch * (sizeof(typename KeyOf<T>::K) + 1);
  return unroll < 0 ? ((base + 127) & ~(size_t)127) + ring_bytes(unroll, nst) : base;
}
template <typename T>
static size_t l0_compact_smem(uint32_t B, int nt, int unroll, uint32_t nst) {
  const size_t base = GRID_SMEM +
                      (MAX_B0 / 32 + l0_compact_qwords((uint32_t)nt, sizeof(typename KeyOf<T>::K)) + HOT_WORDS) * 4u +
                      (size_t)B * 4u;
  return unroll < 0 ? ((base + 127) & ~(size_t)127) + ring_bytes(unroll, nst) : base;
}

// Launch shapes of the two passes: CTA size x 16-byte loads in flight per
// thread (unroll 2, 4 or 8, register streams), unroll -1: the TMA ring (bulk
// copies into shared-memory stages), unroll -2: per-thread async copies into
// shared memory; the default and the autotuner pick among these instantiations.
template <typename T>
struct PassVariant {
  using K = typename KeyOf<T>::K;
  int nt, unroll;
  void (*count)(const T*, uint64_t, const Grid<K>*, Counters*, const Windows<K>*, uint32_t*, uint32_t*, uint32_t);
  void (*compact)(const T*, uint64_t, const Grid<K>*, Counters*, const Windows<K>*, const uint32_t*,
                  const uint32_t*, K*, uint64_t, uint32_t, const uint32_t*);
  void (*coarse)(const T*, uint64_t, const Grid<K>*, Counters*, const uint32_t*, const uint32_t*, K*, uint64_t,
                 uint32_t);
};

template <typename T>
static const PassVariant<T>* pass_variant(int nt, int unroll) {
  static const PassVariant<T> v[] = {
      {256, 4, l0_count<T, 256, 4>, l0_compact<T, 256, 4>, l0_compact_coarse<T, 256, 4>},
      {256, 8, l0_count<T, 256, 8>, l0_compact<T, 256, 8>, l0_compact_coarse<T, 256, 8>},
      {512, 2, l0_count<T, 512, 2>, l0_compact<T, 512, 2>, l0_compact_coarse<T, 512, 2>},
      {512, 4, l0_count<T, 512, 4>, l0_compact<T, 512, 4>, l0_compact_coarse<T, 512, 4>},
      {512, 8, l0_count<T, 512, 8>, l0_compact<T, 512, 8>, l0_compact_coarse<T, 512, 8>},
      {1024, 2, l0_count<T, 1024, 2>, l0_compact<T, 1024, 2>, l0_compact_coarse<T, 1024, 2>},
      {1024, 4, l0_count<T, 1024, 4>, l0_compact<T, 1024, 4>, l0_compact_coarse<T, 1024, 4>},
      {1024, -1, l0_count<T, 1024, -1>, l0_compact<T, 1024, -1>, l0_compact_coarse<T, 1024, -1>},
      {1024, -2, l0_count<T, 1024, -2>, l0_compact<T, 1024, -2>, l0_compact_coarse<T, 1024, -2>},
  };
  for (const auto& x : v)
    if (x.nt == nt && x.unroll == unroll) return &x;
  return nullptr;
}

constexpr int DEFAULT_PASS_NT = 1024;
constexpr int DEFAULT_PASS_UNROLL = 4;  // register streams (the staged ones measure no faster here)

// Stages of the TMA ring of one pass kernel whose other shared memory is
// `base` bytes: as many 32 KB stages (2..4) as fit next to it in what a CTA
// may use (its static shared memory included, with margin).
static uint32_t ring_stages(Context* c, size_t base) {
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device) != cudaSuccess)
    optin = 227 * 1024;
  const size_t margin = 8192 + 128;  // static shared memory of the pass kernels, alignment
  const size_t room = (size_t)optin > base + margin ? (size_t)optin - base - margin : 0;
  return (uint32_t)std::min<size_t>(4, std::max<size_t>(2, room / RING_BYTES));
}

// Stages of the three pass kernels' rings: [0] count, [1] compact, [2] coarse
// (0 for the other streams).
template <typename T>
static void pass_stages(Context* c, const PassVariant<T>* pv, uint32_t B, uint32_t* st) {
  for (int i = 0; i < 3; ++i) st[i] = 0u;
  if (pv->unroll != -1) return;
  st[0] = ring_stages(c, l0_count_smem<T>(B, pv->nt, -1, 0));
  st[1] = ring_stages(c, l0_compact_smem<T>(B, pv->nt, -1, 0));
  st[2] = ring_stages(c, l0_coarse_smem<T>(pv->nt, -1, 0));
}

// The two passes must split the input among CTAs identically (PASS 2 writes
// into per-CTA ranges sized by PASS 1), so both get the same grid: as many
// CTAs as fit on every SM at once for the larger of the two.
template <typename T>
static int l0_ncta(Context* c, const PassVariant<T>* pv, uint32_t B, const uint32_t* nst, uint32_t* ncta) {
  const size_t s1 = l0_count_smem<T>(B, pv->nt, pv->unroll, nst[0]);
  const size_t s2 = l0_compact_smem<T>(B, pv->nt, pv->unroll, nst[1]);
  const size_t s3 = l0_coarse_smem<T>(pv->nt, pv->unroll, nst[2]);
  GGMS_CU(cudaFuncSetAttribute((const void*)pv->count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1));
  GGMS_CU(cudaFuncSetAttribute((const void*)pv->compact, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2));
  GGMS_CU(cudaFuncSetAttribute((const void*)pv->coarse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3));
  int o1 = 0, o2 = 0, o3 = 0;
  GGMS_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o1, (const void*)pv->count, pv->nt, s1));
  GGMS_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o2, (const void*)pv->compact, pv->nt, s2));
  GGMS_CU(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o3, (const void*)pv->coarse, pv->nt, s3));
  *ncta = (uint32_t)(std::max(1, std::min(std::min(o1, o2), o3)) * c->sms);
  return GGMS_OK;
}

// Up to this many ks, the steps between the passes run in one CTA (l0_between).
constexpr uint32_t L0_FUSED_MAX_KS = 65536;

template <typename K>
static int setup_attrs() {
  static bool done = false;
  if (done) return GGMS_OK;
  GGMS_CU(cudaFuncSetAttribute(l0_between<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)l0_between_smem(MAX_B0)));
  GGMS_CU(cudaFuncSetAttribute(l0_scan<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(4u * MAX_B0)));
  GGMS_CU(cudaFuncSetAttribute(setup_sampled<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(SetupSmem<K>)));
  GGMS_CU(cudaFuncSetAttribute(l0_window<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)l0_window_smem<K>(MAX_B0)));
  done = true;
  return GGMS_OK;
}

constexpr int SS_NT = 512;

template <typename InT, typename K = typename KeyOf<InT>::K>
static int launch_small_select(Context* ctx, const InT* src, const Seg<K>* segs_q, const uint32_t* khead_q,
                               const Workspace<K>& w, const Caps& caps, cudaStream_t st) {
  static bool attr = false;
  const size_t sm = SMALL_SELECT_SMEM;
  if (!attr) {
    GGMS_CU(cudaFuncSetAttribute(small_select<InT, SS_NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sm));
    attr = true;
  }
  ++ctx->launches;
  GGMS_CU(launch_pdl(small_select<InT, SS_NT>, ctx->sms * 2, SS_NT, sm, st, src, segs_q, w.smalls, w.C, khead_q,
                     w.knext, w.krank, w.kseg, w.kkey, caps.small_keys, caps));
  // the warp finisher (its own list of segments) runs beside the CTA finisher:
  // it does not wait for it before its work (tiny_select)
  if (caps.tiny_keys) {
    ++ctx->launches;
    GGMS_CU(launch_pdl(tiny_select<InT, TS_NT>, ctx->sms * 8, TS_NT, 0, st, src, segs_q, w.tinies, w.C, khead_q,
                       w.knext, w.krank, w.kseg, w.kkey, caps));
  }
  return GGMS_OK;
}

// Profiling slot of the current call (or null when profiling is off).

// ------------------------------------------------------------------ the single-vector path

// The sample sort's cluster: attributes set once per key type; 16 CTAs when the
// sample has at least one key per thread of 16 CTAs and the device can place a
// 16-CTA cluster of this kernel, else 8; 0: too small for a cluster (S < 8192);
// -1: the attributes could not be set.
template <typename K, int CTAS>
static cudaError_t launch_sort_cluster(cudaStream_t s, const K* drawn, uint32_t S, K* sorted) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CTAS);
  cfg.blockDim = dim3(CS_NT);
  cfg.dynamicSmemBytes = sizeof(ClusterSortSmem<K, CTAS>);
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CTAS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, asg_sort_cluster<K, CTAS>, drawn, S, sorted);
}

template <typename K>
static int sort_cluster_ctas(uint32_t S) {
  static int have16 = -1;  // -1: not probed yet
  if (have16 < 0) {
    have16 = 0;
    if (cudaFuncSetAttribute(asg_sort_cluster<K, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(ClusterSortSmem<K, 8>)) != cudaSuccess ||
        cudaFuncSetAttribute(asg_sort_cluster<K, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(ClusterSortSmem<K, 16>)) != cudaSuccess)
      return -1;
    if (cudaFuncSetAttribute(asg_sort_cluster<K, 16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
        cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(16);
      cfg.blockDim = dim3(CS_NT);
      cfg.dynamicSmemBytes = sizeof(ClusterSortSmem<K, 16>);
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 16;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nclusters = 0;
      if (cudaOccupancyMaxActiveClusters(&nclusters, asg_sort_cluster<K, 16>, &cfg) == cudaSuccess &&
          nclusters >= 1)
        have16 = 1;
    }
    cudaGetLastError();  // a refused probe leaves no error behind
  }
  if (S >= cs_min_s(16) && have16) return 16;
  return S >= cs_min_s(8) ? 8 : 0;
}

// The one-launch path (ggms_direct.cuh) takes calls that leave everything to
// the library: AUTO with no tuning field set, no statistics and no profiling
// (those describe the two-pass pipeline).  The lines below, and where they lie
// (us per call, one launch / pipeline, B200, device ks and answers):
//   bytes: the second read comes from L2 (126 MB) up to 2^24 fp32: 80 / 189
//     for 5 random ks, 86 / 165 for 1000 in the top 1 %.  At 128 MB fp32 it is
//     138 / 241 for 8 random ks, at 160 MB 164 / 265, at 280 MB 331 / 360, and
//     242 / 233 for 300 in the top 1 %.
//   keys: what the buckets of the ks hold is copied and sorted whole, and
//     16384 buckets over more keys hold more each, where the pipeline has a
//     bucket per k or more.  The mixture of eight narrow modes is the worst:
//     300 ks 343 / 349 at 40 M keys; 1000 ks 262 / 287 at 16 M, 334 / 312 at
//     24 M; 4000 ks 261 / 389 at 8 M, 378 / 457 at 16 M fp32 but 733 / 651
//     fp64.  Top-k, one cluster of ks, has no such limit: 146 / 224 for 2^13
//     of 2^25.
//   ks: every k costs each CTA a search up to DIRECT_SLICE_KS; beyond, each CTA
//     searches its own (one more barrier): 2^14 ks took 50 us of searching
//     without it, 10 with it.  DIRECT_MAX_KS is the largest count measured.
//   buckets: one per 8 keys keeps the children of a short vector short (2^16
//     fp32, 1000 ks: 38 us, 45 with one per 32); 16384 instead of 8192 halve
//     the copied keys of a long one (2^24, 1000 ks) and cost a short one 2 us.
//   focus (most buckets to clustered ks): costs 3 us of the map, saves 25 of
//     the copy and sort at 2^22 and 100 at 2^24 with 1000 ks in the top 1 %.
constexpr uint64_t DIRECT_MAX_BYTES = 160ull << 20;
constexpr uint64_t DIRECT_SOME_KS = 512, DIRECT_MANY_KS = 2048;  // more than so many ks: up to ..
constexpr uint64_t DIRECT_SOME_N = 20u << 20, DIRECT_MANY_N = 12u << 20;  // .. so many keys
constexpr uint32_t DIRECT_MAX_KS = 65536;
constexpr uint64_t DIRECT_CTA_KEYS = 1024;    // keys that repay another CTA
constexpr uint64_t DIRECT_BUCKET_KEYS = 8;
constexpr uint64_t DIRECT_WIDE_N = 1u << 23;  // vectors that get all DIRECT_MAX_B buckets
constexpr uint64_t DIRECT_FOCUS_N = 1u << 18;
constexpr uint32_t DIRECT_FOCUS_KS = 16;
constexpr uint32_t DIRECT_SLICE_KS = 2048;

static bool direct_ok(const Context* ctx, const ggms_opts& o, uint64_t n, uint64_t nk, size_t elem, bool topk) {
  const uint64_t max_n = nk > DIRECT_MANY_KS ? DIRECT_MANY_N : nk > DIRECT_SOME_KS ? DIRECT_SOME_N : ~0ull;
  return n * elem <= DIRECT_MAX_BYTES && (topk || n <= max_n) && nk <= DIRECT_MAX_KS && !ctx->profile && !o.stats && !o.autotune &&
         o.assigner == GGMS_ASSIGNER_AUTO && !o.num_buckets && !o.sample_size && o.train_steps <= 0 &&
         !o.pass_threads && !o.pass_unroll && o.window_z == 0.0f && !o.pl_knots;
}

template <typename T>
static int run_direct(Context* ctx, const T* d_in, uint64_t n, const uint32_t* ks, uint32_t nk, T* out,
                      const ggms_opts& o, cudaStream_t st, bool topk) {
  using K = typename KeyOf<T>::K;
  ggms_opts od = o;
  od.num_buckets = (int32_t)std::min<uint64_t>(n < DIRECT_WIDE_N ? DIRECT_MAX_B / 2 : DIRECT_MAX_B,
                                                  std::max<uint64_t>(1024, pow2_floor(n / DIRECT_BUCKET_KEYS)));
  od.sample_size = 1024;  // this path's sample stays in shared memory
  Plan p;
  int rc = make_plan(&p, n, nk, od);
  if (rc) return rc;
  GGMS_CU(cudaSetDevice(ctx->device));
  rc = ensure_arena(ctx, layout<K>(p, nullptr).bytes);
  if (rc) return rc;
  const Workspace<K> w = layout<K>(p, ctx->arena);
  const bool host_k = !o.ks_on_device && !topk, host_out = !o.out_on_device;
  const PinLayout pl = pin_layout(nk, sizeof(T), host_k, host_out);
  rc = ensure_pinned(ctx, pl.bytes);
  if (rc) return rc;
  Counters* pin_C = (Counters*)ctx->pinned;
  uint8_t* pin_k = ctx->pinned + pl.ks;
  T* pin_out = (T*)(ctx->pinned + pl.out);
  if (host_k) {
    if (ctx->pin_busy) GGMS_CU(cudaEventSynchronize(ctx->pin_busy));
    memcpy(pin_k, ks, 4ull * nk);
  }
  const Caps caps{p.cap_seg, p.cap_tiles, p.nk, (uint32_t)(SMALL_SMEM / sizeof(K)), 0u, p.cap_rows};
  const unsigned ctas = (unsigned)std::min<uint64_t>((n + DIRECT_CTA_KEYS - 1) / DIRECT_CTA_KEYS, 1u << 16);
  auto enqueue = [&](cudaStream_t s) -> int {
    DirectArgs<T> a;
    a.in = d_in;
    a.n = n;
    a.ks = topk ? nullptr : (host_k ? (const uint32_t*)pin_k : ks);
    a.seed = p.seed;
    a.B = p.B;
    a.slices = nk > DIRECT_SLICE_KS ? 1u : 0u;
    a.focus = n >= DIRECT_FOCUS_N && nk >= DIRECT_FOCUS_KS && !a.slices ? 1u : 0u;
    a.gact = w.aflag0;
    a.ghist = w.hist0;
    a.gcur = w.cmap0;
    a.gpt = w.crow;
    a.r = refine_args<T>(w, ctx, n, nk, caps, host_out ? pin_out : out, host_out ? pin_C : nullptr);
    return launch_direct<T>(ctx, a, ctas, s);
  };
  const uint64_t key[] = {0xD17ull + sizeof(T) + (topk ? 256u : 0u) + (std::is_signed<T>::value ? 16u : 0u) +
                              (std::is_floating_point<T>::value ? 32u : 0u),
                          (uint64_t)(uintptr_t)d_in, n, host_k ? 1ull : (uint64_t)(uintptr_t)ks, nk,
                          host_out ? 1ull : (uint64_t)(uintptr_t)out, p.seed, (uint64_t)(uintptr_t)ctx->arena,
                          (uint64_t)(uintptr_t)ctx->pinned, (uint64_t)ctx->barrier_limit};
  if (host_out) pin_C->status = GGMS_E_INTERNAL;  // until the launch reports
  rc = run_graphed(ctx, key, (int)(sizeof(key) / sizeof(key[0])), st, enqueue);
  if (rc) return rc;
  rc = mark_done(ctx, st);
  if (rc) return rc;
  if (!host_out) {  // nothing waits for this call: the next one must not overwrite its ks
    if (host_k) {
      if (!ctx->pin_busy) GGMS_CU(cudaEventCreateWithFlags(&ctx->pin_busy, cudaEventDisableTiming));
      GGMS_CU(cudaEventRecord(ctx->pin_busy, st));
    }
    return GGMS_OK;
  }
  GGMS_CU(cudaStreamSynchronize(st));
  if (pin_C->status != GGMS_E_INTERNAL) memcpy(out, pin_out, sizeof(T) * nk);
  return (int)pin_C->status;
}

template <typename T>
static int run_single(Context* ctx, const T* d_in, uint64_t n, const uint32_t* ks, uint64_t nk64,
                      T* out, const ggms_opts& o_in, cudaStream_t st, bool topk = false) {
  using K = typename KeyOf<T>::K;
  if (!d_in || n == 0 || n > 0xFFFFFFFFull || nk64 > 0x7FFFFFFFull) return GGMS_E_INVALID_ARG;
  if (nk64 == 0) return GGMS_OK;
  if ((!ks && !topk) || !out) return GGMS_E_INVALID_ARG;
  if (topk && nk64 > n) return GGMS_E_INVALID_ARG;
  ggms_opts o = o_in;
  if (topk) o.ks_on_device = 1;  // no k array to upload
  if ((uintptr_t)d_in % sizeof(T) != 0) return GGMS_E_INVALID_ARG;
  const uint32_t nk = (uint32_t)nk64;
  if (!o.ks_on_device) {
    for (uint32_t i = 0; i < nk; ++i)
      if (ks[i] < 1u || (uint64_t)ks[i] > n) return GGMS_E_INVALID_ARG;
  }
  if (direct_ok(ctx, o, n, nk, sizeof(T), topk)) return run_direct<T>(ctx, d_in, n, ks, nk, out, o, st, topk);
  Plan p;
  int rc = make_plan(&p, n, nk, o);
  if (rc) return rc;
  GGMS_CU(cudaSetDevice(ctx->device));
  const PassVariant<T>* pv = pass_variant<T>(o.pass_threads ? o.pass_threads : DEFAULT_PASS_NT,
                                              o.pass_unroll ? o.pass_unroll : DEFAULT_PASS_UNROLL);
  if (!pv) return GGMS_E_INVALID_ARG;
  pass_stages<T>(ctx, pv, p.B, p.ring_st);
  rc = l0_ncta<T>(ctx, pv, p.B, p.ring_st, &p.ncta);
  if (rc) return rc;
  Workspace<K> w0 = layout<K>(p, nullptr);
  rc = ensure_arena(ctx, w0.bytes);
  if (rc) return rc;
  Workspace<K> w = layout<K>(p, ctx->arena);
  const bool host_k = !o.ks_on_device && !topk, host_out = !o.out_on_device;
  const PinLayout pl = pin_layout(nk, sizeof(T), host_k, host_out);
  rc = ensure_pinned(ctx, pl.bytes);
  if (rc) return rc;
  Counters* pin_C = (Counters*)ctx->pinned;
  uint8_t* pin_k = ctx->pinned + pl.ks;
  uint8_t* pin_out = ctx->pinned + pl.out;

  const Caps caps{p.cap_seg, p.cap_tiles, p.nk, (uint32_t)(SMALL_SMEM / sizeof(K)), 0u, p.cap_rows};
  if (host_k && !topk) {
    // host side, every call: the previous call's upload from the same pinned
    // buffer may still be queued (calls with device-resident answers return
    // without a sync), so wait for it first
    if (ctx->pin_busy) GGMS_CU(cudaEventSynchronize(ctx->pin_busy));
    memcpy(pin_k, ks, 4ull * nk);
  }
  cudaEvent_t* prof = prof_slot(ctx);
  // the stream-ordered part: captured once and replayed when the call repeats
  auto enqueue = [&](cudaStream_t s) -> int {
    prof_rec(prof, 0, s);
    GGMS_CU(cudaMemsetAsync(w.C, 0, sizeof(Counters), s));
    const uint32_t* d_k = host_k ? (const uint32_t*)pin_k : ks;  // host ks: read once, from the pinned copy
    ++ctx->launches;
    if (topk)
      k_init_topk<<<cdiv(nk, 256), 256, 0, s>>>(nk, n, w.krank, w.kseg);
    else
      k_init_single<<<cdiv(nk, 256), 256, 0, s>>>(d_k, nk, n, w.krank, w.kseg, w.C);

    // ---- level-0 assigner
    const uint32_t S = p.S;
    const int cs_ctas = sort_cluster_ctas<K>(S);
    if (cs_ctas < 0) return GGMS_E_CUDA;
    if (cs_ctas) {  // draw the sample over the whole GPU, sort it in one cluster
      ctx->launches += 2;
      GGMS_CU(launch_pdl(asg_sample<T>, cdiv(S, 256), 256, 0, s, d_in, n, S, p.seed, w.samp_raw));
      const cudaError_t e_sort = cs_ctas == 16 ? launch_sort_cluster<K, 16>(s, w.samp_raw, S, w.samp_sorted)
                                               : launch_sort_cluster<K, 8>(s, w.samp_raw, S, w.samp_sorted);
      GGMS_CU(e_sort);
    } else {  // up to 4096 keys: draw them, then one CTA sorts them
      ctx->launches += 2;
      asg_sample<T><<<cdiv(S, 256), 256, 0, s>>>(d_in, n, S, p.seed, w.samp_raw);
      if (S <= 1024)
        asg_sort_chunks<K, 1024, 1024><<<1, 1024, 0, s>>>(w.samp_raw, w.samp_sorted, S);
      else if (S <= 2048)
        asg_sort_chunks<K, 2048, 1024><<<1, 1024, 0, s>>>(w.samp_raw, w.samp_sorted, S);
      else
        asg_sort_chunks<K, 4096, 1024><<<1, 1024, 0, s>>>(w.samp_raw, w.samp_sorted, S);
    }
    prof_rec(prof, 6, s);
    rc = setup_attrs<K>();
    if (rc) return rc;
    if (p.assigner == GGMS_ASSIGNER_SAMPLED) {
      ++ctx->launches;
      GGMS_CU(launch_pdl(setup_sampled<K>, 1, SETUP_NT, sizeof(SetupSmem<K>), s, w.samp_sorted, S, p.B, &w.asg[0],
                         &w.grid[0]));
    } else {
      // the sampled grid (fallback and judge) is built on a side stream while
      // the learned model's knots and statistics are computed: fork and join
      if (const int r_ = ensure_side(ctx)) return r_;
      GGMS_CU(cudaEventRecord(ctx->fork, s));
      GGMS_CU(cudaStreamWaitEvent(ctx->side, ctx->fork, 0));
      ++ctx->launches;
      setup_sampled<K><<<1, SETUP_NT, sizeof(SetupSmem<K>), ctx->side>>>(w.samp_sorted, S, p.B, &w.asg[0],
                                                                           &w.grid[0]);
      GGMS_CU(cudaEventRecord(ctx->join, ctx->side));
      rc = learn_and_choose<K>(p.assigner, w.samp_sorted, S, p.B, p.train_steps, p.bound, w.asg,
                               w.grid, w.learn, &w.C->asg_choice, w.krank, nk, n, p.window_z, s,
                               &ctx->launches, ctx->join, p.pl_knots);
      if (rc) return rc;
    }

    // ---- PASS 1 windows
    prof_rec(prof, 7, s);
    const bool windows = p.window_z >= 0.0f;
    if (windows) {
      ++ctx->launches;
      GGMS_CU(launch_pdl(l0_window<K>, 1, WIN_NT, l0_window_smem<K>(p.B), s, w.samp_sorted, S, w.krank, nk, n,
                         w.grid, w.C, p.window_z, w.win));
    }

    // ---- PASS 1: count
    const int grid_c = (int)p.ncta;
    // the histogram, the flags and k counts (and, without windows, the windows)
    static_assert(sizeof(Windows<K>) % 4 == 0, "zeroed as words");
    ++ctx->launches;
    GGMS_CU(launch_pdl(zero_words, 8, 1024, 0, s, w.hist0, p.B, w.aflag0, p.B / 32 + p.B,
                       windows ? (uint32_t*)nullptr : (uint32_t*)w.win, (uint32_t)(sizeof(Windows<K>) / 4)));
    prof_rec(prof, 1, s);
    ++ctx->launches;
    GGMS_CU(launch_pdl(pv->count, grid_c, pv->nt, l0_count_smem<T>(p.B, pv->nt, pv->unroll, p.ring_st[0]), s, d_in,
                       n, w.grid, w.C, w.win, w.hist0, w.crow, p.ring_st[0]));
    prof_rec(prof, 2, s);
    if (nk <= L0_FUSED_MAX_KS) {
      // scan, locate and the coarse-mode decision in one CTA
      ++ctx->launches;
      GGMS_CU(launch_pdl(l0_between<K>, 1, 1024, l0_between_smem(p.B), s, w.hist0, p.B, w.C, w.win, nk, w.krank,
                         w.kseg, w.kbin, w.kcnt0, w.aflag0, w.ic, w.aflagc));
    } else {
      ++ctx->launches;
      l0_scan<K><<<1, 1024, 4u * p.B, s>>>(w.hist0, p.B, w.C, w.win, w.aflagc);
      ++ctx->launches;
      lvl_locate_rows<<<cdiv(nk, 256), 256, 0, s>>>(w.hist0, p.B, nk, w.krank, w.kseg, nullptr, 0u, w.kbin,
                                                       w.aflag0, p.B / 32, w.C, w.kcnt0);
      // most buckets hold a k: copy groups of buckets instead (coarse mode)
      ++ctx->launches;
      l0_mode_ks<K><<<cdiv(nk, 256), 256, 0, s>>>(w.hist0, w.aflag0, p.B, w.win, w.C, w.ic, w.aflagc, nk, w.krank,
                                                   w.kseg, w.kbin);
    }
    ++ctx->launches;
    GGMS_CU(launch_pdl(l0_children<K>, cdiv(p.B, 256), 256, 0, s, w.hist0, w.aflag0, p.B, w.grid, w.C, w.win,
                       w.cmap0, w.segs[1], w.cursor[1], w.tiles[1], w.points, w.khead[1], w.smalls, w.bigs[1], caps,
                       w.ic, w.aflagc, w.kcnt0, tiny_keys<K>(), w.tinies));
    ++ctx->launches;
    GGMS_CU(launch_pdl(l0_relabel_bases<K>, ctx->sms * 4, 256, 0, s, w.cmap0, nk, w.kbin, w.kseg, w.kkey, w.points,
                       w.C, w.segs[1], w.khead[1], w.knext, w.crow, p.B, p.ncta, caps));
    // ---- PASS 2: compact the buckets that still need refinement
    prof_rec(prof, 3, s);
    ++ctx->launches;
    GGMS_CU(launch_pdl(pv->compact, grid_c, pv->nt, l0_compact_smem<T>(p.B, pv->nt, pv->unroll, p.ring_st[1]), s,
                       d_in, n, w.grid, w.C, w.win, w.cmap0, w.crow, w.cand[0], (uint64_t)n, p.ring_st[1],
                       w.hist0));
    ++ctx->launches;  // one of the two PASS-2 kernels returns at once
    GGMS_CU(launch_pdl(pv->coarse, grid_c, pv->nt, l0_coarse_smem<T>(pv->nt, pv->unroll, p.ring_st[2]), s, d_in,
                       n, w.grid, w.C, w.cmap0, w.crow, w.cand[0], (uint64_t)n, p.ring_st[2]));
    prof_rec(prof, 4, s);
    {
      // level 0 also has warp-sized children (l0_children); the refinement
      // levels of this path do not
      Caps c0 = caps;
      c0.tiny_keys = tiny_keys<K>();
      rc = launch_small_select<K>(ctx, w.cand[0], w.segs[1], w.khead[1], w, c0, s);
    }
    if (rc) return rc;

    // ---- refinement levels over candidates, answers
    rc = launch_refine<T>(ctx, refine_args<T>(w, ctx, n, nk, caps, host_out ? (T*)pin_out : out,
                                              host_out || o.stats ? pin_C : nullptr), s);
    if (rc) return rc;
    if (cudaGetLastError() != cudaSuccess) return GGMS_E_CUDA;
    prof_rec(prof, 8, s);  // nothing follows: the levels' launch writes the answers
    prof_rec(prof, 5, s);
    return GGMS_OK;
  };
  if (host_out || o.stats) pin_C->status = GGMS_E_INTERNAL;  // until the last launch reports
  if (o.stats || prof) {
    rc = enqueue(st);
  } else {
    const uint64_t key[] = {0x51Eull + sizeof(T) + (topk ? 256u : 0u) + (std::is_signed<T>::value ? 16u : 0u) +
                                (std::is_floating_point<T>::value ? 32u : 0u),
                            (uint64_t)(uintptr_t)d_in, n, host_k ? 1ull : (uint64_t)(uintptr_t)ks, nk,
                            host_out ? 1ull : (uint64_t)(uintptr_t)out,
                            (uint64_t)p.assigner | ((uint64_t)p.B << 8) | ((uint64_t)p.S << 24),
                            p.seed, (uint64_t)(uint32_t)p.train_steps | ((uint64_t)pv->nt << 32),
                            (uint64_t)pv->unroll | ((uint64_t)float_bits(p.bound) << 8),
                            (uint64_t)float_bits(p.window_z), (uint64_t)(uintptr_t)ctx->arena,
                            (uint64_t)(uintptr_t)ctx->pinned, (uint64_t)p.pl_knots, (uint64_t)ctx->barrier_limit};
    rc = run_graphed(ctx, key, (int)(sizeof(key) / sizeof(key[0])), st, enqueue);
  }
  if (rc) return rc;
  rc = mark_done(ctx, st);
  if (rc) return rc;
  if (host_k && !topk) {
    if (!ctx->pin_busy) GGMS_CU(cudaEventCreateWithFlags(&ctx->pin_busy, cudaEventDisableTiming));
    GGMS_CU(cudaEventRecord(ctx->pin_busy, st));
  }
  const bool need_sync = host_out || o.stats;
  if (!need_sync) return GGMS_OK;
  GGMS_CU(cudaStreamSynchronize(st));
  if (pin_C->status == GGMS_E_INTERNAL) return GGMS_E_INTERNAL;  // no answers, and no counters to report
  if (host_out) memcpy(out, pin_out, sizeof(T) * nk);
  if (o.stats) {
    ggms_stats* s = o.stats;
    Grid<K> a_used;
    GGMS_CU(cudaMemcpy(&a_used, &w.grid[pin_C->asg_choice], sizeof(Grid<K>), cudaMemcpyDeviceToHost));
    LearnState ls;
    GGMS_CU(cudaMemcpy(&ls, w.learn, sizeof(LearnState), cudaMemcpyDeviceToHost));
    s->assigner_used = (int32_t)a_used.kind;
    s->num_buckets = (int32_t)p.B;
    s->full_passes = (int32_t)pin_C->passes;
    s->levels = (int32_t)pin_C->levels_run;
    s->candidates = (int64_t)pin_C->cand0;
    s->refine_elements = (int64_t)pin_C->refine_elems;
    s->active_buckets = (int32_t)pin_C->active0;
    s->point_buckets = (int32_t)pin_C->point0;
    s->small_segments = (int32_t)pin_C->small_segs;
    s->sample_size = (int32_t)p.S;
    s->bucket_max_over_mean = (float)pin_C->max_bucket0 / ((float)n / (float)p.B);
    s->model_imbalance = (p.assigner == GGMS_ASSIGNER_SAMPLED) ? 0.0f : ls.imbalance;
    s->model_loss = p.assigner == GGMS_ASSIGNER_SAMPLED        ? 0.0f
                    : p.assigner == GGMS_ASSIGNER_LEARNED_MLP ? ls.mlp_loss
                                                              : ls.loss;
    s->window_runs = (int32_t)pin_C->win_runs;
    if (!o.pad0) s->model_segments = (p.assigner == GGMS_ASSIGNER_SAMPLED || a_used.kind == GGMS_ASSIGNER_SAMPLED)
                                         ? 0 : (int32_t)ls.M;
  }
  if (pin_C->status) return (int)pin_C->status;
  return GGMS_OK;
}


template <typename T>
static int run_single_tuned(Context* c, const T* d_in, uint64_t n, const uint32_t* ks, uint64_t nk, T* out,
                            const ggms_opts& o, cudaStream_t st, bool topk = false) {
  if (!o.autotune || o.num_buckets || o.pass_threads || o.pass_unroll || n == 0 || nk == 0)
    return run_single<T>(c, d_in, n, ks, nk, out, o, st, topk);
  ggms_opts b = o;
  b.autotune = 0;
  const bool direct = direct_ok(c, b, n, nk, sizeof(T), topk);  // the one launch is a candidate
  const uint64_t key[4] = {sizeof(T) | (std::is_signed<T>::value ? 16u : 0u) |
                               (std::is_floating_point<T>::value ? 32u : 0u) | (topk ? 64u : 0u),
                           (uint64_t)bitlen64(n) | ((uint64_t)bitlen64(nk) << 8),
                           (uint64_t)o.assigner | ((uint64_t)o.ks_on_device << 8) | ((uint64_t)o.out_on_device << 9) |
                               ((uint64_t)direct << 10),
                           (uint64_t)float_bits(o.window_z)};
  if (const Context::Tuned* t = tuned_find(c, key)) {
    b.num_buckets = t->B;
    b.pass_threads = t->nt;
    b.pass_unroll = t->unroll;
    return run_single<T>(c, d_in, n, ks, nk, out, b, st, topk);
  }
  static const int Bs[] = {4096, 8192, 16384};
  static const int shapes[][2] = {{1024, 4}, {1024, -2}, {512, 4}, {512, 8}};
  float best = 3.4e38f;
  Context::Tuned pick{{key[0], key[1], key[2], key[3]}, 8192, DEFAULT_PASS_NT, DEFAULT_PASS_UNROLL};
  if (direct) {
    const int rc = time_calls(st, [&] { return run_single<T>(c, d_in, n, ks, nk, out, b, st, topk); }, &best);
    if (rc) return rc;
    pick.B = pick.nt = pick.unroll = 0;
  }
  for (int B : Bs) {
    for (const auto& sh : shapes) {
      ggms_opts t = b;
      t.num_buckets = B;
      t.pass_threads = sh[0];
      t.pass_unroll = sh[1];
      float ms = 0.0f;
      const int rc = time_calls(st, [&] { return run_single<T>(c, d_in, n, ks, nk, out, t, st, topk); }, &ms);
      if (rc) return rc;
      if (ms < best) {
        best = ms;
        pick.B = B;
        pick.nt = sh[0];
        pick.unroll = sh[1];
      }
    }
  }
  c->tuned.push_back(pick);
  b.num_buckets = pick.B;
  b.pass_threads = pick.nt;
  b.pass_unroll = pick.unroll;
  return run_single<T>(c, d_in, n, ks, nk, out, b, st, topk);
}

template <typename T>
static int dropin(const T* d_vector, int length, const uint32_t* kVals, int numKs, T* outputs) {
  if (length <= 0 || numKs < 0) return GGMS_E_INVALID_ARG;
  Context* c = nullptr;
  int rc = default_context(&c);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(c->mu);
  ggms_opts o;
  ggms_default_opts(&o);
  return run_single<T>(c, d_vector, (uint64_t)length, kVals, (uint64_t)numKs, outputs, o, 0);
}

template <typename T>
static int topk_call(ggms_context* cx, const T* d_in, int64_t n, int64_t K, T* out,
                     const ggms_opts* opts, void* stream) {
  if (n <= 0 || K <= 0) return GGMS_E_INVALID_ARG;
  ggms_opts o;
  if (read_opts(opts, &o) != GGMS_OK) return GGMS_E_INVALID_ARG;
  Context* c = (Context*)cx;
  if (!c) {
    int rc = default_context(&c);
    if (rc) return rc;
  }
  std::lock_guard<std::mutex> lk(c->mu);
  return run_single_tuned<T>(c, d_in, (uint64_t)n, nullptr, (uint64_t)K, out, o, (cudaStream_t)stream, true);
}

template <typename T>
static int ex(ggms_context* cx, const T* d_in, int64_t n, const uint32_t* ks, int64_t nk, T* out,
              const ggms_opts* opts, void* stream) {
  if (n <= 0 || nk < 0) return GGMS_E_INVALID_ARG;
  ggms_opts o;
  if (read_opts(opts, &o) != GGMS_OK) return GGMS_E_INVALID_ARG;
  Context* c = (Context*)cx;
  if (!c) {
    int rc = default_context(&c);
    if (rc) return rc;
  }
  std::lock_guard<std::mutex> lk(c->mu);
  return run_single_tuned<T>(c, d_in, (uint64_t)n, ks, (uint64_t)nk, out, o, (cudaStream_t)stream);
}


// ------------------------------------------------------------------ batched segmented path
// Every segment by its length: a team of CTAs, one CTA or one warp
// (ggms_batch.cuh); the children that are still large go through the refinement
// levels, all segments' at once.
template <typename T>
static int run_segmented(Context* ctx, const T* d_in, const int64_t* seg_off, int64_t nseg64,
                         const uint32_t* ks, const int64_t* k_off, T* out, const ggms_opts& o,
                         cudaStream_t st) {
  using K = typename KeyOf<T>::K;
  if (!d_in || !seg_off || !k_off || nseg64 <= 0 || nseg64 > (1 << 30)) return GGMS_E_INVALID_ARG;
  if ((uintptr_t)d_in % sizeof(T) != 0) return GGMS_E_INVALID_ARG;
  const uint32_t nseg = (uint32_t)nseg64;
  GGMS_CU(cudaSetDevice(ctx->device));
  // the totals size the workspace: four words to pinned memory, one sync
  int rc = ensure_pinned(ctx, 64);
  if (rc) return rc;
  if (ctx->pin_busy) GGMS_CU(cudaEventSynchronize(ctx->pin_busy));
  int64_t* h = (int64_t*)ctx->pinned;
  GGMS_CU(cudaMemcpyAsync(&h[0], seg_off, 8, cudaMemcpyDeviceToHost, st));
  GGMS_CU(cudaMemcpyAsync(&h[1], seg_off + nseg, 8, cudaMemcpyDeviceToHost, st));
  GGMS_CU(cudaMemcpyAsync(&h[2], k_off, 8, cudaMemcpyDeviceToHost, st));
  GGMS_CU(cudaMemcpyAsync(&h[3], k_off + nseg, 8, cudaMemcpyDeviceToHost, st));
  GGMS_CU(cudaStreamSynchronize(st));
  if (h[0] != 0 || h[2] != 0 || h[1] < 0 || h[3] < 0) return GGMS_E_INVALID_ARG;
  const uint64_t n = (uint64_t)h[1];
  const uint64_t nk64 = (uint64_t)h[3];
  if (nk64 == 0) return GGMS_OK;
  if (n == 0 || n > 0xFFFFFFFFull || nk64 > 0x7FFFFFFFull || !ks || !out) return GGMS_E_INVALID_ARG;
  const uint32_t nk = (uint32_t)nk64;
  ggms_opts oo = o;
  oo.assigner = GGMS_ASSIGNER_SAMPLED;
  oo.num_buckets = 1024;
  oo.sample_size = 1024;
  Plan p;
  rc = make_plan(&p, n, nk, oo);
  if (rc) return rc;
  p.nlist = nseg;
  p.sms = (uint32_t)ctx->sms;
  rc = ensure_arena(ctx, layout<K>(p, nullptr).bytes);
  if (rc) return rc;
  const Workspace<K> w = layout<K>(p, ctx->arena);
  const Caps caps{p.cap_seg, p.cap_tiles, p.nk, (uint32_t)(SMALL_SMEM / sizeof(K)), 0u, p.cap_rows};
  // the stream-ordered part: captured once and replayed when the call repeats
  auto enqueue = [&](cudaStream_t s) -> int {
    GGMS_CU(cudaMemsetAsync(w.C, 0, sizeof(Counters), s));
    BatchArgs<T> a;
    a.in = d_in;
    a.seg_off = seg_off;
    a.k_off = k_off;
    a.ks = ks;
    a.nseg = nseg;
    a.n = n;
    a.seed = p.seed ^ 0x5E6A11ull;
    a.lists = w.lists;
    a.scratch = w.scratch;
    a.r = refine_args<T>(w, ctx, n, nk, caps, out, nullptr);
    if (const int r = launch_batch<T>(ctx, a, s)) return r;
    return launch_refine<T>(ctx, a.r, s);
  };
  if (o.stats || ctx->profile) {
    rc = enqueue(st);
  } else {
    const uint64_t key[] = {0x5E6ull + sizeof(T), (uint64_t)(uintptr_t)d_in, (uint64_t)(uintptr_t)seg_off, nseg,
                            (uint64_t)(uintptr_t)ks, (uint64_t)(uintptr_t)k_off, (uint64_t)(uintptr_t)out, n,
                            nk, (uint64_t)(uintptr_t)ctx->arena, (uint64_t)std::is_signed<T>::value,
                            (uint64_t)std::is_floating_point<T>::value, p.seed, (uint64_t)ctx->barrier_limit};
    rc = run_graphed(ctx, key, (int)(sizeof(key) / sizeof(key[0])), st, enqueue);
  }
  if (rc) return rc;
  rc = mark_done(ctx, st);
  if (rc) return rc;
  if (o.stats) {
    Counters hc;
    GGMS_CU(cudaMemcpyAsync(&hc, w.C, sizeof(Counters), cudaMemcpyDeviceToHost, st));
    GGMS_CU(cudaStreamSynchronize(st));
    memset(o.stats, 0, sizeof(ggms_stats));
    o.stats->levels = (int32_t)hc.levels_run;
    o.stats->refine_elements = (int64_t)hc.refine_elems;
    o.stats->full_passes = (int32_t)hc.passes;
    if (hc.status) return (int)hc.status;
  }
  return GGMS_OK;
}

template <typename T>
static int segmented(ggms_context* cx, const T* d_in, const int64_t* seg_off, int64_t nseg,
                     const uint32_t* ks, const int64_t* k_off, T* out, const ggms_opts* opts,
                     void* stream) {
  ggms_opts o;
  if (read_opts(opts, &o) != GGMS_OK) return GGMS_E_INVALID_ARG;
  Context* c = (Context*)cx;
  if (!c) {
    int rc = default_context(&c);
    if (rc) return rc;
  }
  std::lock_guard<std::mutex> lk(c->mu);
  return run_segmented<T>(c, d_in, seg_off, nseg, ks, k_off, out, o, (cudaStream_t)stream);
}



GGMS_END
