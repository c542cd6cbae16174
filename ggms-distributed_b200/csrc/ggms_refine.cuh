// ggms_refine.cuh -- the refinement levels and the answers in one launch.
//
// After level 0 a few segments may still be too large for the finishers.  Up
// to three (32-bit keys) or six (64-bit) radix levels refine them: count,
// scan, locate, children, relabel + copy, and the CTA finisher for the
// children that became small.  refine_levels runs all of them as ONE
// cooperative launch whose CTAs meet at grid barriers, and then writes the
// answers (converted to the caller's type, straight to where the caller wants
// them: device memory, or pinned host memory when the answers go to the host).
//
// What bounds it: latency.  A level is seven short steps; launched as kernels
// they cost about 4 us each whether or not a segment is left (the batched path
// launched 28 of them per call for nothing: 130 us of a 525 us call on 20,000
// short rows), a barrier of resident CTAs about 1.5 us, and a call without
// segments to refine pays one launch.  The levels hold too little work to lose
// anything to the fixed grid.
#pragma once
#include "ggms_host.cuh"
#include "ggms_kernels.cuh"

namespace ggms {

constexpr uint32_t RF_TINY = 4096;  // bytes of keys of a child that one warp finishes

template <typename T>
struct RefineArgs {
  using K = typename KeyOf<T>::K;
  Counters* C;
  uint32_t* bar;               // the arena's barrier word
  uint32_t* left;              // CTAs that have left the launch (the word after the barriers' words)
  long long limit;             // cycles a barrier may take
  K* cand[2];
  Seg<K>* segs[2];
  TileRef* tiles[2];
  uint32_t *rows[2], *aflag[2], *bigs[2], *cursor[2], *khead[2];
  uint32_t *knext, *smalls, *tinies, *krank, *kseg, *kbin;
  K *points, *kkey;
  uint32_t nk;
  Caps caps;
  T* out;                      // answers, in the caller's k order
  Counters* report;            // pinned copy of the counters (null: not wanted)
};

// Launches refine_levels on s (ggms_refine.cu).  bar: a zero-initialised word
// that only these launches touch.
template <typename T>
int launch_refine(Context* ctx, const RefineArgs<T>& a, cudaStream_t s);

}  // namespace ggms

GGMS_BEGIN

// Barrier over ncta CTAs of a cooperative launch (all resident at once), one of
// them the leader.  It adds 2^31 - (ncta - 1), the others 1: when all have arrived the top bit
// has flipped and the low bits are back where they were, so the word needs no
// reset between barriers or launches.  In two halves: what the CTA did before
// arrive() is visible to a CTA after its wait().  The wait is bounded by `limit`
// cycles (negative: it gives up at once): false for the whole CTA, with the
// status set, when it ran out.
struct GridBarrier {
  uint32_t old;  // thread 0's
  __device__ __forceinline__ void arrive(uint32_t* bar, uint32_t ncta, bool leader) {
    __syncthreads();
    if (threadIdx.x == 0 && ncta > 1u) {
      __threadfence();
      old = atomicAdd(bar, leader ? 0x80000000u - (ncta - 1u) : 1u);
    }
  }
  __device__ __forceinline__ bool wait(uint32_t* bar, uint32_t ncta, Counters* C, long long limit) {
    bool good = true;
    if (threadIdx.x == 0 && ncta > 1u) {
      const long long t0 = clock64();
      good = limit >= 0;
      while (good) {
        uint32_t now;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(bar) : "memory");
        if ((now ^ old) & 0x80000000u) break;
        good = clock64() - t0 <= limit;
      }
      if (!good) {
        set_status(C, GGMS_E_INTERNAL);
        atomicExch(&C->failed, 1u);
      }
      __threadfence();
    }
    return __syncthreads_and(good) != 0;
  }
};

__device__ __forceinline__ bool grid_barrier(uint32_t* bar, uint32_t ncta, bool leader, Counters* C,
                                             long long limit) {
  GridBarrier b;
  b.arrive(bar, ncta, leader);
  return b.wait(bar, ncta, C, limit);
}

// Every k's answer; a k that is not resolved is an error.  out may be pinned
// host memory: consecutive threads write consecutive answers.
template <typename T>
__device__ __forceinline__ void write_out_body(const typename KeyOf<T>::K* k_key, const uint32_t* k_seg, uint32_t nk,
                                               T* out, Counters* C, uint32_t cta, uint32_t ncta) {
  for (uint32_t i = cta * blockDim.x + threadIdx.x; i < nk; i += ncta * blockDim.x) {
    if (k_seg[i] != K_DONE) set_status(C, GGMS_E_NOT_CONVERGED);
    out[i] = KeyOf<T>::from(k_key[i]);
  }
}

// The end of a call's last cooperative launch: every CTA comes here, also one
// whose barrier ran out, and the last copies the counters to pinned host memory
// (the host reads the status and statistics after its sync).  A barrier that
// ran out, here or in batch_teams, has left its word between two barriers;
// nobody waits any more, so the last CTA zeroes the words for the next call.
// *left is 0 before and after; it is no counter of the call, whose zeroing a
// CTA may still have before it when another one gives up.  All threads call it.
__device__ __forceinline__ void leave_body(const Counters* C, uint32_t* bar, uint32_t* left, Counters* report,
                                           uint32_t ncta) {
  __shared__ uint32_t last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(left, 1u) + 1u == ncta ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  if (__ldcg(&C->failed))
    for (uint32_t* w = bar + threadIdx.x; w < left; w += blockDim.x) *w = 0u;
  if (threadIdx.x == 0) *left = 0u;
  if (report)
    for (uint32_t w = threadIdx.x; w < sizeof(Counters) / 4; w += blockDim.x)
      reinterpret_cast<uint32_t*>(report)[w] = __ldcg(reinterpret_cast<const uint32_t*>(C) + w);
}

constexpr int RF_NT = 512;
constexpr int RF_WARPS = RF_NT / 32;         // warps that finish a CTA's tiny children (all, or half in direct_select)

// The levels first..: level l refines the segments of pool l & 1, reads
// cand[(l - 1) & 1] and writes cand[l & 1].  Returns false after a barrier
// that ran out.  smem: SMALL_SELECT_SMEM bytes.
template <typename T, int NT>
__device__ __forceinline__ bool refine_body(const RefineArgs<T>& a, uint8_t* smem) {
  using K = typename KeyOf<T>::K;
  constexpr int MAXLEV = (KeyBits<K>::value + RADIX_BITS - 1) / RADIX_BITS;
  static_assert(RF_WARPS * (RF_TINY + 1024u) <= SMALL_SELECT_SMEM, "the warps' slices fit");
  static_assert(COMPACT_SMEM<K, NT> <= SMALL_SELECT_SMEM, "the bins of a level and its queues fit");
  __shared__ uint32_t red[72];
  Counters* C = a.C;
  const uint32_t cta = blockIdx.x, ncta = gridDim.x;
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem);
  for (int l = 1; l <= MAXLEV; ++l) {
    const int p = l & 1, q = p ^ 1;
    if (__ldcg(&C->nbig[p]) == 0u) break;  // the same for every CTA: written before the last barrier
    const K* src = a.cand[(l - 1) & 1];
    K* dst = a.cand[l & 1];
    prep_body(a.rows[p], a.aflag[p], C, p, a.caps, cta, ncta);
    if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    count_body<K, NT>(src, a.segs[p], a.tiles[p], C, p, a.rows[p], a.caps, bins, cta, ncta);
    if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    scan_body<NT>(a.rows[p], C, p, a.caps, red, cta, ncta);
    if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    for (uint32_t i = cta * NT + threadIdx.x; i < a.nk; i += ncta * NT)
      locate_in_row(i, a.rows[p], NBIN, a.krank, a.kseg, &a.segs[p]->row, sizeof(Seg<K>) / 4, a.kbin, a.aflag[p],
                    NBIN_WORDS, C, nullptr);
    if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    children_body<K, NT>(a.rows[p], a.aflag[p], a.segs[p], C, p, a.segs[q], a.cursor[q], a.tiles[q], a.points,
                         a.khead[q], a.smalls, a.tinies, a.bigs[p], a.bigs[q], a.caps, cta, ncta);
    if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    for (uint32_t i = cta * NT + threadIdx.x; i < a.nk; i += ncta * NT) {
      const uint32_t s = a.kseg[i];
      if (s < K_OPEN)
        relabel_one<K>(i, a.rows[p][(size_t)a.segs[p][s].row * NBIN + a.kbin[i]], a.kseg, a.kkey, a.points, C, a.segs[q],
                       a.khead[q], a.knext);
    }
    if (l < MAXLEV)
      compact_body<K, NT>(src, a.segs[p], a.tiles[p], C, p, a.rows[p], a.segs[q], a.cursor[q], dst, a.caps, bins,
                          cta, ncta);
    if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    if (l < MAXLEV) {
      // children of up to RF_TINY bytes: a warp each, in the space of the CTA
      // finisher (2^28 keys, 2^14 ks: 16 K children of ~500 keys, 260 us at a
      // CTA each)
      constexpr uint32_t TK = RF_TINY / sizeof(K);
      K* slices = reinterpret_cast<K*>(smem);
      if (threadIdx.x < RF_WARPS * 32)
        tiny_select_body<K, RF_WARPS, TK>(dst, a.segs[q], a.tinies, C, a.khead[q], a.knext, a.krank, a.kseg,
                                        a.kkey, a.caps, slices,
                                        reinterpret_cast<uint32_t*>(slices + RF_WARPS * TK), cta, ncta, a.nk);
      __syncthreads();
      small_select_body<K, NT>(dst, a.segs[q], a.smalls, C, a.khead[q], a.knext, a.krank, a.kseg, a.kkey,
                               a.caps.small_keys, a.caps, smem, cta, ncta);
      if (!grid_barrier(a.bar, ncta, cta == 0u, C, a.limit)) return false;
    }
  }
  return true;
}

template <typename T>
__global__ __launch_bounds__(RF_NT, 2) void refine_levels(const __grid_constant__ RefineArgs<T> a) {
  extern __shared__ __align__(128) uint8_t smem[];
  // (after a team's barrier ran out the segments are incomplete and its words unusable)
  if (!__ldcg(&a.C->failed) && refine_body<T, RF_NT>(a, smem))
    write_out_body<T>(a.kkey, a.kseg, a.nk, a.out, a.C, blockIdx.x, gridDim.x);
  leave_body(a.C, a.bar, a.left, a.report, gridDim.x);
}

GGMS_END
