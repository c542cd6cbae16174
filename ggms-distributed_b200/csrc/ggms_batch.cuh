// ggms_batch.cuh -- the batched path: thousands of vectors of uneven length,
// each with its own ks.
//
// batch_init sorts the segments into classes by length, each with a persistent
// kernel of one CTA per SM:
//
//   teams    a segment longer than a CTA's equal share of the batch goes to a
//            team of CTAs: the one-vector steps of ggms_direct.cuh with the
//            barriers among the team.  All teams work at once, each with CTAs
//            for its length;
//   singles  a segment beyond one CTA's sort: the same steps by one CTA (its
//            barriers are CTA barriers), taken from a shared list, longer ones
//            first, so that the CTAs end together;
//   sorts    a segment of up to 32 KB: one CTA sorts it;
//   rows     up to 8 KB: one warp each.
//
// Children that are still large go to the refinement levels, which write the
// answers.
//
// What bounds it: a single CTA counts and copies with private shared-memory
// histograms and cursors, where tiles of a segment spread over CTAs paid a
// global cursor atomic per copied key: 2^30 fp32 in 4096 segments, 1 M ks:
// 13.3 ms then, 4.2 now, 18 cycles of an SM per 32 keys and pass.  That is the
// chain load -> bucket lookup -> atomic on one CTA of 32 warps per SM (64
// registers a thread), with no unit saturated: 2^27 keys in 4096 segments, issue
// slots 52 % and the shared-memory pipe 44 % busy (23 wavefronts per 32 keys
// over both passes, half of them bank conflicts).
#pragma once
#include "ggms_direct.cuh"

namespace ggms {

// Keys of a segment that one warp finishes (32-bit keys): two classes, whose
// warps hold 1024 and 2048 keys.  A warp takes 10 to 50 us for such a row and
// an SM holds 20 or 10 of them; a CTA sort takes 5 to 10 us and has the SM to
// itself.  So a warp is the better for many rows, and with fewer than
// BT_FEW rows per SM only for the shortest (126 rows of 900 fp32 keys: 52 us by
// warps, 8 by CTAs).
constexpr uint32_t BT_ROW0 = 1024, BT_ROW_FEW = 256, BT_FEW = 4;
// ks of a segment that one CTA selects one by one, where it would sort the
// segment for more.  3000 segments of 3000 fp32 keys, us for 1 / 2 / 3 ks and for
// the sort: normal 134 / 176 / 221 / 261, with ties 164 / 238 / 311 / 331; of 8000
// keys 159 / 213 / 262 / 462.
constexpr uint32_t BT_SELECT_KS = 3;

template <typename T>
struct BatchArgs {
  using K = typename KeyOf<T>::K;
  const T* in;
  const int64_t *seg_off, *k_off;
  const uint32_t* ks;
  uint32_t nseg;
  uint64_t n;
  uint64_t seed;
  uint32_t* lists;             // [BT_CLASSES][nseg] segments of each class
  uint32_t* scratch;           // per CTA: BT_SCRATCH words (a team uses its first CTA's)
  RefineArgs<T> r;
};
constexpr uint32_t BT_SCRATCH = 3 * DIRECT_MAX_B + 2 * (DIRECT_MAX_B / 32) + 32;

// Enqueues batch_init and the classes' kernels (ggms_batch.cu).
template <typename T>
int launch_batch(Context* ctx, const BatchArgs<T>& a, cudaStream_t s);

}  // namespace ggms

GGMS_BEGIN

// A segment's keys and ks; every range is clamped into its array.
struct SegRange {
  uint64_t off;
  uint32_t cnt, k0, nk;
};
template <typename T>
__device__ __forceinline__ SegRange seg_range(const BatchArgs<T>& a, uint32_t s, bool* bad) {
  const int64_t o0 = a.seg_off[s], o1 = a.seg_off[s + 1], q0 = a.k_off[s], q1 = a.k_off[s + 1];
  *bad = o1 < o0 || o0 < 0 || (uint64_t)o1 > a.n || q1 < q0 || q0 < 0 || q1 > (int64_t)a.r.nk;
  SegRange g{0, 0u, 0u, 0u};
  if (!*bad) g = SegRange{(uint64_t)o0, (uint32_t)(o1 - o0), (uint32_t)q0, (uint32_t)(q1 - q0)};
  return g;
}

// A CTA's equal share of the batch, but no fewer keys than repay a team's
// barriers.  Fewer segments than CTAs are longer than it.
__device__ __forceinline__ uint64_t batch_share(uint64_t n, uint32_t ncta) {
  return max((uint64_t)(1u << 18), n / ncta);
}

// Every segment into its class's list.  The ks start as taken by nobody, which
// the answers' kernel reports as an error; the answer of an invalid k is key 0.
template <typename T>
__global__ void batch_init(const __grid_constant__ BatchArgs<T> a, uint32_t ncta) {
  Counters* C = a.r.C;
  const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x, gs = gridDim.x * blockDim.x;
  for (uint32_t i = gt; i < a.r.nk; i += gs) {
    a.r.kseg[i] = K_OPEN;
    a.r.kkey[i] = 0;
  }
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t end = (a.nseg + 31u) & ~31u;  // whole warps: the appends below are per warp
  for (uint32_t s = gt; s < end; s += gs) {
    bool bad = false;
    uint32_t cls = BT_CLASSES;
    if (s < a.nseg) {
      const SegRange g = seg_range(a, s, &bad);
      if (bad) set_status(C, GGMS_E_INVALID_ARG);
      if (g.nk) {
        constexpr uint32_t CAP = direct_cap<typename KeyOf<T>::K>();
        if (g.cnt <= (a.nseg < BT_FEW * ncta ? BT_ROW_FEW : BT_ROW0 << 1)) {
          cls = BT_WARP + (g.cnt > BT_ROW0 ? 1u : 0u);
        } else if (g.cnt <= CAP) {
          cls = BT_SORT;
        } else {
          const uint64_t share = batch_share(a.n, ncta);
          cls = BT_TEAM;
          if (g.cnt <= share) {  // single: halves of the longest a single CTA gets
            cls = BT_SINGLE;
            while (cls + 1u < BT_SORT && (uint64_t)g.cnt << (cls + 1u - BT_SINGLE) <= share) ++cls;
          }
        }
      }
    }
    const uint32_t peers = __match_any_sync(FULL, cls);
    if (cls < BT_CLASSES) {
      uint32_t base = 0;
      const int leader = __ffs(peers) - 1;
      if ((int)lane == leader) base = atomicAdd(&C->nlist[cls], (uint32_t)__popc(peers));
      base = __shfl_sync(peers, base, leader);
      a.lists[(size_t)cls * a.nseg + base + __popc(peers & lanemask_lt())] = s;
    }
  }
}

// direct_body's task for one segment (thread 0 fills it in shared memory: its
// fields are read where they are used and hold no registers through the streams).
template <typename T>
__device__ __forceinline__ void batch_task(const BatchArgs<T>& a, uint32_t s, uint32_t first, uint32_t cta,
                                           uint32_t ncta, uint32_t* bar, DirectTask<T>& t) {
  bool bad = false;
  const SegRange g = seg_range(a, s, &bad);
  t.in = a.in + g.off;
  t.n = g.cnt;
  t.ks = a.ks + g.k0;
  t.nk = g.nk;
  t.seed = a.seed ^ ((uint64_t)s << 32);
  uint32_t B = g.cnt < (1u << 20) ? DIRECT_MAX_B / 2 : DIRECT_MAX_B;
  while (B > 1024u && B > g.cnt / 8u) B >>= 1;
  t.B = B;
  t.focus = 0u;
  t.slices = ncta > 1u && g.nk > 2048u ? 1u : 0u;
  t.ghist = a.scratch + (size_t)first * BT_SCRATCH;
  t.gcur = t.ghist + DIRECT_MAX_B;
  t.gact = t.gcur + DIRECT_MAX_B;
  t.gpt = t.gact + DIRECT_MAX_B / 32 + 32;
  t.bar = bar;
  t.cta = cta;
  t.ncta = ncta;
  t.off = g.off;
  t.k0 = g.k0;
}

constexpr uint32_t TEAM_PER = 8, TEAM_MAX_CTAS = 32 * TEAM_PER;  // segments per lane of the plan below

// Segments of teams, in a cooperative launch: the segments [nc round,
// nc (round + 1)) of the list (nc = gridDim.x; one round where the launch has
// the CTAs it asks for).  Every CTA computes who works on what: with
// ceil(length / T) CTAs a segment, for the smallest T (to 1/64) that the CTAs
// suffice for, no CTA has more than T keys to read.  (Teams of a half, a
// quarter, ... of the grid, one size after the other, and up to two shares to
// a single CTA: 64 segments of 2^20 u32 968 us, and 5 of 6 M 353; 303 and 159.)
template <typename T>
__global__ __launch_bounds__(DR_NT, 1) void batch_teams(const __grid_constant__ BatchArgs<T> a, uint32_t round) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ DirectTask<T> task;
  __shared__ uint32_t seg_s, first_s, size_s;
  Counters* C = a.r.C;
  const uint32_t me = blockIdx.x, nc = gridDim.x, lane = threadIdx.x & 31;
  if (me == 0 && threadIdx.x == 0 && round == 0) {  // the count and the copy read the segments beyond one CTA's sort
    uint32_t m = 0;
    for (uint32_t c = 0; c < BT_SORT; ++c) m += C->nlist[c];
    if (m) atomicAdd(&C->passes, 2u);
  }
  const uint32_t all = C->nlist[BT_TEAM], m = min(nc, all - min(all, nc * round));
  if (m == 0) return;
  if (threadIdx.x < 32) {
    if (lane == 0) size_s = 0u;
    const uint32_t* list = a.lists + (size_t)BT_TEAM * a.nseg + nc * round;
    uint32_t cnt[TEAM_PER], sum = 0, most = 0;  // (all segments together: n < 2^32 keys)
#pragma unroll
    for (uint32_t i = 0; i < TEAM_PER; ++i) {
      const uint32_t j = lane * TEAM_PER + i;
      bool bad = false;
      cnt[i] = j < m ? seg_range(a, list[j], &bad).cnt : 0u;
      sum += cnt[i];
      most = max(most, cnt[i]);
    }
    sum = __reduce_add_sync(FULL, sum);
    most = __reduce_max_sync(FULL, most);
    auto ctas = [&](uint32_t c, uint32_t t) { return c / t + (c % t ? 1u : 0u); };
    uint32_t lo = ctas(sum, nc), hi = most;  // hi suffices: a CTA each
    while (hi > lo && hi - lo > lo / 64u) {
      const uint32_t mid = lo + (hi - lo) / 2u;
      uint32_t need = 0;
#pragma unroll
      for (uint32_t i = 0; i < TEAM_PER; ++i) need += ctas(cnt[i], mid);
      if (__reduce_add_sync(FULL, need) <= nc) hi = mid; else lo = mid + 1u;
    }
    uint32_t mine = 0;
#pragma unroll
    for (uint32_t i = 0; i < TEAM_PER; ++i) mine += ctas(cnt[i], hi);
    uint32_t first = warp_incl_scan_u32(mine, lane) - mine;
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < TEAM_PER; ++i) {
      const uint32_t size = ctas(cnt[i], hi);
      if (me >= first && me < first + size) {
        seg_s = list[lane * TEAM_PER + i];
        first_s = first;
        size_s = size;
      }
      first += size;
    }
    __syncwarp();
    if (lane == 0 && size_s) batch_task<T>(a, seg_s, first_s, me - first_s, size_s, a.r.bar + first_s, task);
  }
  __syncthreads();
  if (size_s) direct_body<T, false, 4>(task, a.r, smem);
}

// Segments of single CTAs: CTA j takes the j-th, longest class first, so the
// hardware's scheduling deals them out as CTAs end.  (A persistent loop took
// registers from the streams: 0.24 ns per key and CTA against 0.15.)
template <typename T>
__global__ __launch_bounds__(DR_NT, 1) void batch_singles(const __grid_constant__ BatchArgs<T> a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ DirectTask<T> task;
  uint32_t cls = BT_SINGLE, j = blockIdx.x;
  for (; cls < BT_SORT; ++cls) {
    const uint32_t m = a.r.C->nlist[cls];
    if (j < m) break;
    j -= m;
  }
  if (cls == BT_SORT) return;
  if (threadIdx.x == 0) batch_task<T>(a, a.lists[(size_t)cls * a.nseg + j], 0u, 0u, 1u, a.r.bar, task);
  __syncthreads();
  direct_body<T, true, 4>(task, a.r, smem);
}

// The m keys of the CTA's registers that lie in [lo, hi], counted into 1024 bins
// uniform in key; thread t gets bin t's count and the inclusive count up to it.
// h: 1024 words, red: 32.  All threads call it; ends with a barrier.
template <typename K, int R>
__device__ __forceinline__ uint2 cta_bins(const K (&k)[R], uint32_t m, K lo, K hi, uint32_t* h, uint32_t* red) {
  const uint32_t tid = threadIdx.x;
  static_assert(DR_NT == 1 << 10, "a bin per thread");
  const int sh = max(0, bitlen((K)(hi - lo)) - 10);
  h[tid] = 0u;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < R; ++j)
    if (tid + j * DR_NT < m && k[j] >= lo && k[j] <= hi) atomicAdd(&h[(uint32_t)((K)(k[j] - lo) >> sh)], 1u);
  __syncthreads();
  const uint32_t c = h[tid];
  uint32_t v[1] = {c};
  block_scan_regs<1>(v, red);
  return make_uint2(c, v[0]);
}

// The key of rank r among those m keys in [lo, hi], whose bins are `b`: the bin
// of the rank is counted again, until it holds one key or one value.  red: 35.
template <typename K, int R>
__device__ __forceinline__ K cta_select(const K (&k)[R], uint32_t m, uint32_t r, K lo, K hi, uint2 b, uint32_t* h,
                                        uint32_t* red, K* one) {
  const uint32_t tid = threadIdx.x;
  while (lo < hi) {
    const int sh = max(0, bitlen((K)(hi - lo)) - 10);
    __syncthreads();  // (red is read until here)
    if (b.y > r && b.y - b.x <= r) {
      red[32] = tid;
      red[33] = b.y - b.x;
      red[34] = b.x;
    }
    __syncthreads();
    const K w = (K)(((K)1 << sh) - 1);
    lo = (K)(lo + ((K)red[32] << sh));
    if ((K)(hi - lo) > w) hi = (K)(lo + w);
    r -= red[33];
    if (red[34] == 1u && lo < hi) {
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (tid + j * DR_NT < m && k[j] >= lo && k[j] <= hi) *one = k[j];
      __syncthreads();
      return *one;
    }
    if (lo < hi) b = cta_bins(k, m, lo, hi, h, red);
  }
  return lo;
}

// Segments of one CTA's sort; with up to BT_SELECT_KS ks a selection each.
template <typename T>
__global__ __launch_bounds__(DR_NT, 1) void batch_sorts(const __grid_constant__ BatchArgs<T> a) {
  using K = typename KeyOf<T>::K;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ K red_k[2][DR_NT / 32];
  SortSmem<K>& sm = *reinterpret_cast<SortSmem<K>*>(smem);
  __shared__ uint32_t red[35], ks_s[BT_SELECT_KS];
  __shared__ K one;
  K* sorted = reinterpret_cast<K*>(smem + sizeof(SortSmem<K>));
  const uint32_t m = a.r.C->nlist[BT_SORT];
  for (uint32_t j = blockIdx.x; j < m; j += gridDim.x) {
    bool bad = false;
    const SegRange g = seg_range(a, a.lists[(size_t)BT_SORT * a.nseg + j], &bad);
    const T* in = a.in + g.off;
    if (g.nk <= BT_SELECT_KS) {
      constexpr int R = (int)(direct_cap<K>() / DR_NT);
      K k[R], mn = key_max<K>(), mx = 0;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const uint32_t i = threadIdx.x + q * DR_NT;
        if (i < g.cnt) k[q] = KeyOf<T>::to(in[i]);
      }
#pragma unroll
      for (int q = 0; q < R; ++q)
        if (threadIdx.x + q * DR_NT < g.cnt) {
          mn = min(mn, k[q]);
          mx = max(mx, k[q]);
        }
      if (threadIdx.x < g.nk) ks_s[threadIdx.x] = a.ks[g.k0 + threadIdx.x];  // (the same k for all threads)
      block_extremes(mn, mx, red_k);
      const uint2 all = cta_bins(k, g.cnt, mn, mx, &sm.hist[0][0], red);
      for (uint32_t i = 0; i < g.nk; ++i) {
        const uint32_t kk = ks_s[i];
        const bool ok = kk >= 1u && kk <= g.cnt;
        const K key = ok ? cta_select(k, g.cnt, g.cnt - kk, mn, mx, all, &sm.hist[0][0], red, &one) : (K)0;
        if (threadIdx.x == 0) {
          if (ok) a.r.kkey[g.k0 + i] = key;
          else set_status(a.r.C, GGMS_E_INVALID_ARG);
          a.r.kseg[g.k0 + i] = K_DONE;
        }
      }
      __syncthreads();
      continue;
    }
    sort_keys<K>(sm, g.cnt, red_k, [&](uint32_t i) { return KeyOf<T>::to(in[i]); },
                 [&](uint32_t i, K key) { sorted[i] = key; });
    for (uint32_t i = threadIdx.x; i < g.nk; i += DR_NT) {
      const uint32_t k = a.ks[g.k0 + i];
      if (k >= 1u && k <= g.cnt) a.r.kkey[g.k0 + i] = sorted[g.cnt - k];
      else set_status(a.r.C, GGMS_E_INVALID_ARG);
      a.r.kseg[g.k0 + i] = K_DONE;
    }
    __syncthreads();
  }
}

// One warp per segment of at most ROW keys: the keys are counted into ROW / 2
// bins uniform in key between the segment's extremes (for floats without the
// gap around zero, as in DirectMap), placed by bin, and each bin that holds a k
// put in order by one lane; every k then reads its rank.  The cost hardly
// depends on the number of ks, where a radix select pays four rounds per k (rows
// of 600 keys with 4-5 ks: 386 us for 12 M keys).  Up to 64 keys: every key's
// rank by comparison.
constexpr int RW_NT = 160;  // 5 warps: 4 and 2 CTAs per SM by shared memory
constexpr int RW_U = 4;     // keys in flight per lane (a lane's accesses are one long chain otherwise)
constexpr uint32_t RW_LANE = 24;
constexpr uint32_t RW_BISECT = 6;  // keys of a bin that repay counting them for a bit of one k, not sorting
template <typename K, uint32_t ROW>
struct RowSmem {
  K v[ROW], w[ROW];
  uint32_t h[ROW / 2];
};

template <typename T, uint32_t ROW>
__global__ __launch_bounds__(RW_NT) void rows_select(const __grid_constant__ BatchArgs<T> a) {
  pdl_entry();
  using K = typename KeyOf<T>::K;
  constexpr uint32_t RW_BINS = ROW / 2;
  constexpr int RW_BITS = ROW == BT_ROW0 ? 9 : 10;
  constexpr uint32_t CLS = BT_WARP + RW_BITS - 9;
  constexpr bool FP = std::is_floating_point<T>::value;
  constexpr K MID = (K)((K)1 << (sizeof(K) * 8 - 1));
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  RowSmem<K, ROW>& sm = reinterpret_cast<RowSmem<K, ROW>*>(smem)[warp];
  Counters* C = a.r.C;
  const uint32_t m = C->nlist[CLS];
  const uint32_t* list = a.lists + (size_t)CLS * a.nseg;
  const uint32_t gw = blockIdx.x * (RW_NT / 32) + warp, nw = gridDim.x * (RW_NT / 32);
  for (uint32_t t0 = gw; t0 < m; t0 += 32u * nw) {
    // lane j loads the j-th segment's ranges: the dependent loads once for 32
    SegRange mine{0, 0u, 0u, 0u};
    bool bad = false;
    if ((uint64_t)t0 + (uint64_t)lane * nw < m) mine = seg_range(a, list[t0 + lane * nw], &bad);
    for (uint32_t j = 0; j < 32u && (uint64_t)t0 + (uint64_t)j * nw < m; ++j) {
      const uint64_t off = __shfl_sync(FULL, mine.off, j);
      const uint32_t cnt = __shfl_sync(FULL, mine.cnt, j), k0 = __shfl_sync(FULL, mine.k0, j),
                     nk = __shfl_sync(FULL, mine.nk, j);
      const T* in = a.in + off;
      K* sorted = sm.w;
      if (cnt <= 64u) {
        const K ka = lane < cnt ? KeyOf<T>::to(in[lane]) : key_max<K>();
        const K kb = lane + 32u < cnt ? KeyOf<T>::to(in[lane + 32u]) : key_max<K>();
        sm.v[lane] = ka;
        sm.v[lane + 32u] = kb;
        __syncwarp();
        uint32_t ra = 0, rb = 0;
        for (uint32_t i = 0; i < cnt; ++i) {
          const K x = sm.v[i];
          ra += (x < ka || (x == ka && i < lane)) ? 1u : 0u;
          rb += (x < kb || (x == kb && i < lane + 32u)) ? 1u : 0u;
        }
        if (lane < cnt) sm.w[ra] = ka;
        if (lane + 32u < cnt) sm.w[rb] = kb;
        __syncwarp();
      } else {
        K lo = key_max<K>(), hi = 0, hn = 0, lp = key_max<K>();
        for (uint32_t i0 = lane; i0 < cnt; i0 += 32u * 8u) {  // eight loads in flight
          K x[8];
#pragma unroll
          for (int q = 0; q < 8; ++q)
            x[q] = i0 + q * 32u < cnt ? KeyOf<T>::to(in[i0 + q * 32u]) : (K)0;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (i0 + q * 32u < cnt) {
              sm.v[i0 + q * 32u] = x[q];
              lo = min(lo, x[q]);
              hi = max(hi, x[q]);
              if (FP && x[q] < MID) hn = max(hn, x[q]);
              if (FP && x[q] >= MID) lp = min(lp, x[q]);
            }
        }
        lo = warp_min(lo);
        hi = warp_max(hi);
        hn = warp_max(hn);
        lp = warp_min(lp);
        if (!FP || lo >= MID || hi < MID) hn = lp = hi;
        for (uint32_t b = lane; b < RW_BINS; b += 32u) sm.h[b] = 0u;
        __syncwarp();
        const K range = (K)((hn - lo) + (hi - lp));
        const uint32_t sh = (uint32_t)max(0, bitlen(range) - RW_BITS);
        static_assert(RW_BINS == 1u << RW_BITS, "two keys a bin");
        auto bin = [&](K k) -> uint32_t {
          return FP ? (uint32_t)((K)((min(k, hn) - lo) + (max(k, lp) - lp)) >> sh) : (uint32_t)((K)(k - lo) >> sh);
        };
        for (uint32_t i0 = lane; i0 < cnt; i0 += 32u * RW_U) {
          uint32_t b[RW_U];
#pragma unroll
          for (int q = 0; q < RW_U; ++q) b[q] = bin(i0 + q * 32u < cnt ? sm.v[i0 + q * 32u] : lo);
#pragma unroll
          for (int q = 0; q < RW_U; ++q)
            if (i0 + q * 32u < cnt) atomicAdd(&sm.h[b[q]], 1u);
        }
        __syncwarp();
        uint32_t run = 0;
        for (uint32_t b0 = 0; b0 < RW_BINS; b0 += 32u) {
          const uint32_t x = sm.h[b0 + lane];
          const uint32_t inc = warp_incl_scan_u32(x, lane);
          sm.h[b0 + lane] = run + inc - x;
          run += __shfl_sync(FULL, inc, 31);
        }
        __syncwarp();
        for (uint32_t i0 = lane; i0 < cnt; i0 += 32u * RW_U) {
          K k[RW_U];
          uint32_t at[RW_U];
#pragma unroll
          for (int q = 0; q < RW_U; ++q) k[q] = i0 + q * 32u < cnt ? sm.v[i0 + q * 32u] : lo;
#pragma unroll
          for (int q = 0; q < RW_U; ++q) at[q] = i0 + q * 32u < cnt ? atomicAdd(&sm.h[bin(k[q])], 1u) : 0u;
#pragma unroll
          for (int q = 0; q < RW_U; ++q)
            if (i0 + q * 32u < cnt) sm.w[at[q]] = k[q];
        }
        __syncwarp();
        // h[b] is now the end of bin b
        auto sort_few = [&](uint32_t s0, uint32_t e) {  // one lane: insertion sort
          for (uint32_t i = s0 + 1u; i < e; ++i) {
            const K x = sm.w[i];
            uint32_t p = i;
            for (; p > s0 && sm.w[p - 1u] > x; --p) sm.w[p] = sm.w[p - 1u];
            sm.w[p] = x;
          }
        };
        auto sort_bin = [&](uint32_t c0, uint32_t len) {  // the warp: bitonic, in v (the row's copy is no longer needed)
          uint32_t N = 64;
          while (N < len) N <<= 1;
          for (uint32_t i = lane; i < N; i += 32u) sm.v[i] = i < len ? sm.w[c0 + i] : key_max<K>();
          __syncwarp();
          for (uint32_t kk = 2; kk <= N; kk <<= 1)
            for (uint32_t jj = kk >> 1; jj > 0; jj >>= 1) {
              for (uint32_t t = lane; t < N / 2; t += 32u) {  // pair t: i has bit jj clear
                const uint32_t i = ((t & ~(jj - 1u)) << 1) | (t & (jj - 1u));
                const K x = sm.v[i], y = sm.v[i | jj];
                if ((x > y) == ((i & kk) == 0)) { sm.v[i] = y; sm.v[i | jj] = x; }
              }
              __syncwarp();
            }
          for (uint32_t i = lane; i < len; i += 32u) sm.w[c0 + i] = sm.v[i];
          __syncwarp();
        };
        auto extremes = [&](uint32_t c0, uint32_t len, K& mn, K& mx) {
          mn = key_max<K>();
          mx = 0;
          for (uint32_t i = lane; i < len; i += 32u) {
            mn = min(mn, sm.w[c0 + i]);
            mx = max(mx, sm.w[c0 + i]);
          }
          mn = warp_min(mn);
          mx = warp_max(mx);
        };
        if (nk <= 32u) {
          // lane j puts the j-th k's bin in order (the first of the lanes with
          // the same bin); a larger bin, a dense spot of the keys, is the
          // warp's.  20,000 rows of 600 keys with one k each: 101 us, and 142 when
          // half of the keys are zero; ordering all bins took 203 and 478.
          const uint32_t k = lane < nk ? a.ks[k0 + lane] : 0u, r = cnt - k;
          const bool ok = k >= 1u && k <= cnt;
          uint32_t b = RW_BINS + lane, s0 = 0, e = 0;
          if (ok) {
            uint32_t l = 0, u = RW_BINS - 1u;
            while (l < u) {
              const uint32_t mid = (l + u) >> 1;
              if (sm.h[mid] > r) u = mid; else l = mid + 1u;
            }
            b = l;
            s0 = b ? sm.h[b - 1u] : 0u;
            e = sm.h[b];
          }
          const uint32_t peers = __match_any_sync(FULL, b);
          const bool first = ok && __ffs(peers) - 1 == (int)lane;
          if (first && e - s0 <= RW_LANE) sort_few(s0, e);
          bool found = false;
          K ans = 0;
          for (uint32_t todo = __ballot_sync(FULL, first && e - s0 > RW_LANE); todo; todo &= todo - 1u) {
            const int src = __ffs(todo) - 1;
            const uint32_t c0 = __shfl_sync(FULL, s0, src), len = __shfl_sync(FULL, e, src) - c0;
            uint32_t who = __shfl_sync(FULL, peers, src);
            K mn, mx;
            extremes(c0, len, mn, mx);
            if (mn == mx) continue;
            if ((uint32_t)(__popc(who) * bitlen((K)(mx - mn))) * RW_BISECT > len) {
              sort_bin(c0, len);
              continue;
            }
            for (; who; who &= who - 1u) {  // the smallest key with more than `at` keys up to it
              const int j = __ffs(who) - 1;
              const uint32_t at = __shfl_sync(FULL, r, j) - c0;
              K lo_k = mn, hi_k = mx;
              while (lo_k < hi_k) {  // two bits a round: the loads are what it waits for
                const K q = (K)((hi_k - lo_k) / 4u), h = (K)((hi_k - lo_k) / 2u);
                const K p1 = (K)(lo_k + q), p2 = (K)(lo_k + h), p3 = (K)(lo_k + h + q);
                uint32_t n1 = 0, n2 = 0, n3 = 0;
#pragma unroll 4
                for (uint32_t i = lane; i < len; i += 32u) {
                  const K x = sm.w[c0 + i];
                  n1 += x <= p1 ? 1u : 0u;
                  n2 += x <= p2 ? 1u : 0u;
                  n3 += x <= p3 ? 1u : 0u;
                }
                n1 = __reduce_add_sync(FULL, n1);
                n2 = __reduce_add_sync(FULL, n2);
                n3 = __reduce_add_sync(FULL, n3);
                if (n3 <= at) lo_k = (K)(p3 + 1u);
                else if (n2 <= at) { lo_k = (K)(p2 + 1u); hi_k = p3; }
                else if (n1 <= at) { lo_k = (K)(p1 + 1u); hi_k = p2; }
                else hi_k = p1;
              }
              if ((int)lane == j) {
                ans = lo_k;
                found = true;
              }
            }
          }
          __syncwarp();
          if (lane < nk) {
            if (ok) a.r.kkey[k0 + lane] = found ? ans : sm.w[r];
            else set_status(C, GGMS_E_INVALID_ARG);
            a.r.kseg[k0 + lane] = K_DONE;
          }
          __syncwarp();
          continue;
        }
        // many ks: every bin, a lane each (large ones: the warp, unless all their keys are equal)
        for (uint32_t b0 = 0; b0 < RW_BINS; b0 += 32u) {
          const uint32_t b = b0 + lane, e = sm.h[b], s0 = b ? sm.h[b - 1u] : 0u;
          const uint32_t large = __ballot_sync(FULL, e - s0 > RW_LANE);
          if (e - s0 <= RW_LANE) sort_few(s0, e);
          for (uint32_t todo = large; todo; todo &= todo - 1u) {
            const int src = __ffs(todo) - 1;
            const uint32_t c0 = __shfl_sync(FULL, s0, src), len = __shfl_sync(FULL, e, src) - c0;
            K mn, mx;
            extremes(c0, len, mn, mx);
            if (mn != mx) sort_bin(c0, len);
          }
        }
        __syncwarp();
      }
      for (uint32_t i = lane; i < nk; i += 32u) {
        const uint32_t k = a.ks[k0 + i];
        if (k >= 1u && k <= cnt) a.r.kkey[k0 + i] = sorted[cnt - k];
        else set_status(C, GGMS_E_INVALID_ARG);
        a.r.kseg[k0 + i] = K_DONE;
      }
      __syncwarp();
    }
  }
}

GGMS_END
