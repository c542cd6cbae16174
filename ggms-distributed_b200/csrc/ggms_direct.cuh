// ggms_direct.cuh -- one vector in one launch: the path of vectors whose second
// read comes from the L2 cache, all or most of it (up to 160 MB; fewer keys with
// many ks: direct_ok).
//
// The two-pass pipeline (ggms_engine.cuh) spends ~100 us around its passes on
// chains of one-CTA kernels (sample sort, model, windows, scan, children,
// finishers), which is repaid only when the passes themselves are long.  For
// such a vector a re-read costs little, so this path keeps the shape (sample ->
// buckets -> count -> copy -> finish) and drops the chain: one cooperative
// launch of four grid barriers (five with many ks, more when large children are
// left), and between the barriers every CTA computes the same small things for
// itself instead of waiting for one CTA to compute them.
//
//   1. every CTA draws the same sample (up to 4096 keys), histograms it over
//      2048 cells uniform in key between its extremes, and turns the cells'
//      prefix sums into a piecewise-linear map key -> bucket (DirectMap);
//   2. it counts its share of the input into a shared-memory histogram and
//      adds that to the global one, which all have zeroed meanwhile (a barrier
//      before and one after);
//   3. it scans the global histogram, locates the ks (many ks: its own, and a
//      barrier), and knows the buckets
//      holding a k (the children) and where each child's keys go in a compact
//      candidate array;
//   4. it reserves a range of every child it holds keys of (one global atomic
//      per child), re-reads its share and copies the keys (barrier);
//   5. the candidate array is in key order up to the order inside each child:
//      every CTA sorts an equal part of it, whole children at a time (barrier),
//      and every k reads its answer at its position.
//
// Step 5 sorts where a selection would do: with children of a few dozen keys a
// selection per k pays for its k lists and histograms whatever the size (2^22
// fp32, 2^14 ks: 390 us of finishing against 30 us), and ks that share a child
// cost nothing extra.  A child of more than 32 KB goes to the
// refinement levels.
// A bucket that only one key can be in (integers of a small range, floats in a
// few units of the last place: more buckets than keys) is no child: its key is
// its ks' answer.  A large child whose keys turn out to be one value (floats of
// 16-bit precision) answers its ks once its true key range is known, and the
// levels, which start from that range, do not read it (40 M fp32, half of them
// zero, one k: 289 us, 329 with a level over them; 19 M of bfloat16 precision,
// 2000 ks: 835 and 919).
//
// A vector that fits one CTA's sort (32 KB) is sorted by it (direct_sort):
// nothing else is as short.
#pragma once
#include "ggms_refine.cuh"

namespace ggms {

constexpr uint32_t DIRECT_MAX_B = 16384;  // buckets
constexpr uint32_t DIRECT_SAMPLE = 4096;  // sampled keys
constexpr uint32_t DIRECT_CELLS = 2048;   // cells of the map
constexpr uint32_t DIRECT_EXT = 16;       // ... of them beyond each extreme of the sample
constexpr uint32_t DIRECT_GAP = 128;      // ... and on each side of the gap around zero (DirectMap)
// A cell's weight: WT per sampled key, WT more for its sampled keys or for the
// mean of its and its four neighbours', whichever is larger, and CELL_WT for
// having keys at all.  Cells hold a sampled key or six: one that drew none by
// chance would be a single bucket of 26,000 keys of 2^23, and a set of 300 ks
// met such a bucket every other time (50 us of levels).  Keys in buckets of
// more than 8192, 2^24 to 2^25 keys, 16384 buckets: normal 0.08 to 0.7 %
// without the neighbours, none with them; Cauchy 0.4 to 1.3 %, 0 to 0.04 %;
// narrow modes keep their buckets, which they lose to a plain smoothing (1.4 %
// to 15 % of a mixture of eight; 0.9 % with the larger of the two).
constexpr uint32_t DIRECT_WT = 4, DIRECT_CELL_WT = 4;

template <typename T>
struct DirectArgs {
  using K = typename KeyOf<T>::K;
  const T* in;
  uint64_t n;
  const uint32_t* ks;          // null: top-k, k_i = i + 1
  uint64_t seed;
  uint32_t B;                  // buckets: a power of two, 1024 .. DIRECT_MAX_B
  uint32_t focus;              // 1: clustered ks get most of the buckets
  uint32_t slices;             // 1: every CTA locates its own ks only (one more barrier)
  uint32_t *ghist, *gcur;      // [B] bucket counts, keys copied so far
  uint32_t* gact;              // [B / 32] buckets holding a k (slices)
  uint32_t* gpt;               // [B / 32 + B] buckets of one key, a sampled position of each
  RefineArgs<T> r;             // workspace of the large children (pool 1) and where the answers go
};

// Launches direct_select over `ctas` CTAs, or direct_sort (ggms_direct.cu).
template <typename T>
int launch_direct(Context* ctx, const DirectArgs<T>& a, unsigned ctas, cudaStream_t s);

}  // namespace ggms

GGMS_BEGIN

constexpr int DR_NT = 1024;

constexpr uint32_t K_SORTED = 0xFFFFFFFEu;   // k_seg value: the answer is at cand[k_rank] once that is sorted

// Monotone map key -> bucket: keys are clamped to the sample's range; cell c
// holds the buckets [base, base + span), spread linearly over its keys.
// TWO (a floating sample of both signs): the range leaves out the keys between
// the sample's largest negative and smallest positive value.  Those differ by
// hundreds of octaves of ever smaller magnitudes that hold next to no values
// but would take nearly all the cells (4 per octave of a normal sample, 73
// without them).
// HI: only the key's high word decides (64-bit keys whose sample spans at
// least 2^16 high words): the passes are bound by integer instructions, and
// the word's clamp, subtraction and interpolation cost a third of the 64-bit
// ones.
template <typename K, bool TWO, bool HI>
struct DirectMap {
  using D = typename std::conditional<HI, uint32_t, K>::type;
  D lo, hi, hn, lp;     // [lo, hi], or TWO: [lo, hn] and [lp, hi]
  uint32_t csh;
  const uint32_t* tab;  // shared memory: base | span << 16 (B <= 32768)
  __device__ __forceinline__ D dist(D k) const {
    if constexpr (TWO) return (D)((min(max(k, lo), hn) - lo) + (min(max(k, lp), hi) - lp));
    else return (D)(min(max(k, lo), hi) - lo);
  }
  __device__ __forceinline__ uint32_t operator()(K key) const {
    D k;
    if constexpr (HI) k = (uint32_t)(key >> 32);
    else k = key;
    const D d = dist(k);
    const uint32_t e = tab[(uint32_t)(d >> csh)];
    if constexpr (sizeof(D) == 4) {
      return (e & 0xFFFFu) + __umulhi(__funnelshift_lc(0u, (uint32_t)d, 32u - csh), e >> 16);
    } else {
      return (e & 0xFFFFu) + grid_lin((D)(d & (D)(((D)1 << csh) - 1)), e >> 16, csh);
    }
  }
};

__device__ __forceinline__ uint32_t warp_min(uint32_t v) { return __reduce_min_sync(FULL, v); }
__device__ __forceinline__ uint32_t warp_max(uint32_t v) { return __reduce_max_sync(FULL, v); }
__device__ __forceinline__ uint64_t warp_min(uint64_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, (uint64_t)__shfl_xor_sync(FULL, (unsigned long long)v, o));
  return v;
}
__device__ __forceinline__ uint64_t warp_max(uint64_t v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, (uint64_t)__shfl_xor_sync(FULL, (unsigned long long)v, o));
  return v;
}

template <typename K>
__device__ __forceinline__ void key_atomic_min(K* p, K v) {
  if constexpr (sizeof(K) == 4) atomicMin(p, v);
  else atomicMin(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
}
template <typename K>
__device__ __forceinline__ void key_atomic_max(K* p, K v) {
  if constexpr (sizeof(K) == 4) atomicMax(p, v);
  else atomicMax(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
}

// Inclusive scan over the block of V consecutive values per thread (thread t
// holds elements V t ..), in registers.  red: 32 words.  Ends with a barrier.
template <int V>
__device__ __forceinline__ void block_scan_regs(uint32_t (&v)[V], uint32_t* red) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 1; i < V; ++i) v[i] += v[i - 1];
  const uint32_t inc = warp_incl_scan_u32(v[V - 1], lane);
  if (lane == 31) red[warp] = inc;
  __syncthreads();
  const uint32_t w = warp_incl_scan_u32(red[lane], lane);  // every warp scans the warp totals
  const uint32_t prev = __shfl_sync(FULL, w, (warp + 31u) & 31u);
  const uint32_t before = inc - v[V - 1] + (warp ? prev : 0u);
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] += before;
  __syncthreads();
}

// The bucket arrays that threads scan (V consecutive entries each) have a pad
// word after every 32: without it the V-strided accesses of a warp share one
// or two banks (13 us of a 16384-bucket call went there).
__host__ __device__ constexpr uint32_t pz(uint32_t b) { return b + (b >> 5); }

// Global counts [B] into their inclusive scan in shared memory: 16-byte loads,
// all of a thread's in flight together, and one scan in registers.
// (One CTA, g null: its own counts own[B].)
template <int V>
__device__ __forceinline__ void scan_counts(const uint32_t* g, const uint32_t* own, uint32_t* I, uint32_t* red) {
  uint32_t v[V];
  if (!g) {
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = own[threadIdx.x * V + i];
  } else if constexpr (V >= 4) {
#pragma unroll
    for (int i = 0; i < V; i += 4) {
      const uint4 q = __ldcg(reinterpret_cast<const uint4*>(g + threadIdx.x * V + i));
      v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = __ldcg(g + threadIdx.x * V + i);
  }
  block_scan_regs<V>(v, red);
#pragma unroll
  for (int i = 0; i < V; ++i) I[pz(threadIdx.x * V + i)] = v[i];
  __syncthreads();
}

// Keys one CTA sorts at a time (32 KB).
template <typename K>
__host__ __device__ constexpr uint32_t direct_cap() { return 32768u / (uint32_t)sizeof(K); }

template <typename K>
struct SortSmem {
  K a[direct_cap<K>()], b[direct_cap<K>()];
  uint32_t hist[DR_NT / 32][256];   // per warp: digit counts, then their prefixes over the warps
  uint32_t mask[DR_NT / 32][256];   // per warp: lanes of the current round holding the digit
  uint32_t part[4][256];            // digit counts of each quarter of the warps
  uint32_t base[256];               // first position of the digit
  uint32_t red[8];
};
template <typename K>
struct DirectSmem {
  union {
    struct {
      uint32_t tab[DIRECT_CELLS];
      uint32_t hist[DIRECT_MAX_B];  // this CTA's counts, then its write cursors
      uint32_t I[pz(DIRECT_MAX_B)];  // sample cells, then the inclusive global counts (padded)
    };
    SortSmem<K> sort;               // once the keys are copied
  };
  uint32_t J[pz(DIRECT_MAX_B)];     // inclusive counts of the children alone (padded)
  uint32_t act[DIRECT_MAX_B / 32];  // buckets holding a k
  uint32_t big[DIRECT_MAX_B / 32];  // ... and more than direct_cap keys
  uint32_t pt[DIRECT_MAX_B / 32];   // ... and one key only (before the ks are located: one key only)
  uint32_t bpre[DIRECT_MAX_B / 32]; // large children before each word
};
template <typename K>
constexpr size_t direct_smem() {
  return sizeof(DirectSmem<K>) > SMALL_SELECT_SMEM ? sizeof(DirectSmem<K>) : SMALL_SELECT_SMEM;
}

// J = inclusive counts of the active buckets alone, from the inclusive counts
// I of all of them; marks the children of more than cap keys in `big`.
template <int V>
__device__ __forceinline__ void child_counts(const uint32_t* I, const uint32_t* act, uint32_t* J, uint32_t* big,
                                             uint32_t cap, uint32_t* red) {
  uint32_t v[V];
  const uint32_t b0 = threadIdx.x * V;
  uint32_t before = b0 ? I[pz(b0 - 1)] : 0u;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const uint32_t b = b0 + i, inc = I[pz(b)];
    v[i] = (act[b >> 5] >> (b & 31)) & 1u ? inc - before : 0u;
    if (v[i] > cap) atomicOr(&big[b >> 5], 1u << (b & 31));
    before = inc;
  }
  block_scan_regs<V>(v, red);
#pragma unroll
  for (int i = 0; i < V; ++i) J[pz(b0 + i)] = v[i];
  __syncthreads();
}

// Sorts m <= direct_cap keys of shared memory (A; Bf: the other buffer) by
// their bits [sh0, sh1); returns the buffer that holds the result.  LSD radix
// sort with 8-bit digits.  Every warp ranks its keys stably, 32 at a time: each
// lane ORs its bit into the warp's mask of its digit and counts the lanes below
// it (the sample sort's scheme).  Latency-bound for few keys (about 0.4 us a
// pass), issue-bound for many; a bitonic sort of 8192 keys takes 91 stages of
// 0.45 us.  All threads call it, after a barrier; it ends with one.
template <typename K>
__device__ K* cta_radix(SortSmem<K>& sm, K* A, K* Bf, uint32_t m, int sh0, int sh1) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = lanemask_lt();
  const uint32_t rounds = (m + DR_NT - 1) / DR_NT;  // of 32 keys per warp
  const uint32_t w0 = warp * 32u * rounds;          // this warp's keys: [w0, w0 + 32 rounds)
  constexpr int RMAX = (int)(direct_cap<K>() / DR_NT);
  for (uint32_t d = lane; d < 256u; d += 32u) sm.mask[warp][d] = 0u;
  for (int sh = sh0; sh < sh1; sh += 8) {
    for (uint32_t d = lane; d < 256u; d += 32u) sm.hist[warp][d] = 0u;
    __syncwarp();
    K key[RMAX];
    uint32_t pos[RMAX];  // digit << 16 | rank among the warp's keys of the digit
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
      if ((uint32_t)r >= rounds) break;
      const uint32_t i = w0 + r * 32u + lane;
      const bool have = i < m;
      key[r] = have ? A[i] : (K)0;
      const uint32_t d = (uint32_t)(key[r] >> sh) & 255u;
      if (have) atomicOr(&sm.mask[warp][d], 1u << lane);
      __syncwarp();
      const uint32_t peers = have ? sm.mask[warp][d] : 0u;
      const uint32_t base = sm.hist[warp][d];
      __syncwarp();
      if (have && (peers & lt) == 0u) {  // the lowest lane of the group
        sm.hist[warp][d] = base + __popc(peers);
        sm.mask[warp][d] = 0u;
      }
      __syncwarp();
      pos[r] = d << 16 | (base + __popc(peers & lt));
    }
    __syncthreads();
    {  // per digit: exclusive prefix over the warps (thread: one digit, a quarter of the warps)
      const uint32_t d = tid & 255u, q = tid >> 8;
      uint32_t c[8], sum = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) { c[j] = sm.hist[q * 8 + j][d]; sum += c[j]; }
      sm.part[q][d] = sum;
      __syncthreads();
      uint32_t run = 0, tot = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t x = sm.part[j][d];
        run += (uint32_t)j < q ? x : 0u;
        tot += x;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) { sm.hist[q * 8 + j][d] = run; run += c[j]; }
      if (q == 0u) {  // the digits' exclusive prefix: 8 warps
        const uint32_t inc = warp_incl_scan_u32(tot, lane);
        if (lane == 31) sm.red[warp] = inc;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        uint32_t before = inc - tot;
        for (uint32_t w = 0; w < warp; ++w) before += sm.red[w];
        sm.base[d] = before;
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RMAX; ++r) {
      if ((uint32_t)r >= rounds) break;
      const uint32_t d = pos[r] >> 16;
      if (w0 + r * 32u + lane < m) Bf[sm.base[d] + sm.hist[warp][d] + (pos[r] & 0xFFFFu)] = key[r];
    }
    __syncthreads();
    K* t = A; A = Bf; Bf = t;
  }
  return A;
}

// f(key) for every key of CTA cta's share of the input, called by all threads
// of the CTA.  The 16-byte vectors of the body are split into equal contiguous
// ranges; CTA 0 also takes the unaligned head and the tail.
template <typename T, int U, typename F>
__device__ __forceinline__ void direct_stream(const T* in, uint64_t n, uint32_t cta, uint32_t ncta, F&& f) {
  constexpr int EPV = Vec16<T>::N;
  const uint32_t tid = threadIdx.x;
  uint64_t head = ((16u - (uint32_t)((uintptr_t)in & 15u)) & 15u) / sizeof(T);
  if (head > n) head = n;
  const uint64_t nvec = (n - head) / EPV;
  const uint64_t v0 = nvec * cta / ncta, v1 = nvec * (cta + 1) / ncta;
  const uint4* body = reinterpret_cast<const uint4*>(in + head);
  uint4 q[U];  // the vectors at i; the next round's are loaded before these are used
  uint64_t i = v0 + tid;
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (i + u * DR_NT < v1) q[u] = __ldg(body + i + u * DR_NT);
  while (i < v1) {
    const uint64_t j = i + DR_NT * U;
    uint4 nx[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (j + u * DR_NT < v1) nx[u] = __ldg(body + j + u * DR_NT);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i + u * DR_NT >= v1) break;
      T e[EPV];
      unpack16<T>(q[u], e);
#pragma unroll
      for (int t = 0; t < EPV; ++t) f(KeyOf<T>::to(e[t]));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = nx[u];
    i = j;
  }
  if (cta == 0) {
    const uint64_t tail0 = head + nvec * EPV, extra = head + (n - tail0);  // < 2 * EPV keys
    if (tid < extra) f(KeyOf<T>::to(in[tid < head ? tid : tail0 + (tid - head)]));
  }
}

// Sorts m <= direct_cap keys (sm.a) of `bits` bits; returns the buffer that
// holds the result.  Up to 24 bits: three radix passes at most.  More (64-bit
// keys above all): three passes order them by their top 24 bits; the few keys
// that share those are put in order by the thread at their run's start.  A
// longer run that is not in order already (equal keys are) sends all bits
// through radix passes: exact for any keys, three passes instead of four to
// eight for most.
template <typename K>
__device__ K* cta_sort(SortSmem<K>& sm, uint32_t m, int bits) {
  constexpr uint32_t RUN = 24;
  const int top = max(bits - 24, 0);
  K* s = cta_radix<K>(sm, sm.a, sm.b, m, top, bits);
  if (top == 0) return s;
  for (uint32_t i = threadIdx.x; i < m; i += DR_NT) {
    const K t = (K)(s[i] >> top);
    if ((i && (K)(s[i - 1] >> top) == t) || i + 1 >= m || (K)(s[i + 1] >> top) != t) continue;
    uint32_t e = i + 2;
    while (e < m && e - i < RUN && (K)(s[e] >> top) == t) ++e;
    if (e < m && (K)(s[e] >> top) == t) continue;  // a longer run
    for (uint32_t j = i + 1; j < e; ++j) {  // insertion sort of [i, e)
      const K x = s[j];
      uint32_t p = j;
      for (; p > i && s[p - 1] > x; --p) s[p] = s[p - 1];
      s[p] = x;
    }
  }
  __syncthreads();
  bool redo = false;  // only a longer run can still be out of order
  for (uint32_t i = threadIdx.x; i + 1 < m; i += DR_NT) redo = redo || s[i] > s[i + 1];
  if (__syncthreads_or(redo)) s = cta_radix<K>(sm, s, s == sm.a ? sm.b : sm.a, m, 0, bits);
  return s;
}

// Extremes of a value over the block; scratch: 2 x 32 keys.  Ends with a barrier.
template <typename K>
__device__ __forceinline__ void block_extremes(K& mn, K& mx, K (*red)[DR_NT / 32]) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  mn = warp_min(mn);
  mx = warp_max(mx);
  if (lane == 0) {
    red[0][warp] = mn;
    red[1][warp] = mx;
  }
  __syncthreads();
  mn = warp_min(red[0][lane]);
  mx = warp_max(red[1][lane]);
  __syncthreads();
}

// Sorts m keys read by get(i) (m <= direct_cap) and hands the i-th smallest to
// put(i, key).  All threads call it.
template <typename K, typename Get, typename Put>
__device__ __forceinline__ void sort_keys(SortSmem<K>& sm, uint32_t m, K (*red)[DR_NT / 32], Get&& get, Put&& put) {
  constexpr int RMAX = (int)(direct_cap<K>() / DR_NT);
  K k[RMAX], mn = key_max<K>(), mx = 0;
#pragma unroll
  for (int r = 0; r < RMAX; ++r) {
    const uint32_t i = threadIdx.x + r * DR_NT;
    if (i < m) k[r] = get(i);
  }
#pragma unroll
  for (int r = 0; r < RMAX; ++r)
    if (threadIdx.x + r * DR_NT < m) {
      mn = min(mn, k[r]);
      mx = max(mx, k[r]);
    }
  block_extremes(mn, mx, red);
#pragma unroll
  for (int r = 0; r < RMAX; ++r) {
    const uint32_t i = threadIdx.x + r * DR_NT;
    if (i < m) sm.a[i] = (K)(k[r] - mn);
  }
  __syncthreads();
  const K* s = cta_sort<K>(sm, m, bitlen((K)(mx - mn)));
  for (uint32_t i = threadIdx.x; i < m; i += DR_NT) put(i, (K)(mn + s[i]));
  __syncthreads();
}

// A vector of at most direct_cap keys: one CTA sorts it and every k reads its
// rank.
template <typename T>
__global__ __launch_bounds__(DR_NT, 1) void direct_sort(const __grid_constant__ DirectArgs<T> a) {
  using K = typename KeyOf<T>::K;
  extern __shared__ __align__(128) uint8_t smem[];
  SortSmem<K>& sm = *reinterpret_cast<SortSmem<K>*>(smem);
  __shared__ K red_k[2][DR_NT / 32];
  const uint32_t tid = threadIdx.x, n = (uint32_t)a.n;
  K* sorted = reinterpret_cast<K*>(smem + sizeof(SortSmem<K>));
  uint32_t bad = 0;
  sort_keys<K>(sm, n, red_k, [&](uint32_t i) { return KeyOf<T>::to(a.in[i]); },
               [&](uint32_t i, K key) { sorted[i] = key; });
  for (uint32_t i = tid; i < a.r.nk; i += DR_NT) {
    const uint32_t k = a.ks ? a.ks[i] : i + 1u;
    const bool ok = k >= 1u && k <= n;
    if (!ok) bad = 1u;
    a.r.out[i] = KeyOf<T>::from(ok ? sorted[n - k] : (K)0);
  }
  const bool any = __syncthreads_or(bad) != 0;
  if (tid < sizeof(Counters) / 4) {
    const uint32_t x = any && tid == offsetof(Counters, status) / 4 ? (uint32_t)GGMS_E_INVALID_ARG : 0u;
    reinterpret_cast<uint32_t*>(a.r.C)[tid] = x;
    if (a.r.report) reinterpret_cast<uint32_t*>(a.r.report)[tid] = x;
  }
}

// One vector for direct_body: its share of the grid, its workspace, its ks.
template <typename T>
struct DirectTask {
  using K = typename KeyOf<T>::K;
  const T* in;
  uint64_t n;
  const uint32_t* ks;          // null: top-k
  uint32_t nk;
  uint64_t seed;
  uint32_t B, focus, slices;
  uint32_t *ghist, *gcur, *gact, *gpt;  // [B], [B], [B / 32 + 2], [B / 32 + B]; one CTA: unused
  uint32_t* bar;               // the barrier word of the vector's CTAs
  uint32_t cta, ncta;          // this CTA among them
  uint64_t off;                // the vector's n candidates: r.cand[0] + off
  uint64_t k0;                 // its ks in the per-k arrays: k0 ..
};

// Steps 1 to 5 for one vector.  On return its ks are resolved but for those in
// large children, which are in pool 1 for the refinement levels, with their
// true key ranges.  False after a barrier that ran out.  ONE: a single CTA's
// vector (a.cta == 0, a.ncta == 1).  U: vectors in flight per thread, twice.
template <typename T, bool ONE, int U>
__device__ __forceinline__ bool direct_body(const DirectTask<T>& a, const RefineArgs<T>& r, uint8_t* smem) {
  using K = typename KeyOf<T>::K;
  constexpr bool FP = std::is_floating_point<T>::value, K64 = sizeof(K) == 8;
  constexpr uint32_t NONE = 0xFFFFFFFFu;
  DirectSmem<K>& sm = *reinterpret_cast<DirectSmem<K>*>(smem);
  __shared__ K red_k[4][DR_NT / 32];
  __shared__ uint32_t red[72];
  const uint32_t cta = ONE ? 0u : a.cta, ncta = ONE ? 1u : a.ncta;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t gt = cta * DR_NT + tid, gs = ncta * DR_NT;
  const uint32_t B = a.B, nk = a.nk;
  // the per-k arrays and the candidates, addressed where they are used: held
  // from here on they would take ten registers through both streams
  auto kbin = [&](uint32_t i) -> uint32_t& { return r.kbin[a.k0 + i]; };
  auto krank = [&](uint32_t i) -> uint32_t& { return r.krank[a.k0 + i]; };
  auto kseg = [&](uint32_t i) -> uint32_t& { return r.kseg[a.k0 + i]; };
  auto kkey = [&](uint32_t i) -> K& { return r.kkey[a.k0 + i]; };

  GGMS_TRACE(0);
  // ---- the global histogram
  if (ncta > 1u)
    for (uint32_t i = gt; i < B; i += gs) {
      a.ghist[i] = 0u;
      a.gcur[i] = 0u;
      if (i <= B / 32) a.gact[i] = 0u;
    }
  // the ranks, staged in device memory (ks may be pinned host memory: each is read once)
  for (uint32_t i = gt; i < nk; i += gs) {
    const uint32_t k = a.ks ? a.ks[i] : i + 1u;
    kbin(i) = k >= 1u && (uint64_t)k <= a.n ? (uint32_t)(a.n - k) : NONE;  // a rank is at most n - 1 < NONE
  }
  GridBarrier zeroed;
  zeroed.arrive(a.bar, ncta, cta == 0u);

  // ---- the map, from a sample every CTA draws for itself
  const uint32_t S = (uint32_t)min(a.n, (uint64_t)DIRECT_SAMPLE);
  auto sampled = [&](uint32_t i) __attribute__((always_inline)) -> K {
    uint64_t pos = i;
    if (a.n > DIRECT_SAMPLE) {  // one key per stratum, at a hashed offset
      const uint64_t p0 = a.n * i / DIRECT_SAMPLE, p1 = a.n * (i + 1) / DIRECT_SAMPLE;
      pos = p0 + (((mix64(a.seed ^ i) >> 32) * (p1 - p0)) >> 32);
    }
    return KeyOf<T>::to(__ldg(a.in + pos));
  };
  K sv[DIRECT_SAMPLE / DR_NT];
  K lo = key_max<K>(), hi = 0, hn = 0, lp = key_max<K>();
  constexpr K MID = (K)((K)1 << (sizeof(K) * 8 - 1));  // floating types: the keys below are negative
#pragma unroll
  for (int j = 0; j < (int)(DIRECT_SAMPLE / DR_NT); ++j) {
    const uint32_t i = tid + j * DR_NT;
    if (i < S) sv[j] = sampled(i);
  }
#pragma unroll
  for (int j = 0; j < (int)(DIRECT_SAMPLE / DR_NT); ++j)
    if (tid + j * DR_NT < S) {
      lo = min(lo, sv[j]);
      hi = max(hi, sv[j]);
      if (FP && sv[j] < MID) hn = max(hn, sv[j]);
      if (FP && sv[j] >= MID) lp = min(lp, sv[j]);
    }
  for (uint32_t i = tid; i < DIRECT_CELLS; i += DR_NT) sm.I[i] = 0u;
  for (uint32_t i = tid; i < B; i += DR_NT) sm.hist[i] = 0u;
  for (uint32_t w = tid; w < B / 32; w += DR_NT) sm.pt[w] = 0u;
  lo = warp_min(lo);
  hi = warp_max(hi);
  if (FP) {
    hn = warp_max(hn);
    lp = warp_min(lp);
  }
  if (lane == 0) {
    red_k[0][warp] = lo;
    red_k[1][warp] = hi;
    red_k[2][warp] = hn;
    red_k[3][warp] = lp;
  }
  __syncthreads();
  lo = warp_min(red_k[0][lane]);
  hi = warp_max(red_k[1][lane]);
  // (every lane takes part in every reduction: as arms of the selects below
  // they gave the wrong arm in one kernel)
  const K hn_all = warp_max(red_k[2][lane]), lp_all = warp_min(red_k[3][lane]);
  const bool two = FP && lo < MID && hi >= MID;
  hn = two ? hn_all : hi;
  lp = two ? lp_all : hi;
  // 64-bit keys: the high word alone when it resolves the sample
  const bool hi32 = K64 && (K)((hi - lo) - (two ? lp - hn : (K)0)) >> (K64 ? 32 : 0) >= (K)(1u << 16);
  auto dom = [&](K k) -> K { return hi32 ? (K)(k >> (K64 ? 32 : 0)) : k; };
  const K dmax = hi32 ? (K)0xFFFFFFFFu : key_max<K>();
  DirectMap<K, FP, false> map;  // in the domain of dom(): used to place the sample
  map.hn = dom(hn);
  map.lp = dom(lp);
  map.lo = dom(lo);
  map.hi = dom(hi);
  // cells over the sample's range, and up to DIRECT_EXT more at either end for
  // the keys beyond it: about n / S keys of a long vector lie beyond each
  // extreme of its sample, and a k near 1 or n is among them
  const K range = (K)((map.hn - map.lo) + (map.hi - map.lp));
  map.csh = (uint32_t)max(0, bitlen(range) - 11);
  static_assert(DIRECT_CELLS == 1u << 11, "cells of 11 bits");
  if ((range >> map.csh) >= (K)(DIRECT_CELLS - 2 * DIRECT_EXT - (two ? 2 * DIRECT_GAP : 0u))) ++map.csh;
  const K ext = a.n > S ? (K)((K)DIRECT_EXT << map.csh) : (K)0;
  map.lo = (K)(map.lo - min(map.lo, ext));
  map.hi = (K)(map.hi + min((K)(dmax - map.hi), ext));
  // ... and likewise for the gap: two sampled keys' worth of values lie in it,
  // which as one bucket would be a large child (90 us of levels at 2^24 fp32)
  if (two) {
    const K half = (K)((map.lp - map.hn) >> 1), g = min((K)((K)DIRECT_GAP << map.csh), half ? (K)(half - 1u) : (K)0);
    map.hn = (K)(map.hn + (a.n > S ? g : (K)0));
    map.lp = (K)(map.lp - (a.n > S ? g : (K)0));
  } else {
    map.hn = map.lp = map.hi;
  }
  map.tab = sm.tab;
  auto cell = [&](K k) { return (uint32_t)((K)((min(max(k, map.lo), map.hn) - map.lo) +
                                               (min(max(k, map.lp), map.hi) - map.lp)) >> map.csh); };
  const uint32_t c_end = cell(map.hi);
#pragma unroll
  for (int j = 0; j < (int)(DIRECT_SAMPLE / DR_NT); ++j)
    if (tid + j * DR_NT < S) atomicAdd(&sm.I[cell(dom(sv[j]))], 1u);
  __syncthreads();
  static_assert(DIRECT_CELLS == 2 * DR_NT, "two cells per thread");
  uint32_t w2[2], raw[2];  // this thread's cells: weights, sampled keys
  {
    uint32_t near[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const uint32_t c = 2 * tid + i - 2u;  // (wraps below 0)
      near[i] = c < DIRECT_CELLS ? sm.I[c] : 0u;
    }
    raw[0] = near[2];
    raw[1] = near[3];
    const uint32_t mid = near[1] + near[2] + near[3] + near[4];
    w2[0] = DIRECT_WT * (raw[0] + max(raw[0], (mid + near[0]) / 5u)) + DIRECT_CELL_WT;
    w2[1] = DIRECT_WT * (raw[1] + max(raw[1], (mid + near[5]) / 5u)) + DIRECT_CELL_WT;
    if (2 * tid > c_end) w2[0] = 0u;
    if (2 * tid + 1 > c_end) w2[1] = 0u;
  }
  const uint32_t own0 = w2[0], own1 = w2[1];
  block_scan_regs<2>(w2, red);
  uint32_t hot = 0;  // the weight of the cells that can hold a k (0: no focus)
  uint32_t nfirst = w2[0] - own0;  // packed prefix before this thread's cells: hot | other << 16
  bool focus = false;
  if (a.focus) {
    if (!zeroed.wait(a.bar, ncta, r.C, r.limit)) return false;
    // clustered ks: their ranks occupy at most a quarter of 64 equal ranges
    unsigned long long occ = 0;
    for (uint32_t i = tid; i < nk; i += DR_NT) {
      const uint32_t rank = __ldcg(&kbin(i));
      if (rank != NONE) occ |= 1ull << (uint32_t)(((uint64_t)rank * 64u) / a.n);
    }
    const uint32_t o0 = __reduce_or_sync(FULL, (uint32_t)occ), o1 = __reduce_or_sync(FULL, (uint32_t)(occ >> 32));
    block_scan_regs<2>(raw, red);  // I: inclusive counts of the sampled keys
    sm.I[2 * tid] = raw[0];
    sm.I[2 * tid + 1] = raw[1];
    if (lane == 0) {
      red[warp] = o0;
      red[32 + warp] = o1;
    }
    __syncthreads();
    focus = __popc(__reduce_or_sync(FULL, red[lane])) + __popc(__reduce_or_sync(FULL, red[32 + lane])) <= 16;
    __syncthreads();
  }
  if (focus) {
    // The sample position of the key of rank q n is binomial: it lies within
    // m = z sqrt(S q (1 - q)) + z + 2 of S q (z = 6).  Cells of those positions,
    // as a difference array; a k outside them costs time, never exactness.
    for (uint32_t i = tid; i < nk; i += DR_NT) {
      const uint32_t rank = __ldcg(&kbin(i));
      if (rank == NONE) continue;
      const float q = ((float)rank + 0.5f) / (float)a.n;
      const float pos = q * (float)S, m = 6.0f * sqrtf((float)S * q * fmaxf(1.0f - q, 0.0f)) + 8.0f;
      const uint32_t p0 = min((uint32_t)fmaxf(pos - m, 0.0f), S - 1u), p1 = (uint32_t)(pos + m) + 1u;
      auto cell_of = [&](uint32_t p) {  // the cell of the p-th sampled key
        uint32_t l = 0, h = c_end;
        while (l < h) {
          const uint32_t mid = (l + h) >> 1;
          if (sm.I[mid] > p) h = mid; else l = mid + 1u;
        }
        return l;
      };
      const uint32_t c0 = p0 ? cell_of(p0) : 0u;
      const uint32_t c1 = p1 < S ? cell_of(p1) : c_end;
      atomicAdd(&sm.hist[c0], 1u);
      if (c1 + 1u < DIRECT_CELLS) atomicAdd(&sm.hist[c1 + 1u], NONE);
    }
    __syncthreads();
    uint32_t d2[2] = {sm.hist[2 * tid], sm.hist[2 * tid + 1]};
    block_scan_regs<2>(d2, red);
    sm.hist[2 * tid] = 0u;
    sm.hist[2 * tid + 1] = 0u;
    // the weight of hot cells in the low half, of the others in the high half
    static_assert(3 * DIRECT_WT * DIRECT_SAMPLE + DIRECT_CELL_WT * DIRECT_CELLS < 65536u, "weights of 16 bits");
    w2[0] = own0 << (d2[0] ? 0 : 16);
    w2[1] = own1 << (d2[1] ? 0 : 16);
    nfirst = w2[0];
    block_scan_regs<2>(w2, red);
    nfirst = w2[0] - nfirst;
  }
  if (tid == DR_NT - 1) {
    red[70] = w2[1];
    red[71] = 0u;
    red[68] = 0u;
  }
  __syncthreads();
  const uint32_t W = (red[70] & 0xFFFFu) + (red[70] >> 16);
  if (focus) hot = red[70] & 0xFFFFu;
  // first bucket of a cell with (packed) weight prefix p: 7/8 of the buckets
  // over the hot cells and 1/8 over the others, or all evenly
  const bool focused = hot && hot < W - W / 8u;
  auto first_bucket = [&](uint32_t p) -> uint32_t {  // (weights < 2^16, B <= 2^15: no overflow)
    const uint32_t ph = p & 0xFFFFu, pc = p >> 16;
    if (!focused) return (ph + pc) * B / W;
    const uint32_t Bh = B - B / 8u;
    return ph * Bh / hot + pc * (B - Bh) / (W - hot);
  };
  {
    const uint32_t b0 = first_bucket(nfirst), b1 = first_bucket(w2[0]), b2 = first_bucket(w2[1]);
    sm.tab[2 * tid] = min(b0, B - 1u) | (b1 - b0) << 16;  // b0 == B only past the last weight
    sm.tab[2 * tid + 1] = min(b1, B - 1u) | (b2 - b1) << 16;
    // some cell has a bucket or more per key
    if (!hi32 && map.csh < 16u && max(b1 - b0, b2 - b1) >> (map.csh & 31u) != 0u) red[71] = 1u;
  }
  __syncthreads();
  // use(m): m is the map in its cheapest form for this sample (the same for every CTA)
  auto with_map = [&](auto&& use) {
    auto as = [&](auto m) {
      using D = decltype(m.lo);
      m.lo = (D)map.lo; m.hi = (D)map.hi; m.hn = (D)map.hn; m.lp = (D)map.lp;
      m.csh = map.csh;
      m.tab = sm.tab;
      use(m);
    };
    if constexpr (K64) {
      if (!hi32) { as(DirectMap<K, FP, false>{}); return; }
      if (FP && two) as(DirectMap<K, true, true>{}); else as(DirectMap<K, false, true>{});
    } else {
      if (FP && two) as(DirectMap<K, true, false>{}); else as(DirectMap<K, false, false>{});
    }
  };

  GGMS_TRACE(1);
  // ---- count
  with_map([&](const auto& m) {
    direct_stream<T, U>(a.in, a.n, cta, ncta, [&](K key) { atomicAdd(&sm.hist[m(key)], 1u); });
  });
  GGMS_TRACE(2);
  if (a.focus) __syncthreads();
  else if (!zeroed.wait(a.bar, ncta, r.C, r.limit)) return false;  // (a CTA barrier too)
  // Buckets of one key, decided by the first CTA for all: the map is monotone, so
  // a bucket that a key's neighbours on both sides miss is that key's alone.
  // (Here and not before the count: there it cost every call 0.5 us.)
  if (cta == 0u) {
    if (red[71]) {
      with_map([&](const auto& m) {
#pragma unroll 1
        for (uint32_t i = tid; i < min(a.n, (uint64_t)DIRECT_SAMPLE); i += DR_NT) {
          const K x = sampled(i);
          const uint32_t b = m(x);
          if ((x != 0 && m((K)(x - 1u)) == b) || (x != key_max<K>() && m((K)(x + 1u)) == b)) continue;
          atomicOr(&sm.pt[b >> 5], 1u << (b & 31));
          if (ONE) sm.J[pz(b)] = i; else a.gpt[B / 32 + b] = i;  // (any of the key's)
        }
      });
      __syncthreads();
      if (ncta > 1u)
        for (uint32_t w = tid; w < B / 32; w += DR_NT) a.gpt[w] = sm.pt[w];
    }
    if (tid == 0 && ncta > 1u) a.gact[B / 32 + 1] = red[71];
  }
  if (ncta > 1u)
    for (uint32_t i = tid; i < B; i += DR_NT) {
      const uint32_t v = sm.hist[i];
      if (v) atomicAdd(&a.ghist[i], v);
    }
  if (!grid_barrier(a.bar, ncta, cta == 0u, r.C, r.limit)) return false;

  GGMS_TRACE(3);
  // ---- scan, locate
  const uint32_t points = ncta > 1u && tid == 0 ? __ldcg(&a.gact[B / 32 + 1]) : 0u;  // (one thread: all of them meet at one word)
  for (uint32_t w = tid; w < B / 32; w += DR_NT) {
    sm.act[w] = 0u;
    sm.big[w] = 0u;
  }
  const uint32_t* counts = ncta > 1u ? a.ghist : nullptr;
  switch (B / DR_NT) {
    case 1: scan_counts<1>(counts, sm.hist, sm.I, red); break;
    case 2: scan_counts<2>(counts, sm.hist, sm.I, red); break;
    case 4: scan_counts<4>(counts, sm.hist, sm.I, red); break;
    case 8: scan_counts<8>(counts, sm.hist, sm.I, red); break;
    default: scan_counts<16>(counts, sm.hist, sm.I, red); break;
  }
  static_assert(DIRECT_MAX_B == 16 * DR_NT, "the largest scan above");
  if (ncta > 1u && tid == 0) red[71] = points;  // read behind the ks
  auto bucket_of = [&](uint32_t rank) {  // the smallest b with I[b] > rank
    uint32_t l = 0, h = B - 1u;
    while (l < h) {
      const uint32_t mid = (l + h) >> 1;
      if (sm.I[pz(mid)] > rank) h = mid; else l = mid + 1u;
    }
    return l;
  };
  if (!a.slices) {  // every CTA locates every k
    for (uint32_t i = tid; i < nk; i += DR_NT) {
      const uint32_t rank = __ldcg(&kbin(i));
      if (rank == NONE) continue;
      const uint32_t b = bucket_of(rank);
      atomicOr(&sm.act[b >> 5], 1u << (b & 31));
    }
  } else {  // many ks: every CTA locates its own, and they meet
    for (uint32_t i = gt; i < nk; i += gs) {
      const uint32_t rank = kbin(i);
      if (rank == NONE) continue;
      const uint32_t b = bucket_of(rank);
      atomicOr(&a.gact[b >> 5], 1u << (b & 31));
    }
    if (!grid_barrier(a.bar, ncta, cta == 0u, r.C, r.limit)) return false;
    for (uint32_t w = tid; w < B / 32; w += DR_NT) sm.act[w] = __ldcg(&a.gact[w]);
  }
  __syncthreads();
  // a bucket of one key is no child; its place in hist holds a sampled position of the key
  if (__builtin_expect(red[71] != 0u, 0)) {
    for (uint32_t w = tid; w < B / 32; w += DR_NT) {
      const uint32_t one = sm.act[w] & (ncta > 1u ? __ldcg(&a.gpt[w]) : sm.pt[w]);
      sm.pt[w] = one;
      sm.act[w] &= ~one;
      for (uint32_t m = one; m; m &= m - 1u) {
        const uint32_t b = w * 32u + __ffs(m) - 1u;
        sm.hist[b] = ONE ? sm.J[pz(b)] : __ldcg(&a.gpt[B / 32 + b]);
      }
    }
    __syncthreads();
  }
  constexpr uint32_t CAP = direct_cap<K>();
  switch (B / DR_NT) {
    case 1: child_counts<1>(sm.I, sm.act, sm.J, sm.big, CAP, red); break;
    case 2: child_counts<2>(sm.I, sm.act, sm.J, sm.big, CAP, red); break;
    case 4: child_counts<4>(sm.I, sm.act, sm.J, sm.big, CAP, red); break;
    case 8: child_counts<8>(sm.I, sm.act, sm.J, sm.big, CAP, red); break;
    default: child_counts<16>(sm.I, sm.act, sm.J, sm.big, CAP, red); break;
  }
  if (warp == 0) {  // large children before each word (B / 32 <= 512 words)
    uint32_t run = 0;
    for (uint32_t w0 = 0; w0 < B / 32; w0 += 32) {
      const uint32_t c = __popc(sm.big[w0 + lane]);
      const uint32_t inc = warp_incl_scan_u32(c, lane);
      sm.bpre[w0 + lane] = run + inc - c;
      run += __shfl_sync(FULL, inc, 31);
    }
    if (lane == 0) red[70] = run;
  }
  __syncthreads();
  const uint32_t nbig = red[70], total = sm.J[pz(B - 1u)];
  auto active = [&](uint32_t b) { return (sm.act[b >> 5] >> (b & 31)) & 1u; };
  auto is_big = [&](uint32_t b) { return (sm.big[b >> 5] >> (b & 31)) & 1u; };
  auto big_of = [&](uint32_t b) { return sm.bpre[b >> 5] + __popc(sm.big[b >> 5] & ((1u << (b & 31)) - 1u)); };
  GGMS_TRACE(4);
  // Where the cursors will end, as a weighted sum: when the caller
  // changes the vector between the count and the copy they end elsewhere, and
  // the call fails.  The stores stay in the workspace: a vector's n keys lie
  // below 2 n of its place in cand[0], which cand[1] follows.  (A bound tested
  // for every copied key cost the batched path 2 to 3 %.)
  uint32_t ends = 0;
  for (uint32_t b0 = tid; b0 < B; b0 += 8u * DR_NT) {
    // this CTA's range of every child it holds keys of: one reservation each,
    // eight in flight per thread
    uint32_t base[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t b = b0 + u * DR_NT;
      base[u] = 0u;
      if (b < B && active(b) && ncta > 1u && sm.hist[b]) base[u] = atomicAdd(&a.gcur[b], sm.hist[b]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t b = b0 + u * DR_NT;
      if (b >= B || !active(b)) continue;
      const uint32_t at = (b ? sm.J[pz(b - 1)] : 0u) + base[u];
      ends += (at + sm.hist[b]) * (2u * b + 1u);
      sm.hist[b] = at;
    }
  }
  ends = __reduce_add_sync(FULL, ends);
  if (lane == 0) atomicAdd(&red[68], ends);
  // ids of the large children: a range of the list of all vectors'
  if (cta == 0 && tid == 0 && nbig) {
    atomicAdd(&r.C->nsegs[1], nbig);
    const uint32_t first = atomicAdd(&r.C->nbig[1], nbig);
    if (ncta > 1u) a.gact[B / 32] = first;
    red[69] = first;
  }
  __syncthreads();

  GGMS_TRACE(5);
  // ---- copy
  if (total) with_map([&](const auto& m) {
    K* cand = r.cand[0] + a.off;
    direct_stream<T, U>(a.in, a.n, cta, ncta, [&](K key) {
      const uint32_t b = m(key);
      if (active(b)) cand[atomicAdd(&sm.hist[b], 1u)] = key;
    });
  });
  GGMS_TRACE(6);
  GridBarrier copied;
  copied.arrive(a.bar, ncta, cta == 0u);
  ends = 0;
  for (uint32_t b = 4u * tid; b < B; b += 4u * DR_NT) {
    const uint32_t some = (sm.act[b >> 5] >> (b & 31)) & 15u;
    if (!some) continue;
    const uint4 h = *reinterpret_cast<const uint4*>(&sm.hist[b]);
    ends += (some & 1u ? h.x * (2u * b + 1u) : 0u) + (some & 2u ? h.y * (2u * b + 3u) : 0u) +
            (some & 4u ? h.z * (2u * b + 5u) : 0u) + (some & 8u ? h.w * (2u * b + 7u) : 0u);
  }
  ends = __reduce_add_sync(FULL, ends);
  if (lane == 0) atomicSub(&red[68], ends);
  if (!copied.wait(a.bar, ncta, r.C, r.limit)) return false;
  if (tid == 0 && red[68]) set_status(r.C, GGMS_E_INTERNAL);
  GGMS_TRACE(7);
  GGMS_TRACE_CTA(0);

  // ---- this CTA's slice of the ks and of the large children
  const uint32_t first_big = !nbig ? 0u : ncta > 1u ? __ldcg(&a.gact[B / 32]) : red[69];
  for (uint32_t i = gt; i < nk; i += gs) {
    const uint32_t rank = __ldcg(&kbin(i));
    if (rank == NONE) {
      set_status(r.C, GGMS_E_INVALID_ARG);
      kseg(i) = K_DONE;
      kkey(i) = 0;
      continue;
    }
    const uint32_t b = bucket_of(rank), in = rank - (b ? sm.I[pz(b - 1)] : 0u);
    if (__builtin_expect((sm.pt[b >> 5] >> (b & 31)) & 1u, 0)) {
      kkey(i) = sampled(sm.hist[b]);
      kseg(i) = K_DONE;
      continue;
    }
    const bool lg = is_big(b);
    krank(i) = lg ? in : (b ? sm.J[pz(b - 1)] : 0u) + in;
    kseg(i) = lg ? first_big + big_of(b) : K_SORTED;
  }
  if (nbig)
    for (uint32_t b = tid; b < B; b += DR_NT) {
      if (!is_big(b)) continue;
      const uint32_t at = big_of(b), id = first_big + at;
      if (at % ncta != cta) continue;
      const uint32_t off = b ? sm.J[pz(b - 1)] : 0u;
      Seg<K> sg;  // refined by levels, from its true key range (below)
      sg.off = a.off + off;
      sg.cnt = sm.J[pz(b)] - off;
      sg.shift = 0u;
      sg.lo = key_max<K>();
      sg.hi = 0;
      sg.row = id;
      sg.pad = 0u;
      const uint32_t nt = (sg.cnt + TILE - 1) / TILE;
      const uint32_t t0 = atomicAdd(&r.C->ntiles[1], nt);
      if (id >= r.caps.rows || id >= r.caps.segs || t0 + nt > r.caps.tiles) {  // cannot happen: the caps bound them
        set_status(r.C, GGMS_E_INTERNAL);
        continue;
      }
      r.bigs[1][id] = id;
      r.segs[1][id] = sg;
      r.cursor[1][id] = 0u;
      for (uint32_t t = 0; t < nt; ++t) r.tiles[1][t0 + t] = TileRef{id, t};
    }

  // ---- sort: whole children whose keys start in this CTA's part of the candidates
  auto boundary = [&](uint32_t x) -> uint32_t {  // the first child boundary at or after position x
    if (x == 0u) return 0u;
    uint32_t l = 0, h = B - 1u;  // J[B - 1] = total >= x
    while (l < h) {
      const uint32_t mid = (l + h) >> 1;
      if (sm.J[pz(mid)] >= x) h = mid; else l = mid + 1u;
    }
    return sm.J[pz(l)];
  };
  auto last_boundary = [&](uint32_t x) -> uint32_t {  // the last child boundary at or before position x
    uint32_t l = 0, h = B;  // the first b with J[b] > x
    while (l < h) {
      const uint32_t mid = (l + h) >> 1;
      if (sm.J[pz(mid)] > x) h = mid; else l = mid + 1u;
    }
    return l ? sm.J[pz(l - 1)] : 0u;
  };
  const uint32_t x_end = boundary((uint32_t)((uint64_t)total * (cta + 1) / ncta));
  for (uint32_t x = boundary((uint32_t)((uint64_t)total * cta / ncta)); x < x_end;) {
    const uint32_t y = min(x_end, last_boundary(x + CAP < x ? total : x + CAP));
    if (y > x) {
      K* c = r.cand[0] + a.off + x;
      sort_keys<K>(sm.sort, y - x, red_k, [&](uint32_t i) { return c[i]; }, [&](uint32_t i, K key) { c[i] = key; });
      x = y;
    } else {  // a large child: the levels refine it
      x = boundary(x + 1u);
    }
  }
  GGMS_TRACE(8);
  GGMS_TRACE_CTA(1);
  if (!grid_barrier(a.bar, ncta, cta == 0u, r.C, r.limit)) return false;
  GGMS_TRACE(9);
  // ks of the sorted children (the barrier makes every child's order visible)
  for (uint32_t i = gt; i < nk; i += gs) {
    if (kseg(i) != K_SORTED) continue;
    kkey(i) = r.cand[0][a.off + krank(i)];
    kseg(i) = K_DONE;
  }
  if (!nbig) return true;
  // the true key range of the large children: their tiles dealt to the CTAs
  uint32_t dealt = 0;
  for (uint32_t w = 0; w < B / 32; ++w)
    for (uint32_t m = sm.big[w]; m; m &= m - 1u) {
      const uint32_t b = w * 32u + __ffs(m) - 1u, id = first_big + big_of(b);
      if (id >= r.caps.rows || id >= r.caps.segs) continue;
      const uint32_t off = b ? sm.J[pz(b - 1)] : 0u, cnt = sm.J[pz(b)] - off;
      const uint32_t nt = (cnt + TILE - 1) / TILE, t0 = (cta + ncta - dealt % ncta) % ncta;
      dealt += nt;
      if (t0 >= nt) continue;
      K mn = key_max<K>(), mx = 0;
      for (uint32_t t = t0; t < nt; t += ncta)
        for (uint32_t i = t * TILE + tid; i < min(cnt, (t + 1u) * TILE); i += DR_NT) {
          const K x = r.cand[0][a.off + off + i];
          mn = min(mn, x);
          mx = max(mx, x);
        }
      mn = warp_min(mn);
      mx = warp_max(mx);
      if (lane == 0 && mn <= mx) {
        key_atomic_min(&r.segs[1][id].lo, mn);
        key_atomic_max(&r.segs[1][id].hi, mx);
      }
    }
  if (!grid_barrier(a.bar, ncta, cta == 0u, r.C, r.limit)) return false;
  for (uint32_t j = first_big + gt; j < min(first_big + nbig, min(r.caps.rows, r.caps.segs)); j += gs) {
    Seg<K>& s = r.segs[1][j];
    s.shift = (uint32_t)max(0, bitlen((K)(__ldcg(&s.hi) - __ldcg(&s.lo))) - RADIX_BITS);
  }
  // a child of one value answers its ks; the levels skip its tiles
  for (uint32_t i = gt; i < nk; i += gs) {
    const uint32_t id = kseg(i);
    if (id >= min(r.caps.rows, r.caps.segs)) continue;  // resolved
    const K lo1 = __ldcg(&r.segs[1][id].lo);
    if (lo1 != __ldcg(&r.segs[1][id].hi)) continue;
    kkey(i) = lo1;
    kseg(i) = K_DONE;
  }
  return true;
}

template <typename T>
__global__ __launch_bounds__(DR_NT, 1) void direct_select(const __grid_constant__ DirectArgs<T> a) {
  extern __shared__ __align__(128) uint8_t smem[];
  const RefineArgs<T>& r = a.r;
  Counters* C = r.C;
  const uint32_t cta = blockIdx.x, ncta = gridDim.x;
  // the call's counters (other CTAs touch them only after the body's first barrier)
  if (cta == 0 && threadIdx.x < sizeof(Counters) / 4) reinterpret_cast<uint32_t*>(C)[threadIdx.x] = 0u;
  DirectTask<T> t;
  t.in = a.in;
  t.n = a.n;
  t.ks = a.ks;
  t.nk = r.nk;
  t.seed = a.seed;
  t.B = a.B;
  t.focus = a.focus;
  t.slices = a.slices;
  t.ghist = a.ghist;
  t.gcur = a.gcur;
  t.gact = a.gact;
  t.gpt = a.gpt;
  t.bar = r.bar;
  t.cta = cta;
  t.ncta = ncta;
  t.off = 0;
  t.k0 = 0;
  bool good = direct_body<T, false, 4>(t, r, smem);
  if (good && __ldcg(&C->nbig[1]))
    good = refine_body<T, DR_NT>(r, smem) && grid_barrier(r.bar, ncta, cta == 0u, C, r.limit);
  if (good) write_out_body<T>(r.kkey, r.kseg, r.nk, r.out, C, cta, ncta);
  leave_body(C, r.bar, r.left, r.report, ncta);
  GGMS_TRACE(10);
}

GGMS_END
