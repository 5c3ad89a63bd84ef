// Merging many sorted runs of one segment, window by window of the merged order.
//
// A segment of n keys is cut into runs of R, each sorted.  Merging by rank (every run
// against every other) takes time with the square of the runs.  Here a CTA takes R
// consecutive places of the merged order instead: it finds where they begin and end in
// every run (run_cuts), puts the pieces in between side by side, in the runs' order, and
// sorts those R keys again.  The time grows with n; only the cuts look at all runs, some
// eighty dependent reads each.  20M instances: in four tiles (2,466 runs) the merge of
// positions takes 15.8 ms where by rank it took 252, in 1,024 tiles (25 runs) 1.6 for
// 2.2; of 64-bit keys in 16 tiles (309 runs) 4.4 for 62.
#pragma once

#include "svr_block.cuh"

namespace svr {

// The first d keys of the merged order, with equal keys in the order of their runs:
// those below v and the first q of those equal to v.
template <typename KT>
struct RunCut {
  KT v;
  uint32_t q;
};

// Shared words of run_cuts, and of the gathering of a window between two cuts (NT
// threads).  How a cut divides the first TRACKED runs is kept from step to step: in
// [lo, hi) of a run lie the keys that the search has not placed yet, in the end those
// equal to v.  Later runs are searched anew in every step.
template <int NT, int TRACKED>
struct WindowSmem {
  uint16_t lo[2][TRACKED], hi[2][TRACKED], mid[2][TRACKED];
  uint32_t off[NT], src[NT];
  uint32_t scan[NT / 32 + 1];
  uint32_t count[3][2];
  unsigned long long least[2], most[2];
};

// A segment's keys as sorted runs of R.
template <typename T, typename KT>
struct SortedRuns {
  const T* keys;
  uint32_t n;
  int R;
  __device__ __forceinline__ uint32_t runs() const { return (n + R - 1) / R; }
  __device__ __forceinline__ int length(uint32_t x) const { return (int)min((uint32_t)R, n - x * R); }
  __device__ __forceinline__ KT at(uint32_t i) const { return (KT)keys[i]; }
  // Keys of run x, out of [lo, hi), that are below v (OR_EQUAL: or equal to it).
  template <bool OR_EQUAL>
  __device__ __forceinline__ int below(uint32_t x, KT v, int lo, int hi) const {
    const T* k = keys + (size_t)x * R;
    while (lo < hi) {
      const int m = (lo + hi) >> 1;
      const KT key = (KT)k[m];
      if (OR_EQUAL ? key <= v : key < v) lo = m + 1;
      else hi = m;
    }
    return lo;
  }
};

// The cuts after the first d[0] and d[1] keys (0 < d < n; others are left alone), by
// bisection of the keys' values, both at once: a step is a few dependent reads and a
// barrier.  Every eighth step the values are narrowed to keys that are there: the 63-bit
// ranks of a shallow octree end in long stretches without any.  Called by the whole CTA.
template <int NT, int TRACKED, typename T, typename KT>
__device__ __forceinline__ void run_cuts(const SortedRuns<T, KT>& s, const uint32_t (&d)[2], RunCut<KT> (&cut)[2],
                                         WindowSmem<NT, TRACKED>& w) {
  const uint32_t tid = threadIdx.x, k = s.runs();
  bool on[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) on[c] = d[c] > 0 && d[c] < s.n;
  const auto lo_of = [&](int c, uint32_t x) { return x < TRACKED ? (int)w.lo[c][x] : 0; };
  const auto hi_of = [&](int c, uint32_t x) { return x < TRACKED ? (int)w.hi[c][x] : s.length(x); };
  for (uint32_t x = tid; x < min(k, (uint32_t)TRACKED); x += NT) {
    w.lo[0][x] = w.lo[1][x] = 0;
    w.hi[0][x] = w.hi[1][x] = (uint16_t)s.length(x);
  }
  KT lo[2], hi[2];  // the smallest v that at least d keys do not exceed lies in [lo, hi]
  const auto narrow = [&](bool start) {
    __syncthreads();
    if (tid < 2) {
      w.least[tid] = ~0ull;
      w.most[tid] = 0ull;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!on[c]) continue;
      KT first = ~(KT)0, last = 0;
      for (uint32_t x = tid; x < k; x += NT) {
        const int a = lo_of(c, x), b = hi_of(c, x);
        if (a >= b) continue;
        first = min(first, s.at(x * s.R + a));
        last = max(last, s.at(x * s.R + b - 1));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
        last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
      }
      if ((tid & 31) == 0) {
        atomicMin(&w.least[c], (unsigned long long)first);
        atomicMax(&w.most[c], (unsigned long long)last);
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!on[c]) continue;
      lo[c] = start ? (KT)w.least[c] : max(lo[c], (KT)w.least[c]);
      hi[c] = start ? (KT)w.most[c] : min(hi[c], (KT)w.most[c]);
    }
  };
  // Sums over the CTA; three sets of words in turn, so that one barrier does.
  int slot = 0;
  if (tid < 6) w.count[tid >> 1][tid & 1] = 0u;
  const auto total = [&](uint32_t (&mine)[2]) {
    const int next = slot == 2 ? 0 : slot + 1;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      mine[c] = __reduce_add_sync(0xffffffffu, mine[c]);
      if ((tid & 31) == 0 && mine[c]) atomicAdd(&w.count[slot][c], mine[c]);
    }
    if (tid < 2) w.count[next][tid] = 0u;  // (last read before the barrier before this one)
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 2; ++c) mine[c] = w.count[slot][c];
    slot = next;
  };
  narrow(true);
  for (int step = 1; (on[0] && lo[0] < hi[0]) || (on[1] && lo[1] < hi[1]); ++step) {
    KT v[2];
    uint32_t n[2] = {0u, 0u};
    bool open[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      open[c] = on[c] && lo[c] < hi[c];
      v[c] = open[c] ? lo[c] + (hi[c] - lo[c]) / 2 : 0;
    }
    for (uint32_t x = tid; x < k; x += NT) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (!open[c]) continue;
        const int m = s.template below<true>(x, v[c], lo_of(c, x), hi_of(c, x));
        if (x < TRACKED) w.mid[c][x] = (uint16_t)m;
        n[c] += (uint32_t)m;
      }
    }
    total(n);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!open[c]) continue;
      const bool enough = n[c] >= d[c];
      for (uint32_t x = tid; x < min(k, (uint32_t)TRACKED); x += NT) (enough ? w.hi : w.lo)[c][x] = w.mid[c][x];
      if (enough) hi[c] = v[c];
      else lo[c] = v[c] + 1;
    }
    if (step % 8 == 0) narrow(false);
  }
  uint32_t n[2] = {0u, 0u};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (!on[c]) continue;
    for (uint32_t x = tid; x < k; x += NT) {
      // the keys equal to v (narrowing may have moved v past others)
      const int a = s.template below<false>(x, lo[c], lo_of(c, x), hi_of(c, x));
      if (x < TRACKED) w.lo[c][x] = (uint16_t)a;
      n[c] += (uint32_t)a;
    }
  }
  total(n);
#pragma unroll
  for (int c = 0; c < 2; ++c)
    if (on[c]) cut[c] = RunCut<KT>{lo[c], d[c] - n[c]};
}

// Puts the keys [d0, d1) of the merged order side by side, in the runs' order:
// put(place in the window, index in the segment, key).  At most R of them.
template <int NT, int TRACKED, typename T, typename KT, class PUT>
__device__ void gather_window(const SortedRuns<T, KT>& s, uint32_t d0, uint32_t d1, WindowSmem<NT, TRACKED>& w,
                              PUT put) {
  const uint32_t tid = threadIdx.x, k = s.runs();
  const uint32_t d[2] = {d0, d1};
  RunCut<KT> cut[2] = {{0, 0}, {0, 0}};
  run_cuts<NT>(s, d, cut, w);
  uint32_t ties0 = 0, ties1 = 0, filled = 0;  // of the runs before the current ones
  for (uint32_t x0 = 0; x0 < k; x0 += NT) {
    const uint32_t x = x0 + tid;
    const int len = x < k ? s.length(x) : 0;
    int a[2], b[2];  // [a, b): the run's keys that equal the cut's v
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (d[c] == 0 || d[c] == s.n || x >= k) {
        a[c] = b[c] = d[c] == 0 ? 0 : len;
      } else {
        a[c] = x < TRACKED ? (int)w.lo[c][x] : s.template below<false>(x, cut[c].v, 0, len);
        b[c] = s.template below<true>(x, cut[c].v, a[c], x < TRACKED ? (int)w.hi[c][x] : len);
      }
    }
    uint32_t t0, t1, m;
    const uint32_t p0 = block_exclusive_scan<NT>((uint32_t)(b[0] - a[0]), w.scan, t0) + ties0;
    const uint32_t p1 = block_exclusive_scan<NT>((uint32_t)(b[1] - a[1]), w.scan, t1) + ties1;
    const int from = a[0] + (int)min((uint32_t)(b[0] - a[0]), cut[0].q - min(cut[0].q, p0));
    const int to = a[1] + (int)min((uint32_t)(b[1] - a[1]), cut[1].q - min(cut[1].q, p1));
    w.off[tid] = block_exclusive_scan<NT>((uint32_t)(to - from), w.scan, m);
    w.src[tid] = x * s.R + (uint32_t)from;
    ties0 += t0;
    ties1 += t1;
    __syncthreads();
    for (uint32_t i = tid; i < m; i += NT) {
      int lo = 0, hi = NT;  // the last piece that starts at i or before
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (w.off[mid] <= i) lo = mid;
        else hi = mid;
      }
      const uint32_t at = w.src[lo] + (i - w.off[lo]);
      put(filled + i, at, s.at(at));
    }
    filled += m;
    __syncthreads();
  }
}

}  // namespace svr
