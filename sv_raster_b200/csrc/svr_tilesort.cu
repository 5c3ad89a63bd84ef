// Batched binning without instance keys: per-tile counts to ranges, and the sort
// of every tile's instances by rank position.
//
// The projection adds every visible (voxel, view) pair's instances to its tiles'
// counts; tile_ranges scans them, the scatter (svr_batch.cu) drops each
// instance's 32-bit rank position into its tile's range, in the order of its
// atomics, and the kernels here sort each range.  A rank position is unique
// inside a tile and names its (voxel, quadrant) pair, so it is key and value at
// once: 4 bytes move where (tile | position) keys with values moved 12, and the
// sorted value is looked up at the end (val_of_pos).
//
// Sorting 26-bit positions by counting digits cost a small tile four passes of
// zeroing, counting and scanning 256 digits: 1,650 warp instructions per 32 keys.
// Here a warp sorts up to 512 keys in registers with a bitonic network (about 70
// per 32 keys); longer segments merge four of those to a run, and their runs.  Eight full-HD views of 8M voxels
// (60M instances, 259,000 tiles): sort 2.23 -> 0.73 ms; 2M voxels, one view: 119 ->
// 52 us.
#include "svr_block.cuh"
#include "svr_common.cuh"
#include "svr_kernels.h"
#include "svr_runs.cuh"

#include <algorithm>
#include <mutex>

namespace svr {

namespace {

constexpr int kScanT = 256;
constexpr int kScanI = 16;
constexpr int kScanPer = kScanT * kScanI;  // tiles per CTA of the range scan

constexpr int kWarpKeys = 512;             // keys a warp sorts in registers
constexpr int kRunWarps = 4;               // 8: 826 us where 4 take 459 and the longer merge 70 more
constexpr int kRun = kWarpKeys * kRunWarps;  // keys of one sorted run of a long segment
constexpr int kTileWarps = 4;
constexpr int kMergeT = 512;
// Segments of more runs are merged by windows: 25 runs 2.2 -> 1.6 ms (20M instances), 6
// to 10 runs by rank 1.05, by windows 1.09 (all of prepare, 2.2M instances).
constexpr uint32_t kManyRuns = 16;
using MergeWindow = WindowSmem<kMergeT, 2816>;

}  // namespace

size_t tile_scan_temp_bytes(int n_tiles) {
  return ((size_t)n_tiles / kScanPer + 2) * sizeof(unsigned long long);
}

// Runs of the segments longer than a warp sorts: at most one per kRun instances
// and one more per such segment.
static uint32_t run_list_cap(size_t cap, int n_tiles) {
  const size_t longs = std::min<size_t>((size_t)n_tiles, cap / (kWarpKeys + 1));
  return (uint32_t)(cap / kRun + longs + 1);
}
size_t tile_sort_temp_bytes(size_t cap, int n_tiles) { return (size_t)run_list_cap(cap, n_tiles) * sizeof(uint4); }

__global__ void __launch_bounds__(kScanT)
tile_counts_reduce_kernel(const uint32_t* __restrict__ counts, int n, unsigned long long* __restrict__ sums) {
  __shared__ unsigned long long s_warp[kScanT / 32 + 1];
  unsigned long long s = 0;
#pragma unroll
  for (int r = 0; r < kScanI; ++r) {
    const int i = blockIdx.x * kScanPer + r * kScanT + threadIdx.x;
    if (i < n) s += counts[i];
  }
  unsigned long long tot;
  block_exclusive_scan<kScanT>(s, s_warp, tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// One warp per tile.
__global__ void __launch_bounds__(256)
tile_copies_kernel(uint32_t* __restrict__ copies, int n_copies, uint32_t stride, int n_tiles,
                   uint32_t* __restrict__ counts) {
  const int lane = threadIdx.x & 31, t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (t >= n_tiles) return;
  uint32_t before = 0;
  for (int c0 = 0; c0 < n_copies; c0 += 32) {
    const int c = c0 + lane;
    const uint32_t x = c < n_copies ? copies[c * stride + t] : 0u;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (c < n_copies) copies[c * stride + t] = before + incl - x;
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) counts[t] = before;
}

void launch_tile_copies(uint32_t* copies, int n_copies, uint32_t stride, int n_tiles, uint32_t* counts,
                        cudaStream_t stream) {
  tile_copies_kernel<<<(n_tiles + 7) / 8, 256, 0, stream>>>(copies, n_copies, stride, n_tiles, counts);
}

// Ranges [start, end) of every tile, clamped to the capacity, empty ones (0, 0);
// counts[t] becomes the tile's scatter cursor.  The last CTA stores the instance
// count and flags one past the capacity.  Tiles longer than a warp sorts are
// listed as runs of kRun instances: (run start, run n, segment start, segment n).
__global__ void __launch_bounds__(kScanT)
tile_ranges_from_counts_kernel(uint32_t* __restrict__ counts, int n, const unsigned long long* __restrict__ sums,
                               uint32_t cap, uint2* __restrict__ ranges, uint32_t* __restrict__ d_total,
                               uint32_t* __restrict__ err, uint4* __restrict__ runs, uint32_t* __restrict__ n_runs,
                               uint32_t runs_cap) {
  __shared__ unsigned long long s_warp[kScanT / 32 + 1];
  unsigned long long before = 0, tot;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kScanT) before += sums[b];
  block_exclusive_scan<kScanT>(before, s_warp, tot);
  const unsigned long long base = tot;
  // thread t owns tiles [t * kScanI, (t + 1) * kScanI) of the CTA's
  const int t0 = blockIdx.x * kScanPer + threadIdx.x * kScanI;
  uint32_t c[kScanI];
  unsigned long long s = 0;
#pragma unroll
  for (int r = 0; r < kScanI; ++r) {
    c[r] = t0 + r < n ? counts[t0 + r] : 0u;
    s += c[r];
  }
  unsigned long long at = block_exclusive_scan<kScanT>(s, s_warp, tot) + base;
#pragma unroll
  for (int r = 0; r < kScanI; ++r) {
    if (t0 + r >= n) break;
    const unsigned long long end = at + c[r];
    const uint32_t a = (uint32_t)min(at, (unsigned long long)cap), b = (uint32_t)min(end, (unsigned long long)cap);
    counts[t0 + r] = a;
    ranges[t0 + r] = a < b ? make_uint2(a, b) : make_uint2(0u, 0u);
    if (b - a > (uint32_t)kWarpKeys) {
      const uint32_t len = b - a, k = (len + kRun - 1) / kRun;
      const uint32_t e0 = atomicAdd(n_runs, k);
      for (uint32_t j = 0; j < k; ++j)
        if (e0 + j < runs_cap) runs[e0 + j] = make_uint4(a + j * kRun, min((uint32_t)kRun, len - j * kRun), a, len);
    }
    at = end;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    const unsigned long long total = base + tot;
    *d_total = (uint32_t)min(total, 0xffffffffull);
    if (total > cap) atomicOr(err, SVR_DEVERR_CAPACITY);
  }
}

// Bitonic network over 32 * K keys, lane l holding places [l * K, (l + 1) * K).
// A step between lanes takes a shuffle and one min or max per key.
template <int K>
__device__ __forceinline__ void warp_sort(uint32_t (&r)[K], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= K) {
        const int m = stride / K;
        const bool up = size == 32 * K || ((lane * K) & size) == 0;
        const bool low = ((lane & m) == 0) == up;
#pragma unroll
        for (int i = 0; i < K; ++i) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, r[i], m);
          r[i] = low ? min(r[i], o) : max(r[i], o);
        }
      } else {
#pragma unroll
        for (int i = 0; i < K; ++i) {
          if (i & stride) continue;
          const bool up = size == 32 * K || (size >= K ? ((lane * K) & size) == 0 : (i & size) == 0);
          const uint32_t a = r[i], b = r[i + stride];
          r[i] = up ? min(a, b) : max(a, b);
          r[i + stride] = up ? max(a, b) : min(a, b);
        }
      }
    }
  }
}

// Sorts n (<= 32 K) keys from global memory and leaves them in s[0, n).
template <int K>
__device__ __forceinline__ void warp_sort_to_shared(const uint32_t* __restrict__ keys, int n, uint32_t* s, int lane) {
  uint32_t r[K];
#pragma unroll
  for (int i = 0; i < K; ++i) r[i] = i * 32 + lane < n ? keys[i * 32 + lane] : 0xffffffffu;
  warp_sort(r, lane);
  if constexpr (K % 4 == 0) {
#pragma unroll
    for (int i = 0; i < K; i += 4)
      reinterpret_cast<uint4*>(s + lane * K)[i / 4] = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) s[lane * K + i] = r[i];
  }
  __syncwarp();
}

// One warp per tile: segments of at most kWarpKeys instances.
__global__ void __launch_bounds__(32 * kTileWarps)
sort_short_tiles_kernel(const uint2* __restrict__ ranges, int n_tiles, const uint32_t* __restrict__ keys,
                        const uint32_t* __restrict__ val_of_pos, uint32_t* __restrict__ vals) {
  __shared__ __align__(16) uint32_t s_keys[kTileWarps][kWarpKeys];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * kTileWarps + warp;
  if (t >= n_tiles) return;
  const uint2 rg = ranges[t];
  const int n = (int)(rg.y - rg.x);
  if (n == 0 || n > kWarpKeys) return;
  uint32_t* s = s_keys[warp];
  const uint32_t* k = keys + rg.x;
  if (n <= 32) warp_sort_to_shared<1>(k, n, s, lane);
  else if (n <= 64) warp_sort_to_shared<2>(k, n, s, lane);
  else if (n <= 128) warp_sort_to_shared<4>(k, n, s, lane);
  else if (n <= 256) warp_sort_to_shared<8>(k, n, s, lane);
  else warp_sort_to_shared<16>(k, n, s, lane);
#pragma unroll 4
  for (int i = lane; i < n; i += 32) vals[rg.x + i] = val_of_pos[s[i]];
}

// Smallest i with a[i] ordered after the first d - i of b: how many of the first
// d merged keys come from a (na and nb keys; no key is in both).
__device__ __forceinline__ int merge_split(const uint32_t* a, int na, const uint32_t* b, int nb, int d) {
  int lo = max(0, d - nb), hi = min(d, na);
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a[mid] < b[d - 1 - mid]) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Merges sorted runs of len keys in s, n keys in all (padded with 0xffffffff to T * PER),
// pairwise until one is left, every thread taking PER consecutive outputs.  Starts with
// a barrier.
template <int T, int PER>
__device__ __forceinline__ void merge_in_shared(uint32_t* s, int len, int n) {
  const int d0 = threadIdx.x * PER;             // first output
  for (; len < n; len <<= 1) {
    __syncthreads();
    uint32_t out[PER];
    const int pair = d0 & ~(2 * len - 1);       // the two runs [pair, pair + len), [pair + len, pair + 2 len)
    const uint32_t* a = s + pair;
    const uint32_t* b = a + len;
    int i = merge_split(a, len, b, len, d0 - pair), j = d0 - pair - i;
    // the heads stay in registers; an exhausted run's is the padding key, which
    // no key is above
    uint32_t x = i < len ? a[i] : 0xffffffffu, y = j < len ? b[j] : 0xffffffffu;
#pragma unroll
    for (int o = 0; o < PER; ++o) {
      const bool from_a = x <= y;
      out[o] = min(x, y);
      i += from_a;
      j += !from_a;
      const bool more = (from_a ? i : j) < len;
      const uint32_t next = more ? (from_a ? a[i] : b[j]) : 0xffffffffu;
      x = from_a ? next : x;
      y = from_a ? y : next;
    }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < PER; o += 4)
      reinterpret_cast<uint4*>(s + d0)[o / 4] = make_uint4(out[o], out[o + 1], out[o + 2], out[o + 3]);
  }
}

// One CTA per listed run: its warps sort kWarpKeys each, then those are merged.  The
// run of a one-run segment is final; others go back in place for the merge below.
__global__ void __launch_bounds__(32 * kRunWarps)
sort_runs_kernel(const uint4* __restrict__ runs, const uint32_t* __restrict__ n_runs, uint32_t runs_cap,
                 uint32_t* __restrict__ keys, const uint32_t* __restrict__ val_of_pos, uint32_t* __restrict__ vals) {
  __shared__ __align__(16) uint32_t s[kRun];
  constexpr int PER = kRun / (32 * kRunWarps);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t count = min(*n_runs, runs_cap);
  for (uint32_t e = blockIdx.x; e < count; e += gridDim.x) {
    const uint4 run = runs[e];
    const int n = (int)run.y;
    warp_sort_to_shared<kWarpKeys / 32>(keys + run.x + warp * kWarpKeys, max(0, n - warp * kWarpKeys),
                                        s + warp * kWarpKeys, lane);
    merge_in_shared<32 * kRunWarps, PER>(s, kWarpKeys, n);
    __syncthreads();
    if (run.w == run.y) {
      for (int i = tid; i < n; i += 32 * kRunWarps) vals[run.x + i] = val_of_pos[s[i]];
    } else {
      for (int i = tid; i < n; i += 32 * kRunWarps) keys[run.x + i] = s[i];
    }
    __syncthreads();
  }
}

// One CTA per run of a longer segment: a key's place is its index in its run
// plus, for every other run, the number of that run's keys below it.  That takes
// time with the square of the runs, so segments of many are merged by windows of as
// many keys instead (svr_runs.cuh).
__global__ void __launch_bounds__(kMergeT, 4)
merge_runs_kernel(const uint4* __restrict__ runs, const uint32_t* __restrict__ n_runs, uint32_t runs_cap,
                  const uint32_t* __restrict__ keys, const uint32_t* __restrict__ val_of_pos,
                  uint32_t* __restrict__ vals) {
  __shared__ __align__(16) uint32_t s_other[kRun];
  __shared__ MergeWindow s_window;
  constexpr int PER = kRun / kMergeT;
  const uint32_t count = min(*n_runs, runs_cap);
  const int tid = threadIdx.x;
  for (uint32_t e = blockIdx.x; e < count; e += gridDim.x) {
    const uint4 run = runs[e];
    if (run.w == run.y) continue;  // already final (uniform over the CTA)
    const int n = (int)run.y;
    const uint32_t r = (run.x - run.z) / kRun, k = (run.w + kRun - 1) / kRun;
    if (k > kManyRuns) {  // (window r has as many keys as run r)
      gather_window<kMergeT>(SortedRuns<uint32_t, uint32_t>{keys + run.z, run.w, kRun}, r * kRun, r * kRun + n,
                             s_window, [&](uint32_t i, uint32_t, uint32_t key) { s_other[i] = key; });
      for (int i = n + tid; i < kRun; i += kMergeT) s_other[i] = 0xffffffffu;
      __syncthreads();
      uint32_t* mine = s_other + (tid >> 5) * 32 * PER;
      const int lane = tid & 31;
      uint32_t x[PER];
#pragma unroll
      for (int o = 0; o < PER; ++o) x[o] = mine[o * 32 + lane];
      warp_sort(x, lane);
      __syncwarp();
#pragma unroll
      for (int o = 0; o < PER; ++o) mine[lane * PER + o] = x[o];
      merge_in_shared<kMergeT, PER>(s_other, 32 * PER, n);
      __syncthreads();
      for (int i = tid; i < n; i += kMergeT) vals[run.x + i] = val_of_pos[s_other[i]];
      __syncthreads();
      continue;
    }
    uint32_t own[PER], below[PER];
#pragma unroll
    for (int o = 0; o < PER; ++o) {
      const int i = tid + o * kMergeT;
      own[o] = i < n ? keys[run.x + i] : 0xffffffffu;
      below[o] = 0u;
    }
    for (uint32_t x = 0; x < k; ++x) {
      if (x == r) continue;
      const int nx = (int)min((uint32_t)kRun, run.w - x * kRun);
      __syncthreads();
      for (int i = tid; i < nx; i += kMergeT) s_other[i] = keys[run.z + x * kRun + i];
      __syncthreads();
#pragma unroll
      for (int o = 0; o < PER; ++o) {
        int lo = 0, hi = nx;  // the keys of run x below own[o]
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_other[mid] < own[o]) lo = mid + 1;
          else hi = mid;
        }
        below[o] += (uint32_t)lo;
      }
    }
#pragma unroll
    for (int o = 0; o < PER; ++o) {
      const int i = tid + o * kMergeT;
      if (i < n) vals[run.z + (uint32_t)i + below[o]] = val_of_pos[own[o]];
    }
  }
}

void launch_tile_ranges_from_counts(uint32_t* counts, int n_tiles, uint32_t cap, uint2* ranges, uint32_t* d_total,
                                    uint32_t* err, void* scan_temp, void* run_list, uint32_t* n_runs,
                                    cudaStream_t stream) {
  if (n_tiles <= 0) return;
  unsigned long long* sums = static_cast<unsigned long long*>(scan_temp);
  const int nb = (n_tiles + kScanPer - 1) / kScanPer;
  if (nb > 1) tile_counts_reduce_kernel<<<nb - 1, kScanT, 0, stream>>>(counts, n_tiles, sums);
  tile_ranges_from_counts_kernel<<<nb, kScanT, 0, stream>>>(counts, n_tiles, sums, cap, ranges, d_total, err,
                                                            static_cast<uint4*>(run_list), n_runs,
                                                            run_list_cap(cap, n_tiles));
}

void launch_tile_sort(const uint2* ranges, int n_tiles, uint32_t* keys, const uint32_t* val_of_pos, uint32_t* vals,
                      size_t cap, const void* run_list, const uint32_t* n_runs, cudaStream_t stream) {
  if (n_tiles <= 0 || cap == 0) return;
  sort_short_tiles_kernel<<<(n_tiles + kTileWarps - 1) / kTileWarps, 32 * kTileWarps, 0, stream>>>(
      ranges, n_tiles, keys, val_of_pos, vals);
  if (cap <= (size_t)kWarpKeys) return;
  const uint32_t runs_cap = run_list_cap(cap, n_tiles);
  const uint4* runs = static_cast<const uint4*>(run_list);
  const int grid = (int)std::min<int64_t>(runs_cap, (int64_t)sm_count() * 8);
  sort_runs_kernel<<<grid, 32 * kRunWarps, 0, stream>>>(runs, n_runs, runs_cap, keys, val_of_pos, vals);
  if (cap <= (size_t)kRun) return;
  const int mgrid = (int)std::min<int64_t>(runs_cap, (int64_t)sm_count() * 4);
  merge_runs_kernel<<<mgrid, kMergeT, 0, stream>>>(runs, n_runs, runs_cap, keys, val_of_pos, vals);
}

// --------------------------------------------------------------------------
// Work order of few tiles in one launch: one CTA counts the eighth-octave cost
// buckets and hands every tile a place, largest first (the order inside a bucket
// is that of its atomics).  Many tiles take the radix sort (launch_tile_order).
// --------------------------------------------------------------------------
constexpr int kOrderT = 1024;
constexpr uint32_t kOrderTiles = 6144;  // 2,400 tiles: 6 us; 17,000: 28 against 10 in four launches
bool small_tile_order_fits(uint32_t n_tiles) { return n_tiles <= kOrderTiles; }

__global__ void __launch_bounds__(kOrderT)
small_tile_order_kernel(const uint2* __restrict__ ranges, const uint32_t* __restrict__ tile_last, uint32_t n,
                        uint32_t* __restrict__ order, uint32_t* __restrict__ counter) {
  __shared__ uint32_t s_at[256];
  __shared__ uint32_t s_warp[kOrderT / 32 + 1];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (tid == 0 && counter) *counter = 0u;
  if (tid < 256) s_at[tid] = 0u;
  __syncthreads();
  const auto bucket = [&](uint32_t t) {
    const uint2 r = ranges[t];
    const uint32_t end = tile_last ? tile_last[t] : r.y;
    const uint32_t cost = end > r.x ? end - r.x : 0u;
    return 255u - min(255u, (uint32_t)(log2f((float)cost + 1.f) * 7.9f));
  };
  constexpr int U = 4;
  const uint32_t n_up = (n + kOrderT * U - 1) / (kOrderT * U) * (kOrderT * U);
  for (int pass = 0; pass < 2; ++pass) {
    for (uint32_t t0 = tid; t0 < n_up; t0 += kOrderT * U) {
      uint32_t b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) b[u] = t0 + u * kOrderT < n ? bucket(t0 + u * kOrderT) : 0xffffffffu;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t peers = __match_any_sync(0xffffffffu, b[u]);
        const int leader = __ffs(peers) - 1;
        uint32_t at = 0;
        if ((int)lane == leader && b[u] != 0xffffffffu) at = atomicAdd(&s_at[b[u]], (uint32_t)__popc(peers));
        at = __shfl_sync(0xffffffffu, at, leader);
        if (pass == 1 && b[u] != 0xffffffffu) order[at + __popc(peers & lanemask_lt())] = t0 + u * kOrderT;
      }
    }
    __syncthreads();
    if (pass == 0) {
      uint32_t tot;
      const uint32_t x = tid < 256 ? s_at[tid] : 0u;
      const uint32_t ex = block_exclusive_scan<kOrderT>(x, s_warp, tot);
      if (tid < 256) s_at[tid] = ex;
      __syncthreads();
    }
  }
}

void launch_small_tile_order(const uint2* ranges, const uint32_t* tile_last, uint32_t n_tiles, uint32_t* order,
                             uint32_t* counter, cudaStream_t stream) {
  small_tile_order_kernel<<<1, kOrderT, 0, stream>>>(ranges, tile_last, n_tiles, order, counter);
}

}  // namespace svr
