// Multi-view batched path: N views of one voxel set projected, binned,
// composited and back-propagated with one launch per stage over all views,
// without any host round trip (capturable in a CUDA graph).
//
// No reference counterpart: the reference renders one view per call and
// reads the instance count back to the host (forward.cu:601-734).  Per view,
// the results are those of the plain path:
//   - projection is project_voxel (preprocess.cu:24-132 arithmetic), fused
//     with the SH colour of each visible (voxel, view) (sh_compute.cu:54-106);
//   - instances of all views share one flat array, tile after tile, sorted
//     inside a tile by rank position: the position of the instance's (voxel,
//     quadrant) pair in the ascending order of all 8P pairs' Morton ranks
//     (ties by voxel, then quadrant: the reference's generation order).  The
//     positions are view-independent, built once per plan by one radix sort,
//     and order instances exactly as the 48-bit ranks do, in ceil(log2 8P)
//     bits instead of 48.  The rank itself is compressed for the position
//     sort: with every voxel at octree level <= L < 16 its lowest 3*(16-L)
//     bits are the quadrant repeated, so (rank >> 3*(16-L)) << 3 | quadrant
//     orders pairs exactly as the full rank does;
//   - compositing / backward are the same per-tile device functions.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/svr_b200.h"
#include "svr_common.cuh"
#include "svr_kernels.h"
#include "svr_project.cuh"
#include "svr_render.cuh"
#include "svr_render_bwd.cuh"
#include "svr_render_fwd.cuh"
#include "svr_sh.cuh"

using namespace svr;

namespace svr {
// Instance keys: tile id above bit 32, rank position below.
constexpr int kPosShift = 32;
}  // namespace svr

namespace {
constexpr size_t kAlign = 256;
inline size_t align_up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }
}  // namespace

namespace svr {

struct GroupTable {
  int n;
  int v0[kMaxViews + 1];          // first view of each group (+ end)
  uint32_t tile_base[kMaxViews];  // first global tile of each group
};

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
// Tiles of a pixel bbox in one view, numbered row by row (none when not on).
constexpr uint32_t kOwnTiles = 4;  // pairs of at most this many tiles: handled by their own thread
struct TileRect {
  uint32_t first, w, n, pitch;
  __device__ __forceinline__ TileRect() {}
  __device__ __forceinline__ TileRect(uint2 bbox, const ViewParams& vp, bool on) : first(0), w(1), n(0), pitch(0) {
    if (!on) return;
    int x0, y0, x1, y1;
    bbox_tile_rect(bbox, vp.grid_x, vp.grid_y, vp.tile_shift, x0, y0, x1, y1);
    pitch = (uint32_t)vp.grid_x;
    first = (uint32_t)y0 * pitch + (uint32_t)x0;
    w = (uint32_t)(x1 - x0 + 1);
    n = w * (uint32_t)(y1 - y0 + 1);
  }
  __device__ __forceinline__ uint32_t tile(uint32_t k) const { return first + k / w * pitch + k % w; }
  __device__ __forceinline__ TileRect from(int lane) const {
    TileRect r;
    r.first = __shfl_sync(0xffffffffu, first, lane);
    r.w = __shfl_sync(0xffffffffu, w, lane);
    r.n = __shfl_sync(0xffffffffu, n, lane);
    r.pitch = __shfl_sync(0xffffffffu, pitch, lane);
    return r;
  }
};

// Copies of the tile counts (and of the scatter's cursors): with many voxels over few
// tiles their atomics meet in a handful of cache lines.  n copies (a power of two),
// stride words apart; 128 consecutive voxels share one.  20M voxels, 64 tiles: the
// projection with its counts 4.98 -> 0.62 ms, the scatter 5.01 -> 0.29.
struct TileCopies {
  uint32_t n, stride;
  __device__ __forceinline__ uint32_t offset(uint32_t voxel) const { return (voxel / 128u & (n - 1u)) * stride; }
};

// View-dependent colour of a visible voxel (sh_compute.cu:54-106); m holds the
// view's w2c and c2w.
template <int DEG, typename TS>
__device__ __forceinline__ void view_colour(const float* m, float cx, float cy, float cz, const float c0[3],
                                            const TS* sh, float* __restrict__ rgb) {
  float dx = cx - m[12 + 3], dy = cy - m[12 + 7], dz = cz - m[12 + 11];
  const float rn = rnorm3df(dx, dy, dz);
  dx = dx * rn; dy = dy * rn; dz = dz * rn;
#pragma unroll
  for (int c = 0; c < 3; ++c) rgb[c] = sh_channel<DEG>(dx, dy, dz, c0[c], sh, c);
}

// One thread per voxel, looping over the views: the voxel's centre and size are
// read once and kept in registers, so each view costs the projection arithmetic
// and the per-(view, voxel) writes only.
// With `counts`, every visible pair also adds its instances to its tiles' counts
// (a warp takes the pairs of many tiles together, one tile per lane): 1.78 -> 2.22
// ms (before SH_LAST) for 8M voxels and eight views, where counting in a pass of its own, which
// re-read 20 bytes per pair, took 0.88.  Blocks take the counts' copies in turn (TileCopies).
//
// SH_LAST (two views and more): the colours follow all projections, with the
// coefficients in registers, so they are read once for all views, all in flight
// at once, and are not alive during the projections (where they cost half the
// occupancy): 2.20 -> 1.96 ms for 8M voxels and eight views. With one view there
// is nothing to share and the coefficients are read through the cache where they
// are used: 123 us for 2M voxels, 142 with SH_LAST, 218 with the rows staged in
// shared memory.
template <int DEG, typename TS, bool SH_LAST>
__global__ void __launch_bounds__(128)
project_sh_kernel(const __grid_constant__ ViewTable views, int P, const float* __restrict__ centers,
                  const float* __restrict__ lengths, const TS* __restrict__ sh0, const TS* __restrict__ shs, int M,
                  const int64_t* __restrict__ octpaths, int level_low_bits, int tight, uint32_t* __restrict__ ndup,
                  uint2* __restrict__ bboxes, uint32_t* __restrict__ quads, float* __restrict__ rgbs,
                  uint32_t* __restrict__ err, unsigned long long* __restrict__ pixels, uint32_t* __restrict__ counts,
                  const TileCopies copies) {
  __shared__ float s_m[kMaxViews][24];           // w2c (12) and c2w (12) of every view
  __shared__ unsigned long long s_pixels;
  if (threadIdx.x == 0) s_pixels = 0ull;
  for (int t = threadIdx.x; t < views.n * 24; t += blockDim.x) {
    const int v = t / 24, k = t % 24;
    s_m[v][k] = k < 12 ? views.v[v].w2c[k] : views.v[v].c2w[k - 12];
  }
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = i < P;
  const size_t iv = in ? i : 0;
  uint32_t px = 0u;  // bbox pixels over the views (each at most 2^20 here: a warp's sum fits 32 bits)
  // voxels deeper than the plan's max level would break the compressed ranks
  if (level_low_bits > 0 && in && ((uint64_t)octpaths[iv] & ((1ull << level_low_bits) - 1ull)) != 0ull)
    atomicOr(err, SVR_DEVERR_LEVEL);
  const float cx = centers[3 * iv], cy = centers[3 * iv + 1], cz = centers[3 * iv + 2];
  const float len = lengths[iv];
  const TS* sh = shs + iv * (M - 1) * 3;
  unsigned long long seen = 0ull;  // the views that see this voxel
  for (int v = 0; v < views.n; ++v) {
    const size_t o = (size_t)v * P + iv;
    const float* m = s_m[v];
    Projection pr = project_voxel(views.v[v], m, m + 12, cx, cy, cz, len);
    if (tight) tighten_bbox(views.v[v], pr);
    if (in) {
      ndup[o] = pr.n;
      bboxes[o] = pr.bbox;
      quads[o] = pr.quads;
    }
    const bool visible = in && pr.n != 0;
    if (counts) {
      const TileRect rect(pr.bbox, views.v[v], visible);
      const uint32_t per_tile = (uint32_t)__popc(pr.quads);
      uint32_t* c = counts + copies.offset(blockIdx.x * blockDim.x) + views.v[v].tile_base;
      if (rect.n <= kOwnTiles) {
        uint32_t t = rect.first, left = rect.w;
        for (uint32_t k = 0; k < rect.n; ++k) {
          atomicAdd(c + t, per_tile);
          ++t;
          if (--left == 0) {
            left = rect.w;
            t += rect.pitch - rect.w;
          }
        }
      }
      for (uint32_t big = __ballot_sync(0xffffffffu, rect.n > kOwnTiles); big; big &= big - 1) {
        const int src = __ffs(big) - 1;
        const TileRect r = rect.from(src);
        const uint32_t q = __shfl_sync(0xffffffffu, per_tile, src);
        for (uint32_t k = threadIdx.x & 31; k < r.n; k += 32) atomicAdd(c + r.tile(k), q);
      }
    }
    if (!visible) continue;
    px += min((bb_xmax(pr.bbox) - bb_xmin(pr.bbox) + 1u) * (bb_ymax(pr.bbox) - bb_ymin(pr.bbox) + 1u), 1u << 20);
    if constexpr (SH_LAST) {
      seen |= 1ull << v;
    } else {
      const float c0[3] = {ldf(sh0, 3 * iv), ldf(sh0, 3 * iv + 1), ldf(sh0, 3 * iv + 2)};
      view_colour<DEG>(m, cx, cy, cz, c0, sh, rgbs + 3 * o);
    }
  }
  if (SH_LAST && seen) {
    constexpr int ROW = sh_row<DEG>();
    float row[ROW > 0 ? ROW : 1];
#pragma unroll
    for (int k = 0; k < ROW; ++k) row[k] = ldf(sh, k);
    const float c0[3] = {ldf(sh0, 3 * iv), ldf(sh0, 3 * iv + 1), ldf(sh0, 3 * iv + 2)};
    for (unsigned long long left = seen; left; left &= left - 1) {
      const int v = __ffsll((long long)left) - 1;
      view_colour<DEG>(s_m[v], cx, cy, cz, c0, row, rgbs + 3 * ((size_t)v * P + iv));
    }
  }
  __syncwarp();
  px = __reduce_add_sync(0xffffffffu, px);
  if ((threadIdx.x & 31) == 0 && px) atomicAdd(&s_pixels, (unsigned long long)px);
  __syncthreads();
  if (threadIdx.x == 0 && s_pixels) atomicAdd(pixels + blockIdx.x % kCoverageSlots, s_pixels);
}

// Counting-sort scatter: the rank position of every instance to the next free
// place of its tile's range (cursor[global tile], starting at the range's
// start).  Places inside a tile follow the atomics' order; the tile sort orders
// them.  Places past the capacity are left out (the range scan flagged it).
// Pairs of few tiles keep their atomics in flight together; a warp takes the
// others tile by tile, one per lane.  Bound by the returning atomics: 60M
// instances in 1.15 ms, where a lane per instance, decoded from a scan of all
// pairs, with keys and values to store took 1.46 and the scan 0.35.  A pair whose
// tiles and quadrants are not the instances that the projection stored for it is
// flagged, as the other duplications do.
// With copies, cursor[copy][tile] counts from the copy's first place in the tile, whose
// own is start[tile]; without (start is null) it holds the place itself.
__global__ void __launch_bounds__(256)
scatter_positions_kernel(const __grid_constant__ ViewTable views, int P, const uint32_t* __restrict__ rank_pos,
                         const uint2* __restrict__ bboxes, const uint32_t* __restrict__ quads,
                         const uint32_t* __restrict__ ndup, uint32_t* __restrict__ cursor,
                         const TileCopies copies, const uint32_t* __restrict__ start, uint32_t* __restrict__ keys,
                         uint32_t cap, uint32_t* __restrict__ err) {
  const ViewParams& vp = views.v[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const size_t o = (size_t)blockIdx.y * P + i;
  const uint32_t qb = i < P ? quads[o] : 0u;
  if (__ballot_sync(0xffffffffu, qb != 0u) == 0u) return;
  const TileRect rect(qb ? bboxes[o] : make_uint2(0u, 0u), vp, qb != 0u);
  if (qb && rect.n * (uint32_t)__popc(qb) != ndup[o]) atomicOr(err, SVR_DEVERR_DUP_MISMATCH);
  uint32_t* c = cursor + copies.offset((uint32_t)(i - lane)) + vp.tile_base;
  const auto place = [&](uint32_t t) { return atomicAdd(c + t, 1u) + (start ? start[vp.tile_base + t] : 0u); };
  if (rect.n <= kOwnTiles) {
    for (uint32_t qs = qb; qs; qs &= qs - 1) {
      const uint32_t pos = rank_pos[8 * (size_t)i + (__ffs(qs) - 1)];
      uint32_t at[kOwnTiles];
      uint32_t t = rect.first, left = rect.w;
#pragma unroll
      for (uint32_t k = 0; k < kOwnTiles; ++k) {
        if (k < rect.n) at[k] = place(t);
        ++t;
        if (--left == 0) {
          left = rect.w;
          t += rect.pitch - rect.w;
        }
      }
#pragma unroll
      for (uint32_t k = 0; k < kOwnTiles; ++k)
        if (k < rect.n && at[k] < cap) keys[at[k]] = pos;
    }
  }
  for (uint32_t big = __ballot_sync(0xffffffffu, rect.n > kOwnTiles); big; big &= big - 1) {
    const int src = __ffs(big) - 1;
    const TileRect r = rect.from(src);
    const size_t vox = (size_t)(i - lane + src);
    for (uint32_t qs = __shfl_sync(0xffffffffu, qb, src); qs; qs &= qs - 1) {
      const uint32_t pos = rank_pos[8 * vox + (__ffs(qs) - 1)];
      for (uint32_t k = lane; k < r.n; k += 32) {
        const uint32_t at = place(r.tile(k));
        if (at < cap) keys[at] = pos;
      }
    }
  }
}

// Instance segment [start, start + count) of each sort group, clamped to the
// capacity so that an overflowing step still stays inside the buffers.
__global__ void group_segments_kernel(const __grid_constant__ GroupTable gt, int P, const uint32_t* __restrict__ scan,
                                      uint32_t cap, uint32_t* __restrict__ segs) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= gt.n) return;
  const size_t v0 = gt.v0[g], v1 = gt.v0[g + 1];
  const uint32_t start = min(v0 == 0 ? 0u : scan[v0 * P - 1], cap);
  const uint32_t end = min(scan[v1 * P - 1], cap);
  segs[2 * g] = start;
  segs[2 * g + 1] = end - start;
}

// Position of the k-th (0-based) set bit of m (k < popc(m)).
__device__ __forceinline__ int nth_set_bit(uint32_t m, int k) {
  int pos = 0;
  int c = __popc(m & 0xFFFFu);
  if (k >= c) { k -= c; pos += 16; m >>= 16; }
  c = __popc(m & 0xFFu);
  if (k >= c) { k -= c; pos += 8; m >>= 8; }
  c = __popc(m & 0xFu);
  if (k >= c) { k -= c; pos += 4; m >>= 4; }
  c = __popc(m & 0x3u);
  if (k >= c) { k -= c; pos += 2; m >>= 2; }
  if (k >= (int)(m & 1u)) pos += 1;
  return pos;
}

// Duplication for the radix grouping by tile, with the stores of a warp
// coalesced.  The instances of the warp's 32 consecutive (view, voxel) pairs form
// one contiguous run of the scan; the warp walks that run 32 instances at a time,
// each lane decoding its instance (owning voxel, then quadrant / tile row / tile
// column in the plain path's generation order: quadrants ascending, tiles
// row-major, forward.cu:540-562) and writing its key and value at its slot.
__global__ void __launch_bounds__(256)
duplicate_batch_kernel(const __grid_constant__ ViewTable views, int P, const uint32_t* __restrict__ rank_pos,
                       const uint2* __restrict__ bboxes, const uint32_t* __restrict__ quads,
                       const uint32_t* __restrict__ ndup, const uint32_t* __restrict__ scan,
                       uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t cap,
                       uint32_t* __restrict__ err) {
  const int view = blockIdx.y;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool valid = idx < P;
  const size_t o = (size_t)view * P + (valid ? idx : 0);
  const ViewParams& vp = views.v[view];
  const uint32_t n = valid ? ndup[o] : 0u;
  const uint32_t end = valid ? scan[o] : 0u;
  if (n > 0 && end > cap) atomicOr(err, SVR_DEVERR_CAPACITY);
  int tx0 = 0, ty0 = 0, tx1 = 0, ty1 = 0;
  uint32_t qb = 0;
  if (n > 0) {
    bbox_tile_rect(bboxes[o], vp.grid_x, vp.grid_y, vp.tile_shift, tx0, ty0, tx1, ty1);
    qb = quads[o];
    const uint32_t tiles = (uint32_t)((tx1 - tx0 + 1) * (ty1 - ty0 + 1));
    if (tiles * (uint32_t)__popc(qb) != n) atomicOr(err, SVR_DEVERR_DUP_MISMATCH);
  }
  // exclusive scan of n over the warp; the run starts at the first lane's scan offset
  uint32_t incl = n;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  if (total == 0u) return;
  const uint32_t off = incl - n;
  const uint32_t run0 = __shfl_sync(0xffffffffu, end - n, 0) + 0u;  // lane 0's start (valid even if n == 0)
  const uint32_t w = (uint32_t)(tx1 - tx0 + 1);
  const uint32_t tiles = w * (uint32_t)(ty1 - ty0 + 1);
  for (uint32_t cb = 0; cb < total; cb += 32) {
    const uint32_t p = cb + lane;
    // owning lane: the largest s with off_s <= p (offsets are non-decreasing)
    int sl = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const uint32_t t = __shfl_sync(0xffffffffu, off, sl + step);
      if (t <= p) sl += step;
    }
    const uint32_t k = p - __shfl_sync(0xffffffffu, off, sl);
    const uint32_t s_tiles = __shfl_sync(0xffffffffu, tiles, sl);
    const uint32_t s_w = __shfl_sync(0xffffffffu, w, sl);
    const int s_tx0 = __shfl_sync(0xffffffffu, tx0, sl), s_ty0 = __shfl_sync(0xffffffffu, ty0, sl);
    const uint32_t s_qb = __shfl_sync(0xffffffffu, qb, sl);
    const uint32_t slot = run0 + p;
    const bool active = p < total && slot < cap;
    uint32_t q = 0, vid = 0, local = 0;
    if (active) {
      const uint32_t qi = k / s_tiles, rem = k - qi * s_tiles;
      const uint32_t ty = (uint32_t)s_ty0 + rem / s_w, tx = (uint32_t)s_tx0 + rem % s_w;
      q = (uint32_t)nth_set_bit(s_qb, (int)qi);
      vid = (uint32_t)(blockIdx.x * blockDim.x + (threadIdx.x & ~31) + sl);
      local = ty * (uint32_t)vp.grid_x + tx;
    }
    if (active) {
      keys[slot] = ((uint64_t)(vp.sort_tile_off + local) << kPosShift) | rank_pos[8 * (size_t)vid + q];
      vals[slot] = make_sort_val(vid, q);
    }
  }
}

// Rank-position table, step 1: the (compressed) Morton rank of every
// (voxel, quadrant) pair, pair i = 8 * voxel + quadrant, and its index.
// Thread 0 stores the pair count the sort reads.
__global__ void rank_pos_keys_kernel(int P, const int64_t* __restrict__ octpaths, int rank_bits,
                                     uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                     uint32_t* __restrict__ d_n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *d_n = (uint32_t)(8 * (size_t)P);
  if (i >= 8 * (size_t)P) return;
  const uint64_t path = (uint64_t)octpaths[i >> 3];
  const uint32_t q = (uint32_t)(i & 7);
  const int low = (rank_bits == kRankBits) ? 0 : kRankBits - (rank_bits - 3);  // 3*(16-L)
  const uint64_t full = order_rank(path, q);
  keys[i] = (low == 0) ? full : (((full >> low) << 3) | q);
  vals[i] = (uint32_t)i;
}

// Step 2: after a stable sort of the keys, position k holds pair vals[k]; back
// from a position to its instance value (quadrant | voxel).
__global__ void rank_pos_scatter_kernel(size_t n, const uint32_t* __restrict__ sorted_pairs,
                                        uint32_t* __restrict__ rank_pos, uint32_t* __restrict__ val_of_pos) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t pair = sorted_pairs[k];
  rank_pos[pair] = (uint32_t)k;
  val_of_pos[k] = make_sort_val(pair >> 3, pair & 7u);
}

// dL/dSH of every voxel summed over views: sum_v basis(dir_v) * dL/drgb_v
// (sh_compute.cu:110-176 per view), and the subdivision priority summed over
// views (backward.cu:514).  Views where the voxel got no colour gradient are
// skipped.  Each CTA stages its voxels' 3 + 3*(M-1) outputs in shared
// memory and stores them as contiguous rows (the per-voxel rows of dsh0 and
// dshs are 12 B and 180 B long, too short for coalesced per-thread stores).
constexpr int kShBwThreads = 128;

// n staged values to global memory from an even place on, rounded to 16 bits in
// pairs or as they are.
__device__ __forceinline__ void store_staged(float* out, const float* s, int n) {
  for (int e = threadIdx.x; e < n; e += kShBwThreads) out[e] = s[e];
}
__device__ __forceinline__ void store_staged(__nv_bfloat16* out, const float* s, int n) {
  for (int e = threadIdx.x; e < n / 2; e += kShBwThreads)
    reinterpret_cast<__nv_bfloat162*>(out)[e] = __floats2bfloat162_rn(s[2 * e], s[2 * e + 1]);
  if ((n & 1) && threadIdx.x == 0) out[n - 1] = __float2bfloat16_rn(s[n - 1]);
}

// OT: fp32, or bf16 where the coefficients are stored so (the sums are fp32 and
// rounded once either way; writing 16 bits here instead of 32 and casting them
// afterwards: 2M voxels, one view, 70 + 89 -> 53 us; four views' rows in flight
// at once changed nothing).
template <int DEG, typename OT>
__global__ void __launch_bounds__(kShBwThreads)
sh_bw_batch_kernel(const __grid_constant__ ViewTable views, int P, int M, const float* __restrict__ centers,
                   const float4* __restrict__ drgbs, OT* __restrict__ dsh0, OT* __restrict__ dshs,
                   float* __restrict__ subdiv) {
  constexpr int NB = (DEG + 1) * (DEG + 1) - 1;
  __shared__ float s_pos[kMaxViews][3];
  extern __shared__ __align__(16) float s_out[];  // [kShBwThreads][3 + 3 * (M - 1)] then written out
  for (int v = threadIdx.x; v < views.n; v += blockDim.x) {
    s_pos[v][0] = views.v[v].c2w[3];
    s_pos[v][1] = views.v[v].c2w[7];
    s_pos[v][2] = views.v[v].c2w[11];
  }
  __syncthreads();
  const int rest = 3 * (M - 1);
  const int i0 = blockIdx.x * kShBwThreads;
  const int i = i0 + threadIdx.x;
  float a0[3] = {0.f, 0.f, 0.f};
  float sub = 0.f;
  float acc[NB > 0 ? NB : 1][3];
#pragma unroll
  for (int k = 0; k < (NB > 0 ? NB : 1); ++k) acc[k][0] = acc[k][1] = acc[k][2] = 0.f;
  if (i < P) {
    const float cx = centers[3 * (size_t)i], cy = centers[3 * (size_t)i + 1], cz = centers[3 * (size_t)i + 2];
    for (int v = 0; v < views.n; ++v) {
      const float4 g = drgbs[(size_t)v * P + i];
      const float g0 = g.x, g1 = g.y, g2 = g.z;
      sub += g.w;
      if (g0 == 0.f && g1 == 0.f && g2 == 0.f) continue;
      float x = cx - s_pos[v][0], y = cy - s_pos[v][1], z = cz - s_pos[v][2];
      const float rn = rnorm3df(x, y, z);
      x = x * rn; y = y * rn; z = z * rn;
      float basis[15];
      sh_basis_rest<DEG>(x, y, z, basis);
      a0[0] += kC0 * g0; a0[1] += kC0 * g1; a0[2] += kC0 * g2;
#pragma unroll
      for (int k = 0; k < NB; ++k) {
        acc[k][0] += basis[k] * g0;
        acc[k][1] += basis[k] * g1;
        acc[k][2] += basis[k] * g2;
      }
    }
  }
  if (subdiv && i < P) subdiv[i] = sub;
  // stage: dsh0 rows first ([kShBwThreads][3]), then dshs rows ([kShBwThreads][rest])
  float* s0 = s_out;
  float* s1 = s_out + 3 * kShBwThreads;
  const int t = threadIdx.x;
  s0[3 * t + 0] = a0[0];
  s0[3 * t + 1] = a0[1];
  s0[3 * t + 2] = a0[2];
#pragma unroll
  for (int k = 0; k < NB; ++k) {
    s1[t * rest + 3 * k + 0] = acc[k][0];
    s1[t * rest + 3 * k + 1] = acc[k][1];
    s1[t * rest + 3 * k + 2] = acc[k][2];
  }
  for (int k = 3 * NB; k < rest; ++k) s1[t * rest + k] = 0.f;  // coefficients above the degree
  __syncthreads();
  const int nv = min(kShBwThreads, P - i0);
  store_staged(dsh0 + 3 * (size_t)i0, s0, 3 * nv);  // i0 is even: the pairs are aligned
  if (rest > 0) store_staged(dshs + (size_t)rest * i0, s1, rest * nv);
}

inline int bit_width_u64(uint64_t n) {
  int b = 0;
  while (b < 64 && (n >> b)) ++b;
  return b;
}

}  // namespace svr

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
struct svr_batch_plan {
  ViewTable vt;
  GroupTable gt;
  int V;
  int64_t P;
  size_t cap;
  int n_samp;
  int rank_bits;  // compressed Morton rank width (position-table sort)
  int pos_bits;   // bits of a rank position (ceil(log2(8P)))
  int key_bits;   // widest group key (all groups sorted with this many passes)
  bool pos_ready;                 // rank-position tables built for pos_paths in workspace pos_ws
  const int64_t* pos_paths;
  const void* pos_ws;
  int64_t total_tiles, total_pixels;
  // compositing schedule (svr_batch_plan_set_schedule)
  int order_flags;        // bit 0: forward tiles largest first, bit 1: backward (else tile order)
  int fwd_ctas_per_sm;    // resident CTAs per SM of the persistent launches (0 = as many as fit)
  int bwd_ctas_per_sm;
  int seg_small_n, seg_chunk;  // segment-sort buckets (svr_batch_plan_set_sort_buckets)
  int tile_size;               // compositing tile size (8, 16 or 32), fixed at creation
  int stage;                   // records staged per round (svr_batch_plan_set_staging)
  int stage_bwd;               // the backward's, when set apart (svr_batch_plan_set_backward_staging)
  int exact;                   // compositing arithmetic (svr_batch_plan_set_arithmetic): 1 exact, 0 fast
  int pair;                    // two pixels per compositing thread (svr_batch_plan_set_pixels_per_thread)
  int pair_bwd;                // the backward's, when set apart (-1: as pair)
  TileCopies copies;           // of the counting sort's tile counts
  int adaptive;                // the backward's form and staging also by size (svr_batch_plan_set_backward_adaptive)
  int culling;                 // pixel bbox (svr_batch_plan_set_culling): -1 follows exact, 0 rounded, 1 tight
  int binning;                 // 1: counting sort by tile, 0: radix over the tile bits (svr_batch_plan_set_binning)
  // workspace layout (byte offsets)
  size_t o_header, o_ndup, o_scan, o_bbox, o_quad, o_scan_tmp, o_rgbs, o_drgbs;
  size_t o_ka, o_kb, o_va, o_vb, o_sort_tmp, o_ranges, o_tile_last, o_ncontrib;
  size_t o_okey, o_oval, o_order_fwd, o_order_bwd, o_order_tmp, o_pos, o_valpos, o_copies;
  size_t bytes;
};

namespace {

struct BatchPtrs {
  uint32_t* header;
  uint32_t* ndup;
  uint32_t* scan;
  uint2* bbox;
  uint32_t* quad;
  void* scan_tmp;
  float* rgbs;
  float* drgbs;
  uint64_t *ka, *kb;
  uint32_t *va, *vb;
  void* sort_tmp;
  uint2* ranges;
  uint32_t* tile_last;
  uint32_t* ncontrib;
  uint64_t* okey;       // [2][T] order sort keys
  uint32_t* oval;       // [T] order sort input values
  uint32_t* order_fwd;  // [T]
  uint32_t* order_bwd;  // [T]
  void* order_tmp;
  uint32_t* rank_pos;   // [8P] position of (voxel, quadrant) in rank order
  uint32_t* val_of_pos; // [8P] instance value of a position
  uint32_t* counts;     // [T] instances per tile, then the scatter's cursors (after the header)
  uint32_t* copies;     // [copies.n][copies.stride] their copies, when there are several
};

// Header words: [0] instance count, [1] error word, [2] forward work counter,
// [3] backward work counter, [4] tile count read by the order sort, [5] pair
// count read by the rank-position sort, [6] listed runs of long tiles
// (counting sort), [16..] group segments, then the 64-bit pixel counts of
// CoverageCount.  The tile counts follow.
constexpr int kCoverageWord = 16 + 2 * kMaxViews;
constexpr int kHeaderWords = kCoverageWord + 2 * kCoverageSlots;

BatchPtrs ptrs(const svr_batch_plan* p, void* ws) {
  char* b = static_cast<char*>(ws);
  BatchPtrs q;
  q.header = reinterpret_cast<uint32_t*>(b + p->o_header);
  q.ndup = reinterpret_cast<uint32_t*>(b + p->o_ndup);
  q.scan = reinterpret_cast<uint32_t*>(b + p->o_scan);
  q.bbox = reinterpret_cast<uint2*>(b + p->o_bbox);
  q.quad = reinterpret_cast<uint32_t*>(b + p->o_quad);
  q.scan_tmp = b + p->o_scan_tmp;
  q.rgbs = reinterpret_cast<float*>(b + p->o_rgbs);
  q.drgbs = reinterpret_cast<float*>(b + p->o_drgbs);
  q.ka = reinterpret_cast<uint64_t*>(b + p->o_ka);
  q.kb = reinterpret_cast<uint64_t*>(b + p->o_kb);
  q.va = reinterpret_cast<uint32_t*>(b + p->o_va);
  q.vb = reinterpret_cast<uint32_t*>(b + p->o_vb);
  q.sort_tmp = b + p->o_sort_tmp;
  q.ranges = reinterpret_cast<uint2*>(b + p->o_ranges);
  q.tile_last = reinterpret_cast<uint32_t*>(b + p->o_tile_last);
  q.ncontrib = reinterpret_cast<uint32_t*>(b + p->o_ncontrib);
  q.okey = reinterpret_cast<uint64_t*>(b + p->o_okey);
  q.oval = reinterpret_cast<uint32_t*>(b + p->o_oval);
  q.order_fwd = reinterpret_cast<uint32_t*>(b + p->o_order_fwd);
  q.order_bwd = reinterpret_cast<uint32_t*>(b + p->o_order_bwd);
  q.order_tmp = b + p->o_order_tmp;
  q.rank_pos = reinterpret_cast<uint32_t*>(b + p->o_pos);
  q.val_of_pos = reinterpret_cast<uint32_t*>(b + p->o_valpos);
  q.counts = q.header + kHeaderWords;
  q.copies = reinterpret_cast<uint32_t*>(b + p->o_copies);
  return q;
}

unsigned long long* coverage_words(const BatchPtrs& q) {
  return reinterpret_cast<unsigned long long*>(q.header + kCoverageWord);
}

// Several copies of 65,536 voxels and more, where the smallest view has at least 256 per
// tile: as many as spread its counters over 32,768 words, where they help no more, and
// within a million words for all views.  Their clearing and summing take 3 us: a view of
// 16 tiles with 20,000 voxels 21.5 / 24.9 us, 50,000 31.9 / 33.0, 100,000 38.7 / 37.0.  All of prepare, without and with: 2M voxels on 64 tiles 1.21 /
// 0.33 ms, on 1,024 0.64 / 0.23, on 4,096 (490 a tile) 0.30 / 0.22; a step of 2M voxels
// and 16 views of 640x480 to 1600x1200 (four copies) 11.70 / 11.34.
TileCopies tile_copies(const ViewTable& vt, int64_t total_tiles, int64_t P) {
  int64_t fewest = total_tiles;
  for (int v = 0; v < vt.n; ++v) fewest = std::min(fewest, (int64_t)vt.v[v].grid_x * vt.v[v].grid_y);
  int64_t n = 1;
  if (P >= 65536 && P >= 256 * fewest)
    while (n < 64 && 2 * n * fewest <= 32768 && 2 * n * total_tiles <= 1 << 20) n *= 2;
  return TileCopies{(uint32_t)n, (uint32_t)((total_tiles + 31) / 32 * 32)};
}

// Largest-first work order of all tiles into `order`, and the work counter back
// to zero.
void build_tile_order(const svr_batch_plan* p, const BatchPtrs& q, const uint32_t* tile_last, uint32_t* order,
                      uint32_t* counter, cudaStream_t stream) {
  const uint32_t T = (uint32_t)p->total_tiles;
  if (small_tile_order_fits(T)) {
    launch_small_tile_order(q.ranges, tile_last, T, order, counter, stream);
    return;
  }
  cudaMemsetAsync(counter, 0, sizeof(uint32_t), stream);
  launch_tile_order(q.ranges, tile_last, T, q.okey, q.oval, order, q.header + 4, q.order_tmp, stream);
}

inline int check_last() { return cudaGetLastError() == cudaSuccess ? SVR_OK : SVR_ERR_CUDA; }

}  // namespace

extern "C" {

int svr_batch_plan_create(int n_views, const svr_camera* cams, int64_t P, int64_t capacity, int n_samp_per_vox,
                          int max_level, int tile_size, svr_batch_plan** out, size_t* workspace_bytes) {
  if (!out || !workspace_bytes || !cams || n_views < 1 || n_views > kMaxViews || P < 1 ||
      P >= (1ll << kVoxIdBits) || capacity < 0 || capacity > 0xffffffffll || n_samp_per_vox < 1 ||
      n_samp_per_vox > kMaxSamples || max_level < 1 || max_level > kMaxLevels ||
      !(tile_size == 8 || tile_size == 16 || tile_size == 32))
    return SVR_ERR_SHAPE;
  const int tile_shift = tile_size == 8 ? 3 : (tile_size == 16 ? 4 : 5);
  svr_batch_plan* p = new svr_batch_plan();
  memset(&p->vt, 0, sizeof(p->vt));
  p->tile_size = tile_size;
  p->stage = tile_size == 8 ? 64 : 256;
  p->stage_bwd = p->stage;
  p->V = n_views;
  p->P = P;
  p->cap = (size_t)capacity;
  p->n_samp = n_samp_per_vox;
  p->rank_bits = (max_level >= kMaxLevels) ? kRankBits : 3 * max_level + 3;
  p->pos_bits = bit_width_u64((uint64_t)(8 * P - 1));
  p->pos_ready = false;
  p->pos_paths = nullptr;
  p->pos_ws = nullptr;
  p->vt.n = n_views;
  int64_t tiles = 0, pix = 0;
  for (int v = 0; v < n_views; ++v) {
    const svr_camera& c = cams[v];
    if (c.width <= 0 || c.height <= 0 || c.width >= 65536 || c.height >= 65536 || !c.w2c || !c.c2w) {
      delete p;
      return SVR_ERR_SHAPE;
    }
    ViewParams& vp = p->vt.v[v];
    vp.W = c.width;
    vp.H = c.height;
    vp.grid_x = (c.width + tile_size - 1) / tile_size;
    vp.grid_y = (c.height + tile_size - 1) / tile_size;
    vp.tile_shift = tile_shift;
    vp.tanfovx = c.tanfovx;
    vp.tanfovy = c.tanfovy;
    vp.cx = c.cx;
    vp.cy = c.cy;
    vp.focal_x = 0.5f * c.width / c.tanfovx;
    vp.focal_y = 0.5f * c.height / c.tanfovy;
    vp.near_plane = c.near_plane;
    vp.bg = c.bg_color;
    vp.w2c = c.w2c;
    vp.c2w = c.c2w;
    vp.tile_base = (uint32_t)tiles;
    vp.pix_base = (uint32_t)pix;
    tiles += (int64_t)vp.grid_x * vp.grid_y;
    pix += (int64_t)c.width * c.height;
  }
  if (pix > 0xffffffffll) {
    delete p;
    return SVR_ERR_SHAPE;
  }
  p->total_tiles = tiles;
  p->total_pixels = pix;
  // Greedy sort groups: consecutive views while the group's key fits 64 bits
  // (SVR_MAX_KEY_BITS lowers that limit, to exercise grouping in tests).
  int key_limit = 64;
  if (const char* e = getenv("SVR_MAX_KEY_BITS")) key_limit = std::max(1, std::min(64, atoi(e)));
  p->gt.n = 0;
  p->key_bits = 0;
  int v = 0;
  while (v < n_views) {
    const int g = p->gt.n++;
    p->gt.v0[g] = v;
    p->gt.tile_base[g] = p->vt.v[v].tile_base;
    uint64_t gt_tiles = 0;
    int kb = 0;
    while (v < n_views) {
      const uint64_t t2 = gt_tiles + (uint64_t)p->vt.v[v].grid_x * p->vt.v[v].grid_y;
      const int kb2 = kPosShift + bit_width_u64(t2);
      if (kb2 > key_limit && gt_tiles > 0) break;
      if (kb2 > 64) {  // a single view does not fit
        delete p;
        return SVR_ERR_KEYBITS;
      }
      p->vt.v[v].sort_group = g;
      p->vt.v[v].sort_tile_off = (uint32_t)gt_tiles;
      gt_tiles = t2;
      kb = kb2;
      ++v;
    }
    p->key_bits = std::max(p->key_bits, kb);
  }
  p->gt.v0[p->gt.n] = n_views;
  // workspace layout
  const size_t VP = (size_t)n_views * (size_t)P;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = align_up(off);
    const size_t r = off;
    off += bytes;
    return r;
  };
  p->o_header = take((kHeaderWords + (size_t)tiles) * sizeof(uint32_t));
  p->o_ndup = take(VP * 4);
  p->o_scan = take(VP * 4);
  p->o_bbox = take(VP * 8);
  p->o_quad = take(VP * 4);
  p->o_scan_tmp = take(std::max(scan_temp_bytes(VP), tile_scan_temp_bytes((int)tiles)));
  p->o_rgbs = take(VP * 12);
  p->o_drgbs = take(VP * 16);  // [V,P,4]: dL/drgb (xyz) and the subdivision priority (w)
  // the instance arrays also serve the one-time sort of the 8P rank keys
  const size_t kv = std::max(p->cap, (size_t)(8 * P));
  p->o_ka = take(kv * 8);
  p->o_kb = take(kv * 8);
  p->o_va = take(kv * 4);
  p->o_vb = take(kv * 4);
  p->o_sort_tmp = take(std::max({sort_temp_bytes(kv), seg_sort_temp_bytes(p->cap, (int)tiles),
                                 tile_sort_temp_bytes(p->cap, (int)tiles)}));
  p->o_ranges = take((size_t)tiles * 8);
  p->o_tile_last = take((size_t)tiles * 4);
  p->o_ncontrib = take((size_t)pix * 4);
  p->o_okey = take((size_t)tiles * 16);
  p->o_oval = take((size_t)tiles * 4);
  p->o_order_fwd = take((size_t)tiles * 4);
  p->o_order_bwd = take((size_t)tiles * 4);
  p->o_order_tmp = take(sort_temp_bytes((size_t)tiles));
  p->o_pos = take((size_t)(8 * P) * 4);
  p->o_valpos = take((size_t)(8 * P) * 4);
  p->copies = tile_copies(p->vt, tiles, P);
  p->o_copies = take(p->copies.n > 1 ? (size_t)p->copies.n * p->copies.stride * 4 : 0);
  p->bytes = align_up(off) + kAlign;
  p->order_flags = 3;
  p->fwd_ctas_per_sm = 0;
  p->bwd_ctas_per_sm = 0;
  p->seg_small_n = 512;
  p->seg_chunk = 4096;
  p->exact = 0;
  p->pair = 0;
  p->pair_bwd = -1;
  p->adaptive = 1;
  p->culling = -1;
  p->binning = 1;
  ensure_segsort_attributes();
  ensure_fwd_batch_attributes();
  ensure_bwd_batch_attributes();
  ensure_sort_attributes();
  *out = p;
  *workspace_bytes = p->bytes;
  return SVR_OK;
}

void svr_batch_plan_destroy(svr_batch_plan* plan) { delete plan; }

int svr_batch_plan_invalidate_geometry(svr_batch_plan* p) {
  if (!p) return SVR_ERR_SHAPE;
  p->pos_ready = false;
  return SVR_OK;
}

int svr_batch_plan_positions_ready(const svr_batch_plan* p, const void* ws, const int64_t* octree_paths) {
  return p && p->pos_ready && p->pos_ws == ws && p->pos_paths == octree_paths;
}

int svr_batch_plan_set_schedule(svr_batch_plan* p, int order_flags, int fwd_ctas_per_sm, int bwd_ctas_per_sm) {
  if (!p || order_flags < 0 || order_flags > 3 || fwd_ctas_per_sm < 0 || bwd_ctas_per_sm < 0 ||
      fwd_ctas_per_sm > 32 || bwd_ctas_per_sm > 32)
    return SVR_ERR_SHAPE;
  p->order_flags = order_flags;
  p->fwd_ctas_per_sm = fwd_ctas_per_sm;
  p->bwd_ctas_per_sm = bwd_ctas_per_sm;
  return SVR_OK;
}
int svr_batch_plan_set_staging(svr_batch_plan* p, int stage) {
  if (!p || !batch_tile_supported(p->tile_size, stage)) return SVR_ERR_SHAPE;
  p->stage = stage;
  p->stage_bwd = stage;
  return SVR_OK;
}

int svr_batch_plan_set_backward_staging(svr_batch_plan* p, int stage) {
  if (!p || !batch_tile_supported(p->tile_size, stage)) return SVR_ERR_SHAPE;
  p->stage_bwd = stage;
  return SVR_OK;
}

int svr_batch_plan_tile_size(const svr_batch_plan* p) { return p ? p->tile_size : 0; }

int svr_batch_plan_set_pixels_per_thread(svr_batch_plan* p, int pixels) {
  if (!p || (pixels != 1 && pixels != 2)) return SVR_ERR_SHAPE;
  p->pair = pixels == 2;
  return SVR_OK;
}

int svr_batch_plan_set_backward_pixels_per_thread(svr_batch_plan* p, int pixels) {
  if (!p || pixels < 0 || pixels > 2) return SVR_ERR_SHAPE;
  p->pair_bwd = pixels == 0 ? -1 : (pixels == 2);
  return SVR_OK;
}

int svr_batch_plan_set_backward_adaptive(svr_batch_plan* p, int adaptive) {
  if (!p || (adaptive != 0 && adaptive != 1)) return SVR_ERR_SHAPE;
  p->adaptive = adaptive;
  return SVR_OK;
}

int svr_batch_plan_set_arithmetic(svr_batch_plan* p, int exact) {
  if (!p || (exact != 0 && exact != 1)) return SVR_ERR_SHAPE;
  p->exact = exact;
  return SVR_OK;
}

int svr_batch_plan_set_culling(svr_batch_plan* p, int culling) {
  if (!p || culling < -1 || culling > 1) return SVR_ERR_SHAPE;
  p->culling = culling;
  return SVR_OK;
}

int svr_batch_plan_set_reduction(svr_batch_plan* p, int atomic_lanes) {
  if (!p || atomic_lanes < 1 || atomic_lanes > 32) return SVR_ERR_SHAPE;
  return SVR_OK;
}

int svr_batch_plan_set_binning(svr_batch_plan* p, int binning) {
  if (!p || (binning != 0 && binning != 1)) return SVR_ERR_SHAPE;
  p->binning = binning;
  return SVR_OK;
}

int svr_batch_plan_set_sort_buckets(svr_batch_plan* p, int small_n, int chunk) {
  if (!p || !seg_buckets_supported(small_n, chunk)) return SVR_ERR_SHAPE;
  p->seg_small_n = small_n;
  p->seg_chunk = chunk;
  return SVR_OK;
}

int64_t svr_batch_plan_pixels(const svr_batch_plan* p) { return p ? p->total_pixels : 0; }
int64_t svr_batch_plan_tiles(const svr_batch_plan* p) { return p ? p->total_tiles : 0; }
int svr_batch_plan_groups(const svr_batch_plan* p) { return p ? p->gt.n : 0; }

const uint32_t* svr_batch_count_ptr(const svr_batch_plan* p, const void* ws) {
  return reinterpret_cast<const uint32_t*>(static_cast<const char*>(ws) + p->o_header);
}
const uint64_t* svr_batch_bbox_ptr(const svr_batch_plan* p, const void* ws) {
  return reinterpret_cast<const uint64_t*>(static_cast<const char*>(ws) + p->o_bbox);
}

uint32_t* svr_batch_error_ptr(const svr_batch_plan* p, void* ws) {
  return reinterpret_cast<uint32_t*>(static_cast<char*>(ws) + p->o_header) + 1;
}

int svr_batch_arrays(const svr_batch_plan* p, const void* ws, const float** rgbs, const float** drgbs,
                     const uint64_t** ranges, const uint32_t** tile_last, const uint32_t** n_contrib,
                     const uint32_t** ndup, const uint32_t** sorted_vals) {
  if (!p || !ws) return SVR_ERR_SHAPE;
  BatchPtrs q = ptrs(p, const_cast<void*>(ws));
  if (rgbs) *rgbs = q.rgbs;
  if (drgbs) *drgbs = q.drgbs;
  if (ranges) *ranges = reinterpret_cast<const uint64_t*>(q.ranges);
  if (tile_last) *tile_last = q.tile_last;
  if (n_contrib) *n_contrib = q.ncontrib;
  if (ndup) *ndup = q.ndup;
  if (sorted_vals) *sorted_vals = q.vb;
  return SVR_OK;
}

int svr_batch_prepare(svr_batch_plan* p, void* ws, const int64_t* octree_paths, const float* vox_centers,
                      const float* vox_lengths, const void* sh0, const void* shs, int sh_bf16, int sh_degree, int M,
                      void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!p || !ws || !octree_paths || !vox_centers || !vox_lengths || !sh0 || sh_degree < 0 || sh_degree > 3 ||
      M - 1 < (sh_degree + 1) * (sh_degree + 1) - 1 || (M > 1 && !shs))
    return SVR_ERR_SHAPE;
  BatchPtrs q = ptrs(p, ws);
  const int P = (int)p->P;
  const size_t VP = (size_t)p->V * p->P;
  cudaMemsetAsync(q.header, 0, (kHeaderWords + (size_t)p->total_tiles) * sizeof(uint32_t), stream);
  const bool copied = p->binning && p->copies.n > 1;
  uint32_t* counts = p->binning ? (copied ? q.copies : q.counts) : nullptr;
  if (copied) cudaMemsetAsync(q.copies, 0, (size_t)p->copies.n * p->copies.stride * sizeof(uint32_t), stream);
  const dim3 pgrid((P + 127) / 128);
  const int level_low = (p->rank_bits == kRankBits) ? 0 : kRankBits - (p->rank_bits - 3);  // 3*(16-L)
  const int tight = p->culling < 0 ? !p->exact : p->culling;
#define SVR_PROJ_AS(D, TS, LAST)                                                                              \
  project_sh_kernel<D, TS, LAST><<<pgrid, 128, 0, stream>>>(                                                  \
      p->vt, P, vox_centers, vox_lengths, (const TS*)sh0, (const TS*)shs, M, octree_paths, level_low, tight,  \
      q.ndup, q.bbox, q.quad, q.rgbs, q.header + 1, coverage_words(q), counts,           \
      p->copies)
#define SVR_PROJ(D)                                                                                           \
  if (sh_bf16) {                                                                                              \
    if (p->V > 1) SVR_PROJ_AS(D, __nv_bfloat16, true);                                                        \
    else SVR_PROJ_AS(D, __nv_bfloat16, false);                                                                \
  } else {                                                                                                    \
    if (p->V > 1) SVR_PROJ_AS(D, float, true);                                                                \
    else SVR_PROJ_AS(D, float, false);                                                                        \
  }
  const dim3 grid((P + 255) / 256, p->V);
  switch (sh_degree) {
    case 0: SVR_PROJ(0) break;
    case 1: SVR_PROJ(1) break;
    case 2: SVR_PROJ(2) break;
    default: SVR_PROJ(3) break;
  }
#undef SVR_PROJ
#undef SVR_PROJ_AS
  // (counting alone, as capacity fitting does, needs no positions)
  if (p->cap > 0 && !svr_batch_plan_positions_ready(p, ws, octree_paths)) {
    // Rank positions of all (voxel, quadrant) pairs: one stable radix sort of
    // the 8P compressed ranks in the (still free) instance arrays.
    const size_t n8 = 8 * (size_t)P;
    rank_pos_keys_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, stream>>>(P, octree_paths, p->rank_bits, q.ka, q.va,
                                                                          q.header + 5);
    const int in_b = launch_radix_sort(q.ka, q.va, q.kb, q.vb, nullptr, q.header + 5, (uint32_t)n8, p->rank_bits,
                                       q.sort_tmp, stream);
    rank_pos_scatter_kernel<<<(unsigned)((n8 + 255) / 256), 256, 0, stream>>>(n8, in_b ? q.vb : q.va, q.rank_pos, q.val_of_pos);
    // The tables are there from now on, unless these launches failed or were only
    // recorded (a graph that is never replayed builds nothing).
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(stream, &capturing);
    p->pos_ready = capturing == cudaStreamCaptureStatusNone && cudaPeekAtLastError() == cudaSuccess;
    p->pos_paths = octree_paths;
    p->pos_ws = ws;
  }
  if (p->binning) {
    // Counting sort by tile: the projection's counts to ranges, every instance's
    // rank position scattered into its tile's range, each range sorted.
    uint32_t* keys = reinterpret_cast<uint32_t*>(q.ka);
    if (copied) launch_tile_copies(q.copies, (int)p->copies.n, p->copies.stride, (int)p->total_tiles, q.counts, stream);
    launch_tile_ranges_from_counts(q.counts, (int)p->total_tiles, (uint32_t)p->cap, q.ranges, q.header, q.header + 1,
                                   q.scan_tmp, q.sort_tmp, q.header + 6, stream);
    if (p->cap > 0) {
      scatter_positions_kernel<<<grid, 256, 0, stream>>>(p->vt, P, q.rank_pos, q.bbox, q.quad, q.ndup, counts,
                                                         p->copies, copied ? q.counts : nullptr, keys,
                                                         (uint32_t)p->cap, q.header + 1);
      launch_tile_sort(q.ranges, (int)p->total_tiles, keys, q.val_of_pos, q.vb, p->cap, q.sort_tmp, q.header + 6,
                       stream);
    }
    return check_last();
  }
  launch_scan_inclusive(q.ndup, q.scan, VP, q.scan_tmp, q.header, (unsigned long long)p->cap, q.header + 1, stream);
  cudaMemsetAsync(q.ranges, 0, (size_t)p->total_tiles * sizeof(uint2), stream);
  if (p->cap > 0) {
    // Two-level sort: LSD radix passes over the tile bits only put every
    // tile's instances together in generation order (ending in ka/va), then
    // one CTA per tile sorts its segment by the rank-position bits into kb/vb.
    uint32_t* segs = q.header + 16;
    group_segments_kernel<<<1, 64, 0, stream>>>(p->gt, P, q.scan, (uint32_t)p->cap, segs);
    const bool odd = (sort_passes(p->key_bits - kPosShift) & 1) != 0;
    uint64_t* k0 = odd ? q.kb : q.ka;
    uint32_t* v0 = odd ? q.vb : q.va;
    uint64_t* k1 = odd ? q.ka : q.kb;
    uint32_t* v1 = odd ? q.va : q.vb;
    duplicate_batch_kernel<<<grid, 256, 0, stream>>>(p->vt, P, q.rank_pos, q.bbox, q.quad, q.ndup, q.scan, k0, v0,
                                                     (uint32_t)p->cap, q.header + 1);
    for (int g = 0; g < p->gt.n; ++g) {
      launch_radix_sort(k0, v0, k1, v1, segs + 2 * g, segs + 2 * g + 1, (uint32_t)p->cap, p->key_bits,
                        q.sort_tmp, stream, kPosShift);
      const uint32_t g_tiles = (g + 1 < p->gt.n ? p->gt.tile_base[g + 1] : (uint32_t)p->total_tiles) -
                               p->gt.tile_base[g];
      launch_tile_ranges(q.ka, segs + 2 * g, segs + 2 * g + 1, (uint32_t)p->cap, kPosShift, p->gt.tile_base[g],
                         g_tiles, q.ranges, stream);
    }
    // the radix histograms in sort_tmp are dead here; the segment sort reuses it
    launch_tile_segment_sort(q.ranges, (int)p->total_tiles, q.ka, q.va, q.kb, q.vb, p->pos_bits, p->cap,
                             q.sort_tmp, stream, p->seg_small_n, p->seg_chunk);
  }
  return check_last();
}

// Compositing of all views with the densities either per voxel (geos) or
// as grid points read through the voxels' corner indices (va.key).
static int batch_render(svr_batch_plan* p, void* ws, VoxelArrays va, float* out_color, float* out_T,
                        cudaStream_t stream) {
  BatchPtrs q = ptrs(p, ws);
  va.bboxes = q.bbox;
  va.rgbs = q.rgbs;
  FwdTileOut out{q.tile_last, q.ncontrib, out_color, nullptr, nullptr, out_T, nullptr};
  const bool ordered = (p->order_flags & 1) != 0;
  if (ordered) build_tile_order(p, q, nullptr, q.order_fwd, q.header + 2, stream);
  else cudaMemsetAsync(q.header + 2, 0, sizeof(uint32_t), stream);
  launch_render_fwd_batch(p->vt, (int)p->total_tiles, q.ranges, p->cap > 0 ? q.vb : nullptr, va, (int)p->P,
                          (size_t)p->P * 3, out, p->n_samp, p->tile_size, p->stage, !p->exact, p->pair,
                          ordered ? q.order_fwd : nullptr, q.header + 2, p->fwd_ctas_per_sm, stream);
  return check_last();
}

static int batch_backward(svr_batch_plan* p, void* ws, VoxelArrays va, const float* out_T, const float* dL_dcolor,
                          const float* dL_dT, BwdTileOut out, cudaStream_t stream) {
  BatchPtrs q = ptrs(p, ws);
  cudaMemsetAsync(q.drgbs, 0, (size_t)p->V * p->P * 16, stream);
  va.bboxes = q.bbox;
  va.rgbs = q.rgbs;
  BwdTileIn in{out_T, q.ncontrib, dL_dcolor, nullptr, nullptr, dL_dT, nullptr, nullptr, 0.f, 0.f, 0.f};
  out.dL_drgbs = q.drgbs;
  out.err = q.header + 1;
  const bool ordered = (p->order_flags & 2) != 0;
  if (ordered) build_tile_order(p, q, q.tile_last, q.order_bwd, q.header + 3, stream);
  else cudaMemsetAsync(q.header + 3, 0, sizeof(uint32_t), stream);
  launch_render_bwd_batch(p->vt, (int)p->total_tiles, q.ranges, q.tile_last, p->cap > 0 ? q.vb : nullptr, va,
                          (int)p->P, (size_t)p->P * 3, (size_t)p->P * 4, in, out, p->n_samp, p->tile_size,
                          p->stage_bwd, !p->exact, p->pair_bwd < 0 ? p->pair : p->pair_bwd, p->adaptive != 0,
                          CoverageCount{coverage_words(q), q.header}, ordered ? q.order_bwd : nullptr, q.header + 3,
                          p->bwd_ctas_per_sm, stream);
  return check_last();
}

int svr_batch_render(svr_batch_plan* p, void* ws, const float* vox_centers, const float* vox_lengths,
                     const void* geos, int geos_bf16, float* out_color, float* out_T, void* stream_) {
  if (!p || !ws || !vox_centers || !vox_lengths || !geos || !out_color || !out_T) return SVR_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(geos) & 15u) != 0) return SVR_ERR_ALIGN;
  VoxelArrays va{nullptr, vox_centers, vox_lengths, geos_bf16 ? nullptr : (const float*)geos,
                 geos_bf16 ? (const __nv_bfloat16*)geos : nullptr, nullptr};
  return batch_render(p, ws, va, out_color, out_T, static_cast<cudaStream_t>(stream_));
}

int svr_batch_render_grid(svr_batch_plan* p, void* ws, const float* vox_centers, const float* vox_lengths,
                          const int64_t* vox_key, const void* grid, int grid_bf16, float* out_color, float* out_T,
                          void* stream_) {
  if (!p || !ws || !vox_centers || !vox_lengths || !vox_key || !grid || !out_color || !out_T) return SVR_ERR_SHAPE;
  VoxelArrays va{nullptr, vox_centers, vox_lengths, nullptr, nullptr, nullptr};
  va.key = vox_key;
  va.grid = grid_bf16 ? nullptr : (const float*)grid;
  va.grid_bf16 = grid_bf16 ? (const __nv_bfloat16*)grid : nullptr;
  return batch_render(p, ws, va, out_color, out_T, static_cast<cudaStream_t>(stream_));
}

int svr_batch_backward(svr_batch_plan* p, void* ws, const float* vox_centers, const float* vox_lengths,
                       const void* geos, int geos_bf16, const float* out_T, const float* dL_dcolor,
                       const float* dL_dT, float* dL_dgeos, void* stream_) {
  if (!p || !ws || !vox_centers || !vox_lengths || !geos || !out_T || !dL_dcolor || !dL_dT || !dL_dgeos)
    return SVR_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(geos) & 15u) != 0 || (reinterpret_cast<uintptr_t>(dL_dgeos) & 15u) != 0)
    return SVR_ERR_ALIGN;
  VoxelArrays va{nullptr, vox_centers, vox_lengths, geos_bf16 ? nullptr : (const float*)geos,
                 geos_bf16 ? (const __nv_bfloat16*)geos : nullptr, nullptr};
  BwdTileOut out{dL_dgeos, nullptr, nullptr, nullptr, 1};
  return batch_backward(p, ws, va, out_T, dL_dcolor, dL_dT, out, static_cast<cudaStream_t>(stream_));
}

int svr_batch_backward_grid(svr_batch_plan* p, void* ws, const float* vox_centers, const float* vox_lengths,
                            const int64_t* vox_key, const void* grid, int grid_bf16, const float* out_T,
                            const float* dL_dcolor, const float* dL_dT, float* dL_dgrid, void* stream_) {
  if (!p || !ws || !vox_centers || !vox_lengths || !vox_key || !grid || !out_T || !dL_dcolor || !dL_dT || !dL_dgrid)
    return SVR_ERR_SHAPE;
  VoxelArrays va{nullptr, vox_centers, vox_lengths, nullptr, nullptr, nullptr};
  va.key = vox_key;
  va.grid = grid_bf16 ? nullptr : (const float*)grid;
  va.grid_bf16 = grid_bf16 ? (const __nv_bfloat16*)grid : nullptr;
  BwdTileOut out{nullptr, nullptr, nullptr, nullptr, 0};
  out.key = vox_key;
  out.grid_grad = dL_dgrid;
  return batch_backward(p, ws, va, out_T, dL_dcolor, dL_dT, out, static_cast<cudaStream_t>(stream_));
}

int svr_batch_sh_backward_as(svr_batch_plan* p, void* ws, const float* vox_centers, int sh_degree, int M, void* dL_dsh0,
                             void* dL_dshs, int out_bf16, float* subdiv, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!p || !ws || !vox_centers || !dL_dsh0 || sh_degree < 0 || sh_degree > 3 ||
      M - 1 < (sh_degree + 1) * (sh_degree + 1) - 1 || (M > 1 && !dL_dshs))
    return SVR_ERR_SHAPE;
  if (out_bf16 && ((reinterpret_cast<uintptr_t>(dL_dsh0) | reinterpret_cast<uintptr_t>(dL_dshs)) & 3u) != 0)
    return SVR_ERR_ALIGN;
  BatchPtrs q = ptrs(p, ws);
  const int P = (int)p->P;
  const int g = (P + kShBwThreads - 1) / kShBwThreads;
  const size_t smem = (size_t)kShBwThreads * (3 + 3 * (M - 1)) * sizeof(float);
  if (smem > 48 * 1024) return SVR_ERR_SHAPE;  // M <= 32 coefficients per channel
  const float4* d4 = reinterpret_cast<const float4*>(q.drgbs);
  const auto run = [&](auto f32, auto b16) {
    if (out_bf16)
      b16<<<g, kShBwThreads, smem, stream>>>(p->vt, P, M, vox_centers, d4, static_cast<__nv_bfloat16*>(dL_dsh0),
                                             static_cast<__nv_bfloat16*>(dL_dshs), subdiv);
    else
      f32<<<g, kShBwThreads, smem, stream>>>(p->vt, P, M, vox_centers, d4, static_cast<float*>(dL_dsh0),
                                             static_cast<float*>(dL_dshs), subdiv);
  };
  switch (sh_degree) {
    case 0: run(sh_bw_batch_kernel<0, float>, sh_bw_batch_kernel<0, __nv_bfloat16>); break;
    case 1: run(sh_bw_batch_kernel<1, float>, sh_bw_batch_kernel<1, __nv_bfloat16>); break;
    case 2: run(sh_bw_batch_kernel<2, float>, sh_bw_batch_kernel<2, __nv_bfloat16>); break;
    default: run(sh_bw_batch_kernel<3, float>, sh_bw_batch_kernel<3, __nv_bfloat16>); break;
  }
  return check_last();
}

int svr_batch_sh_backward(svr_batch_plan* p, void* ws, const float* vox_centers, int sh_degree, int M,
                          float* dL_dsh0, float* dL_dshs, float* subdiv, void* stream) {
  return svr_batch_sh_backward_as(p, ws, vox_centers, sh_degree, M, dL_dsh0, dL_dshs, 0, subdiv, stream);
}

}  // extern "C"
