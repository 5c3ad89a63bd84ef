// Binning of octrees 21 levels deep (the reference's new_cuda backend,
// backends/new_cuda/src/config.h:16,24-34 and forward.cu:660-752).
//
// The Morton rank then takes 3 * 21 = 63 bits, so a (tile, rank) key no
// longer fits in 64 bits; the reference sorts 128-bit keys
// (auxiliary.h:17-25,66-87).  Here the same order comes from the 16-level path's
// two levels: a stable LSD radix sort of the instances by tile, carrying their
// generation index, then the stable sort of every tile's segment by the 63 rank
// bits.  Equal (tile, rank) pairs keep generation order -- exactly what one
// stable sort of the wide key gives.  Sorting all instances by rank first, in seven
// radix passes, and then stably by tile gives it too, in a time that does not depend on
// how long the tiles' lists are: 300k voxels, 801x601, all of binning 158 us where 77 are
// taken; 2M voxels on 144 tiles (15,000 instances each) 409 and 380 us, on 64 (33,000) 403
// and 449; 20M on 256 tiles (82,000) 4.23 and 4.54 ms, on 16 (1.3M) 4.1 and 6.5, on one
// 4.0 and 36.  So lists that are long on average are sorted by rank first.
// The wide keys (as lo = tile << 63 | rank, hi = tile >> 1, the reference's
// SortKey128 halves), the sorted values and the tile ranges are left where the
// 16-level path leaves its own, so compositing and its backward read them
// unchanged.
#include "svr_common.cuh"
#include "svr_kernels.h"

namespace svr {

__host__ __device__ constexpr uint64_t octant_repeat_deep(uint64_t q) {
  uint64_t v = 0;
  for (int l = 0; l < kDeepLevels; ++l) v = (v << 3) | q;
  return v;
}

constexpr uint32_t kLongLists = 1u << 15;  // instances per tile on average

// One (tile, index) pair per instance in generation order (forward.cu:518-571
// of new_cuda, with the instance's own index as the carried value), plus the
// instance's rank and sort value by index.  BY_RANK: (rank, index) pairs, and the
// tile by index.
template <bool BY_RANK>
__global__ void __launch_bounds__(256)
duplicate_deep_kernel(const __grid_constant__ ViewParams vp, int P, const int64_t* __restrict__ octpaths,
                      const uint2* __restrict__ bboxes, const uint32_t* __restrict__ quads,
                      const uint32_t* __restrict__ ndup, const uint32_t* __restrict__ scan,
                      uint64_t* __restrict__ sort_keys, uint32_t* __restrict__ sort_idx,
                      uint64_t* __restrict__ rank_of, uint32_t* __restrict__ tile_of, uint32_t* __restrict__ val_of,
                      uint32_t cap, uint32_t* __restrict__ err) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= P) return;
  const uint32_t n = ndup[idx];
  if (n == 0) return;
  const uint32_t end = scan[idx];
  uint32_t off = end - n;
  if (end > cap) atomicOr(err, SVR_DEVERR_CAPACITY);
  const uint32_t wend = min(end, cap);
  if ((uint32_t)idx >= (1u << kVoxIdBits)) {
    atomicOr(err, SVR_DEVERR_VOXID);
    return;
  }
  int tx0, ty0, tx1, ty1;
  bbox_tile_rect(bboxes[idx], vp.grid_x, vp.grid_y, vp.tile_shift, tx0, ty0, tx1, ty1);
  const uint64_t path = (uint64_t)octpaths[idx];
  const uint32_t qb = quads[idx];
  for (uint32_t q = 0; q < 8; ++q) {
    if (!(qb & (1u << q))) continue;
    const uint64_t rank = path ^ octant_repeat_deep(q);
    const uint32_t val = make_sort_val((uint32_t)idx, q);
    for (int y = ty0; y <= ty1; ++y) {
      for (int x = tx0; x <= tx1; ++x) {
        if (off < wend) {
          const uint32_t tile = (uint32_t)(y * vp.grid_x + x);
          sort_keys[off] = BY_RANK ? rank : tile;
          if (BY_RANK) tile_of[off] = tile;
          sort_idx[off] = off;
          rank_of[off] = rank;
          val_of[off] = val;
        }
        ++off;
      }
    }
  }
  if (off != end) atomicOr(err, SVR_DEVERR_DUP_MISMATCH);
}

// The tile-sorted instances' keys (the tile's lowest bit above the rank, as the
// wide key's low half has it) and values, and the wide keys' high halves: a
// segment sort by rank does not move an instance out of its tile.
__global__ void deep_segment_keys_kernel(uint32_t n, const uint32_t* __restrict__ d_n,
                                         const uint64_t* __restrict__ tiles, const uint32_t* __restrict__ idx,
                                         const uint64_t* __restrict__ rank_of, const uint32_t* __restrict__ val_of,
                                         uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                         uint64_t* __restrict__ keys_hi) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= min(n, *d_n)) return;
  const uint64_t tile = tiles[i];
  const uint32_t k = idx[i];
  keys[i] = (tile << kDeepRankBits) | rank_of[k];
  vals[i] = val_of[k];
  keys_hi[i] = tile >> (64 - kDeepRankBits);
}

// The rank-sorted indices keyed by their tile, for the stable sort by tile.
__global__ void deep_tile_keys_kernel(uint32_t n, const uint32_t* __restrict__ d_n, const uint32_t* __restrict__ idx,
                                      const uint32_t* __restrict__ tile_of, uint64_t* __restrict__ keys,
                                      uint32_t* __restrict__ vals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= min(n, *d_n)) return;
  const uint32_t k = idx[i];
  keys[i] = tile_of[k];
  vals[i] = k;
}

// Wide keys and values from the (tile, index) pairs in their final order (may run in
// place: every thread reads its own place before writing it).
__global__ void deep_finalize_kernel(uint32_t n, const uint32_t* __restrict__ d_n, const uint64_t* tiles,
                                     const uint32_t* idx, const uint64_t* __restrict__ rank_of,
                                     const uint32_t* __restrict__ val_of, uint64_t* keys, uint32_t* vals,
                                     uint64_t* __restrict__ keys_hi) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= min(n, *d_n)) return;
  const uint64_t tile = tiles[i];
  const uint32_t k = idx[i];
  keys[i] = (tile << kDeepRankBits) | rank_of[k];
  vals[i] = val_of[k];
  keys_hi[i] = tile >> (64 - kDeepRankBits);
}

void launch_binning_deep(const ViewParams& vp, int P, const int64_t* octpaths, const uint2* bboxes,
                         const uint32_t* quads, const uint32_t* ndup, const uint32_t* scan, const uint32_t* d_n,
                         uint32_t n, const DeepBinning& b, uint2* ranges, uint32_t* err, cudaStream_t stream) {
  if (P <= 0 || n == 0) return;
  const uint32_t n_tiles = (uint32_t)vp.grid_x * (uint32_t)vp.grid_y;
  int tile_bits = 0;
  while (tile_bits < 32 && ((n_tiles - 1) >> tile_bits)) ++tile_bits;
  tile_bits = std::max(tile_bits, 1);
  const unsigned g = (n + 255) / 256;
  if (n / n_tiles >= kLongLists) {
    uint32_t* tile_of = reinterpret_cast<uint32_t*>(b.keys_hi);  // (written last)
    uint64_t* k[2] = {b.keys_a, b.keys_b};
    uint32_t* v[2] = {b.vals_a, b.vals_b};
    duplicate_deep_kernel<true><<<(P + 255) / 256, 256, 0, stream>>>(vp, P, octpaths, bboxes, quads, ndup, scan, k[0],
                                                                    v[0], b.rank_of, tile_of, b.val_of, n, err);
    const int r1 = launch_radix_sort(k[0], v[0], k[1], v[1], nullptr, d_n, n, kDeepRankBits, b.sort_temp, stream);
    deep_tile_keys_kernel<<<g, 256, 0, stream>>>(n, d_n, v[r1], tile_of, k[1 - r1], v[1 - r1]);
    const int r2 = launch_radix_sort(k[1 - r1], v[1 - r1], k[r1], v[r1], nullptr, d_n, n, tile_bits, b.sort_temp,
                                     stream);
    const int fin = r2 ? r1 : 1 - r1;  // the pair holding (tile, index)
    launch_tile_ranges(k[fin], nullptr, d_n, n, 0, 0u, n_tiles, ranges, stream);
    deep_finalize_kernel<<<g, 256, 0, stream>>>(n, d_n, k[fin], v[fin], b.rank_of, b.val_of, b.keys_b, b.vals_b,
                                                b.keys_hi);
    return;
  }
  // the radix passes end in (keys_b, vals_b), the segment keys go to (keys_a,
  // vals_a) and the sorted segments back
  const bool odd = (sort_passes(tile_bits) & 1) != 0;
  uint64_t *k0 = odd ? b.keys_a : b.keys_b, *k1 = odd ? b.keys_b : b.keys_a;
  uint32_t *v0 = odd ? b.vals_a : b.vals_b, *v1 = odd ? b.vals_b : b.vals_a;
  duplicate_deep_kernel<false><<<(P + 255) / 256, 256, 0, stream>>>(vp, P, octpaths, bboxes, quads, ndup, scan, k0, v0,
                                                                   b.rank_of, nullptr, b.val_of, n, err);
  launch_radix_sort(k0, v0, k1, v1, nullptr, d_n, n, tile_bits, b.sort_temp, stream);
  launch_tile_ranges(b.keys_b, nullptr, d_n, n, 0, 0u, n_tiles, ranges, stream);
  deep_segment_keys_kernel<<<g, 256, 0, stream>>>(n, d_n, b.keys_b, b.vals_b, b.rank_of, b.val_of, b.keys_a, b.vals_a,
                                                 b.keys_hi);
  launch_tile_segment_sort(ranges, (int)n_tiles, b.keys_a, b.vals_a, b.keys_b, b.vals_b, kDeepRankBits, n,
                           b.sort_temp, stream);
}

}  // namespace svr
