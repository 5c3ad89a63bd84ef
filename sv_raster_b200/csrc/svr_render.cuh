// Per-tile compositing shared by the forward and backward kernels.
//
// A CTA of TS*TS threads owns one TSxTS pixel tile (16x16 on the plain path,
// as the reference); each warp owns an 8x4 micro-tile (forward.cu:77-92).
// Voxel instances of the tile's sorted list are staged into shared memory in
// batches of SB records (structure of arrays, vector loads where the layout
// allows), then every warp builds a
// ballot mask of the staged records whose packed bbox overlaps its 8x4
// micro-tile and whose camera quadrant matches a ray quadrant present in the
// warp.  Lanes walk only those records, in list order, so every pixel sees
// exactly the records the reference's per-pixel loop would accept
// (forward.cu:182-200), in the same order, with the same arithmetic.
#pragma once

#include <cuda_bf16.h>
#include <math_constants.h>

#include "svr_block.cuh"
#include "svr_common.cuh"
#include "svr_views.cuh"

namespace svr {

// Tile geometry and staging depth of a compositing kernel: TS x TS pixel
// tiles (TS = 8, 16 or 32), one thread per pixel, warps laid out row-major as
// 8x4 micro-tiles, SB records staged per round.
template <int TS_, int SB_>
struct TileCfg {
  static constexpr int TS = TS_;
  static constexpr int NT = TS * TS;      // threads per CTA
  static constexpr int NW = NT / 32;      // warps per CTA
  static constexpr int MX = TS / 8;       // micro-tiles per tile row
  static constexpr int SB = SB_;          // records staged per round
  static constexpr int GROUPS = SB / 32;  // 32-record ballot groups per round
  static_assert(TS == 8 || TS == 16 || TS == 32, "tile size");
  static_assert(SB % 32 == 0 && SB >= 32, "staging depth");
};
// The plain path keeps the reference's 16x16 tile lists (config.h:14-15)
// and composites each with four 8x8 CTAs that share the list.
using PlainTile = TileCfg<8, 64>;
constexpr int kPlainSub = 4;  // 8x8 CTAs per 16x16 list
static_assert(PlainTile::SB <= PlainTile::NT, "ListReader stages one record per thread, and its ring holds two rounds");

// Resident CTAs per SM the compositing kernels are register-bounded for at
// 256 threads; other CTA sizes keep the same threads per SM.  The forward's was
// chosen by measurement on the c4 step at 8x8 tiles: 3 / 4 / 5 / 6 gave 15.0 /
// 13.9 / 14.4 / 14.9 ms.
constexpr int kFwdMinBlocks = 4;
constexpr int kBwdMinBlocks = 3;
template <class CFG>
constexpr int fwd_min_blocks() { return CFG::NT >= 1024 ? 1 : kFwdMinBlocks * 256 / CFG::NT; }
// The one-pixel backward: its CTAs of 64 threads run 14 (32 staged records) or 12 (64)
// to an SM, which the bounds of 13 and 11 come to: the compiler rounds to 72 and 80
// registers.  Nothing spills with one sample and fast arithmetic; the plain forms spill
// 20 to 136 bytes but for the simplest (16 CTAs at 64 registers: the plain backward 1.69
// -> 2.08 ms on a 2M-voxel view).
template <class CFG>
constexpr int bwd_min_blocks() {
  return CFG::NT >= 1024 ? 1 : (CFG::NT == 64 ? (CFG::SB <= 32 ? 13 : 11) : kBwdMinBlocks * 256 / CFG::NT);
}

// Pixel of thread `tid` inside its tile: warp w owns micro-tile
// (w % MX, w / MX) of 8x4 pixels, lanes row-major inside it.
template <class CFG>
__device__ __forceinline__ void tile_pixel_of(int tid, int& lx, int& ly) {
  const int warp = tid >> 5, lane = tid & 31;
  lx = (warp % CFG::MX) * 8 + (lane & 7);
  ly = (warp / CFG::MX) * 4 + (lane >> 3);
}

// Voxel attributes of one view as the kernels read them.
struct VoxelArrays {
  const uint2* bboxes;        // [P] packed pixel bbox (this view)
  const float* centers;       // [P,3]
  const float* lengths;       // [P]
  const float* geos;          // [P,8] fp32, or nullptr when geos_bf16 is set
  const __nv_bfloat16* geos_bf16;  // [P,8] bf16 storage
  const float* rgbs;          // [P,3] (this view)
  // Grid-point densities (batched grid entry points): when key is set, corner
  // c of voxel v is grid[key[8 v + c]] (fp32 grid, or grid_bf16), read while
  // staging the record, and geos / geos_bf16 are unused.
  const int64_t* key = nullptr;
  const float* grid = nullptr;
  const __nv_bfloat16* grid_bf16 = nullptr;
};

// One staged record where lanes each read a record of their own (the forward,
// and the backward with one pixel per thread).  Per-record terms of the slab
// test and of the sample position are computed once here instead of once per
// pixel, by the same IEEE operations on the same operands, so the per-pixel
// results are unchanged bit for bit.  32 lanes on different records make a
// 16-byte read cost 3.9 wavefronts on average, and wavefronts bound the forward
// next to instruction issue (143 M of them and 638 M instructions in 196 M SM
// cycles for 5.6 M instances): so a record is five 16-byte words to read, and
// the two planes of each slab are formed per lane from (c - o, l/2).
template <int SB>
struct FwdStage {
  uint4 box[SB];      // xmin, xmax - xmin, ymin, (ymax - ymin) | quadrant << 16
  float4 rel[SB];     // c - o (xyz), l/2 (w)
  float4 corner[SB];  // c - l/2 (xyz), 1/l (w)
  float4 geo[SB][2];  // 8 corner densities, or their polynomial (fast arithmetic)
  float4 rgb[SB];     // rgb (xyz), voxel id as int bits (w)
};

// One staged record of the two-pixel backward, whose lanes all read the same
// record (one wavefront per word): the slab's planes are staged in the order
// in which rays of the record's octant cross them.
template <int SB>
struct BwdStage {
  uint4 box[SB];      // as in FwdStage
  float4 near[SB];    // (c - o) -/+ l/2 (xyz), the plane crossed first; 1/l (w)
  float4 far[SB];     // (c - o) +/- l/2 (xyz), the other
  float4 corner[SB];  // c - l/2 (xyz), voxel id as int bits (w)
  float4 geo[SB][2];  // 8 corner densities, or their polynomial (fast arithmetic)
  float4 rgb[SB];     // rgb (xyz)
};

// The trilinear interpolant of 8 corner densities as a polynomial in the
// place (x, y, z) in the unit cube: (1, z, y, yz) then (x, xz, xy, xyz).  Seven
// multiply-adds evaluate it (trilinear_poly), against fifteen multiplies for
// the corner weights and eight multiply-adds over them; 12 subtractions per
// staged record set it up.
__device__ __forceinline__ void trilinear_coefficients(const float g[8], float4& lo, float4& hi) {
  const float z0 = g[1] - g[0], z1 = g[3] - g[2], z2 = g[5] - g[4], z3 = g[7] - g[6];
  lo = make_float4(g[0], z0, g[2] - g[0], z1 - z0);
  hi = make_float4(g[4] - g[0], z2 - z0, (g[6] - g[4]) - (g[2] - g[0]), (z3 - z2) - (z1 - z0));
}
// The polynomial of densities as they come.  Its coefficients are differences of
// corners, which infinities turn into NaN (an opaque voxel, and NaN gradients) and
// corners past half the largest float into infinities; and next to a corner at
// -1e8 and below the ordinary ones vanish in their rounding.  Such records, seldom
// met, get coefficients that evaluate as the corners weighted one by one do:
//   - an infinite (or NaN) corner makes the density that everywhere inside;
//   - so does a corner that is lower than the others by more than rounding keeps:
//     the interpolant is far below zero except next to the voxel's far end, in less
//     than rounding resolves (corners masked with a type's lowest value);
//   - others are clamped to where differences of differences still fit: only their
//     sign matters.
constexpr float kWideDensity = 1e8f, kHugeDensity = 1e37f;
__device__ __forceinline__ void density_polynomial(float g[8], float4& lo, float4& hi) {
  float top = 0.f;
#pragma unroll
  for (int c = 0; c < 8; ++c) top = fmaxf(top, fabsf(g[c]));
  if (top >= kWideDensity) {
    float least = g[0], most = g[0], endless = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      least = fminf(least, g[c]);
      most = fmaxf(most, g[c]);
      if (!(fabsf(g[c]) < CUDART_INF_F)) endless += g[c];
    }
    const bool empty = least < -kWideDensity * fmaxf(1.f, most);
    if (endless != 0.f || empty) {
      lo = make_float4(endless != 0.f ? endless : -CUDART_INF_F, 0.f, 0.f, 0.f);
      hi = make_float4(0.f, 0.f, 0.f, 0.f);
      return;
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) g[c] = fminf(fmaxf(g[c], -kHugeDensity), kHugeDensity);
  }
  trilinear_coefficients(g, lo, hi);
}
__device__ __forceinline__ float trilinear_poly(const float4& lo, const float4& hi, float qx, float qy, float qz) {
  const float a = fmaf(lo.y, qz, lo.x), b = fmaf(lo.w, qz, lo.z);
  const float c = fmaf(hi.y, qz, hi.x), d = fmaf(hi.w, qz, hi.z);
  return fmaf(fmaf(d, qy, c), qx, fmaf(b, qy, a));
}

// MAYBE_GRID = false compiles the grid-point read out (kernels instantiated
// apart for the per-voxel densities).
template <bool MAYBE_GRID>
__device__ __forceinline__ void read_densities(const VoxelArrays& va, uint32_t vid, float g[8]) {
  if (MAYBE_GRID && va.key) {
    const int64_t* k = va.key + 8 * (size_t)vid;
#pragma unroll
    for (int c = 0; c < 8; ++c) g[c] = va.grid_bf16 ? __bfloat162float(va.grid_bf16[k[c]]) : va.grid[k[c]];
  } else if (va.geos_bf16) {
    const uint4 raw = *reinterpret_cast<const uint4*>(va.geos_bf16 + 8 * (size_t)vid);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 f = __bfloat1622float2(h[c]);
      g[2 * c] = f.x;
      g[2 * c + 1] = f.y;
    }
  } else {
    const float4* p = reinterpret_cast<const float4*>(va.geos + 8 * (size_t)vid);
    const float4 a = p[0], b = p[1];
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
    g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
  }
}

template <bool FAST, bool MAYBE_GRID, int SB>
__device__ __forceinline__ void stage_record(FwdStage<SB>& s, int slot, uint32_t val, const VoxelArrays& va, float ox,
                                             float oy, float oz) {
  const uint32_t vid = val_vox_id(val);
  const uint2 bb = va.bboxes[vid];
  s.box[slot] = make_uint4(bb_xmin(bb), bb_xmax(bb) - bb_xmin(bb), bb_ymin(bb),
                           (bb_ymax(bb) - bb_ymin(bb)) | (val_quadrant(val) << 16));
  const float* c = va.centers + 3 * (size_t)vid;
  const float cx = c[0], cy = c[1], cz = c[2], len = va.lengths[vid];
  const float rad = 0.5f * len;
  s.rel[slot] = make_float4(cx - ox, cy - oy, cz - oz, rad);
  s.corner[slot] = make_float4(cx - rad, cy - rad, cz - rad, 1.f / len);
  float g[8];
  read_densities<MAYBE_GRID>(va, vid, g);
  const float* rgb = va.rgbs + 3 * (size_t)vid;
  const float red = rgb[0], green = rgb[1], blue = rgb[2];  // (under way before the densities are looked at)
  if (FAST) {
    density_polynomial(g, s.geo[slot][0], s.geo[slot][1]);
  } else {
    s.geo[slot][0] = make_float4(g[0], g[1], g[2], g[3]);
    s.geo[slot][1] = make_float4(g[4], g[5], g[6], g[7]);
  }
  s.rgb[slot] = make_float4(red, green, blue, __int_as_float((int)vid));
}

template <bool FAST, bool MAYBE_GRID, int SB>
__device__ __forceinline__ void stage_record(BwdStage<SB>& s, int slot, uint32_t val, const VoxelArrays& va, float ox,
                                             float oy, float oz) {
  const uint32_t vid = val_vox_id(val), quad = val_quadrant(val);
  const uint2 bb = va.bboxes[vid];
  s.box[slot] = make_uint4(bb_xmin(bb), bb_xmax(bb) - bb_xmin(bb), bb_ymin(bb),
                           (bb_ymax(bb) - bb_ymin(bb)) | (quad << 16));
  const float* c = va.centers + 3 * (size_t)vid;
  const float cx = c[0], cy = c[1], cz = c[2], len = va.lengths[vid];
  const float rad = 0.5f * len;
  const float sx = (quad & 4u) ? -rad : rad, sy = (quad & 2u) ? -rad : rad, sz = (quad & 1u) ? -rad : rad;
  const float dx = cx - ox, dy = cy - oy, dz = cz - oz;
  s.near[slot] = make_float4(dx - sx, dy - sy, dz - sz, 1.f / len);
  s.far[slot] = make_float4(dx + sx, dy + sy, dz + sz, 0.f);
  s.corner[slot] = make_float4(cx - rad, cy - rad, cz - rad, __int_as_float((int)vid));
  float g[8];
  read_densities<MAYBE_GRID>(va, vid, g);
  const float* rgb = va.rgbs + 3 * (size_t)vid;
  const float red = rgb[0], green = rgb[1], blue = rgb[2];  // (under way before the densities are looked at)
  if (FAST) {
    density_polynomial(g, s.geo[slot][0], s.geo[slot][1]);
  } else {
    s.geo[slot][0] = make_float4(g[0], g[1], g[2], g[3]);
    s.geo[slot][1] = make_float4(g[4], g[5], g[6], g[7]);
  }
  s.rgb[slot] = make_float4(red, green, blue, 0.f);
}

// A plain CTA composites an 8x8 block but walks the list of the 16x16 tile
// around it, most of whose records do not reach the block.  The list is read
// NT entries at a time (value and bbox only, the next entries fetched while
// the staged ones are composited); entries that reach the block wait in a ring
// with their list positions until a round of them can be staged.
template <class CFG>
struct ListFilter {
  uint2 ring[2 * CFG::NT];      // value, list position (from the walk's end of the list)
  uint32_t hits[2][CFG::NW];    // per warp, alternating between chunks
  uint32_t pos[CFG::SB];        // list positions of the staged records
};

// BACK: entries from the end of the range.  All members are uniform over the
// CTA but the fetched entry.
template <class CFG, bool BACK>
struct ListReader {
  uint2 range;
  int total, next, head, tail, flip;
  uint32_t bx0, by0;
  uint32_t val;
  uint2 bb;
  bool got;

  __device__ __forceinline__ void fetch(const uint32_t* __restrict__ vals, const VoxelArrays& va) {
    const int i = next + (int)threadIdx.x;
    got = i < total;
    if (got) {
      val = vals[BACK ? range.y - 1 - i : range.x + i];
      bb = va.bboxes[val_vox_id(val)];
    }
  }
  __device__ __forceinline__ void init(uint2 r, int tile_x, int tile_y, const uint32_t* __restrict__ vals,
                                       const VoxelArrays& va) {
    range = r;
    total = (int)(r.y - r.x);
    next = head = tail = flip = 0;
    bx0 = tile_x * CFG::TS;
    by0 = tile_y * CFG::TS;
    fetch(vals, va);
  }
  // Next round of records (0: the list is through), left in ring entries
  // [head - n, head).  Called by the whole CTA.
  __device__ __forceinline__ int round(ListFilter<CFG>& f, const uint32_t* __restrict__ vals, const VoxelArrays& va) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    while (tail - head < CFG::SB && next < total) {
      const bool hit = got && bb_xmin(bb) <= bx0 + (CFG::TS - 1) && bb_xmax(bb) >= bx0 &&
                       bb_ymin(bb) <= by0 + (CFG::TS - 1) && bb_ymax(bb) >= by0;
      const uint32_t m = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) f.hits[flip][warp] = __popc(m);
      const uint32_t v = val;
      const int i = next + (int)threadIdx.x;
      next += CFG::NT;
      fetch(vals, va);
      __syncthreads();
      int at = tail;
#pragma unroll
      for (int w = 0; w < CFG::NW; ++w) {
        const int c = (int)f.hits[flip][w];
        if (w < warp) at += c;
        tail += c;
      }
      if (hit) f.ring[(at + __popc(m & lanemask_lt())) & (2 * CFG::NT - 1)] = make_uint2(v, (uint32_t)i);
      flip ^= 1;
    }
    __syncthreads();
    const int n = min(CFG::SB, tail - head);
    head += n;
    return n;
  }
  __device__ __forceinline__ uint2 entry(const ListFilter<CFG>& f, int n, int i) const {
    return f.ring[(head - n + i) & (2 * CFG::NT - 1)];
  }
};

// Slab test (auxiliary.h:240-253) of a ray of the record's octant: the octant
// says which plane of each slab comes first, so no minima of the two are
// needed.  A ray in a slab's plane (0 * inf) gives NaN, which fails a <= b: it
// misses, as with the minima.  Here and below x and y share an instruction where
// both need the same operation (the forward of eight full-HD views: 6.34 -> 6.17
// ms; the bits are the same).
__device__ __forceinline__ float2 octant_ray_box(const float4& rel, const PixelRay& r) {
  const float2 half = make_float2(rel.w, rel.w), at = make_float2(rel.x, rel.y), inv = make_float2(r.ix, r.iy);
  const float2 nr = mul2(fma2(make_float2(-r.sx, -r.sy), half, at), inv);
  const float2 fr = mul2(fma2(make_float2(r.sx, r.sy), half, at), inv);
  return make_float2(max3_nan(nr.x, nr.y, fmaf(-r.sz, rel.w, rel.z) * r.iz),
                     min3_nan(fr.x, fr.y, fmaf(r.sz, rel.w, rel.z) * r.iz));
}

// The same from the two planes staged in crossing order.
__device__ __forceinline__ float2 near_far_ray_box(const float4& nr, const float4& fr, const PixelRay& r) {
  const float2 inv = make_float2(r.ix, r.iy);
  const float2 n2 = mul2(make_float2(nr.x, nr.y), inv), f2 = mul2(make_float2(fr.x, fr.y), inv);
  return make_float2(max3_nan(n2.x, n2.y, nr.z * r.iz), min3_nan(f2.x, f2.y, fr.z * r.iz));
}

// Place in the unit cube of the point at t, from the voxel's corner (xyz) and 1/l.
__device__ __forceinline__ void place_in_voxel(const PixelRay& r, float t, const float4& corner, float inv_l, float& qx,
                                               float& qy, float& qz) {
  const float2 at = fma2(make_float2(t, t), make_float2(r.dx, r.dy), make_float2(r.ox, r.oy));
  const float2 q = mul2(add2(at, make_float2(-corner.x, -corner.y)), make_float2(inv_l, inv_l));
  qx = q.x;
  qy = q.y;
  qz = (fmaf(t, r.dz, r.oz) - corner.z) * inv_l;
}

// Fast arithmetic: exp(-optical depth) of a segment from its samples' summed
// activations.  The backward divides T by 1 - alpha, which for an opaque voxel
// keeps few digits, so both passes call this: from the same ray they arrive at the
// same alpha bit for bit (make_pixel_ray says how far their rays agree).
__device__ __forceinline__ float fast_transmittance(float step_sz, float act_sum) {
  return ex2_approx((-kStepScale * kLog2E * step_sz) * act_sum);
}

// Transmittance exp(-optical depth) of the ray segment [a, b] through staged
// record j (forward.cu:228-248): midpoint samples of the activated trilinear
// density.  local_alpha (or nullptr) receives each sample's own opacity.
template <int NS, bool FAST, int SB>
__device__ __forceinline__ float record_transmittance(const FwdStage<SB>& s, int j, const PixelRay& ray, float a,
                                                      float b, float* local_alpha) {
  const float4 cr = s.corner[j], glo = s.geo[j][0], ghi = s.geo[j][1];
  float vol_int = 0.f;
  const float vox_l_inv = cr.w;
  const float step_sz = (b - a) * (1.f / NS);
  const float stx = step_sz * ray.dx, sty = step_sz * ray.dy, stz = step_sz * ray.dz;
  const float t0 = a + 0.5f * step_sz;
  float qx, qy, qz;
  place_in_voxel(ray, t0, cr, vox_l_inv, qx, qy, qz);
  const float qsx = stx * vox_l_inv, qsy = sty * vox_l_inv, qsz = stz * vox_l_inv;
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    if (FAST) {
      vol_int += density_act_f<true>(trilinear_poly(glo, ghi, qx, qy, qz));
    } else {
      const float geo[8] = {glo.x, glo.y, glo.z, glo.w, ghi.x, ghi.y, ghi.z, ghi.w};
      float w[8];
      trilinear_weights(qx, qy, qz, w);
      float d = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) d += geo[c] * w[c];
      const float lvi = kStepScale * step_sz * density_act(d);
      vol_int += lvi;
      if (local_alpha) local_alpha[k] = fminf(kMaxAlpha, 1.f - expf(-lvi));
    }
    qx = qx + qsx; qy = qy + qsy; qz = qz + qsz;
  }
  return FAST ? fast_transmittance(step_sz, vol_int) : expf(-vol_int);
}

// Does staged record `slot` possibly touch a pixel of this warp's 8x4
// micro-tile with a matching ray quadrant?
template <class STAGE>
__device__ __forceinline__ bool record_hits_warp(const STAGE& s, int slot, uint32_t wx0, uint32_t wy0,
                                                 uint32_t quad_mask) {
  const uint4 b = s.box[slot];
  return b.x <= wx0 + 7u && b.x + b.y >= wx0 && b.z <= wy0 + 3u && b.z + (b.w & 0xFFFFu) >= wy0 &&
         ((quad_mask >> (b.w >> 16)) & 1u);
}

// 32x32 bit matrix held one row per lane (bit l of lane j's word = entry
// (j, l)) to its transpose: lane l returns the column l as a word, bit j =
// entry (j, l).  Five exchanges swapping off-diagonal blocks of 16, 8, 4, 2
// and 1 columns.
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t v, uint32_t lane) {
  const uint32_t keep[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 16 >> k;
    const uint32_t x = __shfl_xor_sync(0xffffffffu, v, d);
    const uint32_t m = keep[k];
    v = (lane & (uint32_t)d) ? ((v & ~m) | ((x >> d) & m)) : ((v & m) | ((x & m) << d));
  }
  return v;
}

// Pixels of the 8x4 block with corner (bx0, by0) that staged box b covers, as
// a 32-bit lane mask (lane = row * 8 + column; byte r = row r): the
// record_hits_pixel bbox test for 32 pixels at once.  0 when disjoint.
__device__ __forceinline__ uint32_t block_cover_mask(const uint4& b, uint32_t bx0, uint32_t by0) {
  const uint32_t x1 = b.x + b.y, y1 = b.z + (b.w & 0xFFFFu);
  if (b.x > bx0 + 7u || x1 < bx0 || b.z > by0 + 3u || y1 < by0) return 0u;
  const uint32_t cx0 = max(b.x, bx0) - bx0, cx1 = min(x1, bx0 + 7u) - bx0;
  const uint32_t ry0 = max(b.z, by0) - by0, ry1 = min(y1, by0 + 3u) - by0;
  const uint32_t cols = (0xFFu >> (7u - cx1)) & (0xFFu << cx0);
  const uint32_t rows = (0x01010101u >> (8u * (3u - ry1))) & (0x01010101u << (8u * ry0));
  return cols * rows;
}

// The reference's per-pixel test: pixel inside the packed bbox and ray
// quadrant equal to the instance's (forward.cu:186), as two unsigned range
// checks on the staged (min, extent) form.
template <class STAGE>
__device__ __forceinline__ bool record_hits_pixel(const STAGE& s, int j, uint32_t px, uint32_t py,
                                                  uint32_t quad) {
  const uint4 b = s.box[j];
  return (px - b.x) <= b.y && (py - b.z) <= (b.w & 0xFFFFu) && (b.w >> 16) == quad;
}

template <class STAGE>
__device__ __forceinline__ void load_geo(const STAGE& s, int j, float g[8]) {
  const float4 a = s.geo[j][0], b = s.geo[j][1];
  g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
  g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
}

// Linear-gradient "normal" of the trilinear field (forward.cu:301-310).
__device__ __forceinline__ void field_normal(const float g[8], float& nx, float& ny, float& nz) {
  nx = ((g[4] + g[5] + g[6] + g[7]) - (g[0] + g[1] + g[2] + g[3]));
  ny = ((g[2] + g[3] + g[6] + g[7]) - (g[0] + g[1] + g[4] + g[5]));
  nz = ((g[1] + g[3] + g[5] + g[7]) - (g[0] + g[2] + g[4] + g[6]));
}

}  // namespace svr
