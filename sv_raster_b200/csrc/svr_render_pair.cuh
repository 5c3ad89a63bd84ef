// Compositing with two pixels per thread (batched path, colour and
// transmittance only).
//
// A warp covers an 8x8 block of the tile: lane l owns the pixels
// (l & 7, l >> 3) and (l & 7, (l >> 3) + 4).  A staged record that a warp's
// ballot selects is tested against both pixels; the records' shared-memory
// fields are read once for the pair, and in the backward the two pixels'
// gradients are added in registers and take one row.
//
// The per-pixel arithmetic is the one of svr_render_fwd.cuh /
// svr_render_bwd.cuh (forward.cu:182-316, backward.cu:246-418) without the
// depth, distortion, normal and regulariser terms, expression for expression,
// so images, T and contributor counts equal the one-pixel kernels' bit for
// bit; gradients differ only in the order of additions.
#pragma once

#include "svr_render_bwd.cuh"
#include "svr_render_fwd.cuh"

namespace svr {

// TS x TS tiles, TS*TS/2 threads, warps laid out row-major as 8x8 blocks,
// SB records staged per round.
template <int TS_, int SB_>
struct PairCfg {
  static constexpr int TS = TS_;
  static constexpr int NT = TS * TS / 2;  // threads per CTA
  static constexpr int NW = NT / 32;      // warps per CTA
  static constexpr int MX = TS / 8;       // 8x8 blocks per tile row
  static constexpr int SB = SB_;
  static constexpr int GROUPS = SB / 32;
  static_assert(TS == 8 || TS == 16, "tile size");
  static_assert(SB % 32 == 0 && SB >= 32, "staging depth");
};

// Resident CTAs per SM the pair kernels are register-bounded for, per 32
// threads: 20 warps of 32 threads leave each thread about 100 registers for
// the two pixels' state.
constexpr int kPairWarpsPerSM = 20;
template <class CFG>
constexpr int pair_min_blocks() { return kPairWarpsPerSM / CFG::NW; }

// Does staged record `slot` possibly touch a pixel of this warp's 8x8 block
// with a matching ray quadrant?
template <class STAGE>
__device__ __forceinline__ bool record_hits_block8(const STAGE& s, int slot, uint32_t wx0, uint32_t wy0,
                                                   uint32_t quad_mask) {
  const uint4 b = s.box[slot];
  return b.x <= wx0 + 7u && b.x + b.y >= wx0 && b.z <= wy0 + 7u && b.z + (b.w & 0xFFFFu) >= wy0 &&
         ((quad_mask >> (b.w >> 16)) & 1u);
}

template <class CFG, int NS, bool FAST>
__device__ __forceinline__ void render_tile_fwd_pair(const ViewParams& vp, const float* __restrict__ c2w_s,
                                                     int tile_x, int tile_y, uint2 range,
                                                     const uint32_t* __restrict__ vals, const VoxelArrays& va,
                                                     const FwdTileOut& out, uint32_t* last_slot,
                                                     FwdStage<CFG::SB>& s, uint32_t* s_red /*[CFG::NW]*/) {
  constexpr int SB = CFG::SB;
  const int W = vp.W, H = vp.H;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t wx0 = tile_x * CFG::TS + (warp % CFG::MX) * 8, wy0 = tile_y * CFG::TS + (warp / CFG::MX) * 8;
  const uint32_t px = wx0 + (lane & 7);
  uint32_t py[2];
  bool inside[2], done[2];
  PixelRay ray[2];
  float T[2], Cx[2], Cy[2], Cz[2];
  uint32_t last_contrib[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    py[k] = wy0 + (lane >> 3) + 4 * k;
    inside[k] = px < (uint32_t)W && py[k] < (uint32_t)H;
    ray[k] = make_pixel_ray((float)px, (float)py[k], W, H, vp.tanfovx, vp.tanfovy, vp.cx, vp.cy, c2w_s);
    done[k] = !inside[k];
    T[k] = 1.f;
    Cx[k] = Cy[k] = Cz[k] = 0.f;
    last_contrib[k] = 0;
  }

  const int todo_total = (int)(range.y - range.x);
  const int rounds = (todo_total + SB - 1) / SB;
  for (int r = 0; r < rounds; ++r) {
    if (__syncthreads_count(done[0] && done[1]) == CFG::NT) break;
    const int base = r * SB;
    const int n_here = min(SB, todo_total - base);
    for (int i = tid; i < n_here; i += CFG::NT)
      stage_record<FAST, true>(s, i, vals[range.x + base + i], va, ray[0].ox, ray[0].oy, ray[0].oz);
    __syncthreads();

    const uint32_t quad_mask = __reduce_or_sync(
        0xffffffffu, (done[0] ? 0u : (1u << ray[0].quad)) | (done[1] ? 0u : (1u << ray[1].quad)));
    if (quad_mask == 0u) continue;
    for (int g = 0; g < CFG::GROUPS && g * 32 < n_here; ++g) {
      const int slot = g * 32 + lane;
      const bool hit = slot < n_here && record_hits_block8(s, slot, wx0, wy0, quad_mask);
      uint32_t m = __ballot_sync(0xffffffffu, hit);
      while (m) {
        const int j = g * 32 + __ffs(m) - 1;
        m &= m - 1;
        const float4 rel = s.rel[j];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (done[k] || !record_hits_pixel(s, j, px, py[k], ray[k].quad)) continue;
          const float2 ab = octant_ray_box(rel, ray[k]);
          const float a = ab.x, b = ab.y;
          if (!(a <= b)) continue;
          const float alpha = fminf(kMaxAlpha, 1.f - record_transmittance<NS, FAST>(s, j, ray[k], a, b, nullptr));
          if (alpha < kMinAlpha) continue;
          const float pt_w = T[k] * alpha;
          const float4 rgbv = s.rgb[j];
          Cx[k] = Cx[k] + pt_w * rgbv.x;
          Cy[k] = Cy[k] + pt_w * rgbv.y;
          Cz[k] = Cz[k] + pt_w * rgbv.z;
          T[k] *= (1.f - alpha);
          done[k] |= (T[k] < kEarlyStopT);
          last_contrib[k] = (uint32_t)(base + j + 1);
        }
      }
    }
  }

  const size_t HW = (size_t)H * W;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!inside[k]) continue;
    const uint32_t pix_id = (uint32_t)W * py[k] + px;
    out.n_contrib[pix_id] = last_contrib[k];
    out.color[0 * HW + pix_id] = Cx[k] + T[k] * vp.bg;
    out.color[1 * HW + pix_id] = Cy[k] + T[k] * vp.bg;
    out.color[2 * HW + pix_id] = Cz[k] + T[k] * vp.bg;
    out.T[pix_id] = T[k];
  }
  const uint32_t mine = max(inside[0] ? last_contrib[0] : 0u, inside[1] ? last_contrib[1] : 0u);
  const uint32_t lc = __reduce_max_sync(0xffffffffu, mine);
  if (lane == 0) s_red[warp] = lc;
  __syncthreads();
  if (tid == 0) {
    uint32_t mx = 0;
#pragma unroll
    for (int w = 0; w < CFG::NW; ++w) mx = max(mx, s_red[w]);
    *last_slot = range.x + mx;
  }
}

// Gradient rows of one warp: 12 values (8 corner densities, 3 colour, 1
// subdivision priority) from each lane that contributes to a record, a record's
// rows next to each other.  When they run out of room, or the tile ends,
// flush_rows adds each record's rows up and sends the sums to global memory.
// Against reducing each record over the warp as it is visited (13 shuffles and
// as many selects, or a transposition for few lanes), the sums of many records
// run side by side (the backward of eight full-HD views of 8M voxels: 15.3 ->
// 13.7 ms together with the shorter arithmetic).  96 rows: 128 take more of the
// L1 cache from the staging's gathers than they save in flushes (15.2 ms), 64
// and 40 flush more often (14.0, 15.0).
constexpr int kPairRows = 96;
struct PairRows {
  float4 row[kPairRows][3];
  uint2 recs[32];  // voxel id, first row | rows << 16
};

// Per-pixel state of the two-pixel backward.
struct PairPix {
  PixelRay ray;
  float T, last_dL_dT;
  float gx, gy, gz;
};

// v[c] += x times the corner weights at (qx, qy, qz), split axis by axis.
__device__ __forceinline__ void add_split(float x, float qx, float qy, float qz, float v[8]) {
  const float mz = 1.f - qz;
  const float x1 = x * qx, x0 = x - x1;
  const float x0y1 = x0 * qy, x0y0 = x0 - x0y1;
  const float x1y1 = x1 * qy, x1y0 = x1 - x1y1;
  v[0] += x0y0 * mz; v[1] += x0y0 * qz;
  v[2] += x0y1 * mz; v[3] += x0y1 * qz;
  v[4] += x1y0 * mz; v[5] += x1y0 * qz;
  v[6] += x1y1 * mz; v[7] += x1y1 * qz;
}

// A staged record in registers, read once for both pixels and before either
// needs it.
struct PairRecord {
  float4 near, far, corner, geo_lo, geo_hi, rgb;
};
template <int SB>
__device__ __forceinline__ PairRecord load_record(const BwdStage<SB>& s, int j) {
  return PairRecord{s.near[j], s.far[j], s.corner[j], s.geo[j][0], s.geo[j][1], s.rgb[j]};
}

// One (pixel, staged record) step: slab test, recomputed quadrature, T
// recovery and the 12 gradients, added to gp.  False, with gp as it was, when the
// record does not contribute.
template <int NS, bool FAST>
__device__ __forceinline__ bool pair_pixel_record(const PairRecord& rec, PairPix& p, float gp[12]) {
  const float4 &nr = rec.near, &fr = rec.far, &cr = rec.corner, &glo = rec.geo_lo, &ghi = rec.geo_hi, &rgbv = rec.rgb;
  const float2 ab = near_far_ray_box(nr, fr, p.ray);
  const float a = ab.x, b = ab.y;
  const float vox_l_inv = nr.w;
  const float step_sz = (b - a) * (1.f / NS);
  const float t0 = a + 0.5f * step_sz;
  float qx, qy, qz;
  place_in_voxel(p.ray, t0, cr, vox_l_inv, qx, qy, qz);
  constexpr bool kSplit = FAST && NS == 1;
  float exp_neg, dd_dd = 0.f;  // one sample: d(optical depth)/d(density) at it
  float dI_dgeo[8];            // several samples: d(optical depth)/d(corner densities)
  if (kSplit) {
    float act, act_grad;
    density_act_and_grad_f<true>(trilinear_poly(glo, ghi, qx, qy, qz), act, act_grad);
    exp_neg = fast_transmittance(step_sz, act);
    dd_dd = kStepScale * step_sz * act_grad;
  } else {
    const float geo[8] = {glo.x, glo.y, glo.z, glo.w, ghi.x, ghi.y, ghi.z, ghi.w};
    const float stx = step_sz * p.ray.dx, sty = step_sz * p.ray.dy, stz = step_sz * p.ray.dz;
    const float qsx = stx * vox_l_inv, qsy = sty * vox_l_inv, qsz = stz * vox_l_inv;
    float vol_int = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) dI_dgeo[c] = 0.f;
#pragma unroll
    for (int n = 0; n < NS; ++n) {
      float w[8], d = 0.f;
      if (FAST) {
        d = trilinear_poly(glo, ghi, qx, qy, qz);
      } else {
        trilinear_weights(qx, qy, qz, w);
#pragma unroll
        for (int c = 0; c < 8; ++c) d += geo[c] * w[c];
      }
      float act, act_grad;
      density_act_and_grad_f<FAST>(d, act, act_grad);
      vol_int += FAST ? act : kStepScale * step_sz * act;
      const float dd = kStepScale * step_sz * act_grad;
      if (FAST) {
        add_split(dd, qx, qy, qz, dI_dgeo);
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) dI_dgeo[c] += dd * w[c];
      }
      qx = qx + qsx; qy = qy + qsy; qz = qz + qsz;
    }
    exp_neg = FAST ? fast_transmittance(step_sz, vol_int) : expf(-vol_int);
  }
  const float alpha = fminf(kMaxAlpha, 1.f - exp_neg);
  if (!(a <= b) || alpha < kMinAlpha) return false;
  p.T = div_f<FAST>(p.T, 1.f - alpha);
  const float pt_w = alpha * p.T;
  const float dL_dpt_w = p.gx * rgbv.x + p.gy * rgbv.y + p.gz * rgbv.z;
  const float diff = dL_dpt_w - p.last_dL_dT;
  const float dL_dalpha = p.T * diff;
  p.last_dL_dT += alpha * diff;
  const float dL_dI = dL_dalpha * exp_neg;
  if (kSplit) {
    add_split(dL_dI * dd_dd, qx, qy, qz, gp);
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) gp[c] += dL_dI * dI_dgeo[c];
  }
  gp[8] += pt_w * p.gx;
  gp[9] += pt_w * p.gy;
  gp[10] += pt_w * p.gz;
  gp[11] += fabsf(dL_dalpha) * alpha;
  return true;
}

__device__ __forceinline__ void store_row(float4* row, const float gp[12]) {
  row[0] = make_float4(gp[0], gp[1], gp[2], gp[3]);
  row[1] = make_float4(gp[4], gp[5], gp[6], gp[7]);
  row[2] = make_float4(gp[8], gp[9], gp[10], gp[11]);
}

// GRID: densities as grid points (VoxelArrays::key / BwdTileOut::key set);
// the per-voxel form is instantiated without the grid reads.
template <class CFG, int NS, bool FAST, bool GRID>
__device__ __forceinline__ void render_tile_bwd_pair(const ViewParams& vp, const float* __restrict__ c2w_s,
                                                     int tile_x, int tile_y, uint2 range_raw, uint32_t tile_last,
                                                     const uint32_t* __restrict__ vals, const VoxelArrays& va,
                                                     const BwdTileIn& in, const BwdTileOut& out,
                                                     BwdStage<CFG::SB>& s, PairRows* s_rows /*[CFG::NW]*/) {
  constexpr int SB = CFG::SB;
  const int W = vp.W, H = vp.H;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t wx0 = tile_x * CFG::TS + (warp % CFG::MX) * 8, wy0 = tile_y * CFG::TS + (warp / CFG::MX) * 8;
  const uint32_t px = wx0 + (lane & 7);

  // Range check (replaces the __trap at backward.cu:122-133).
  if (tile_last > range_raw.y || range_raw.x > tile_last) {
    if (tid == 0) atomicOr(out.err, SVR_DEVERR_RANGE);
    return;
  }
  const uint2 range = make_uint2(range_raw.x, tile_last);
  const size_t HW = (size_t)H * W;
  const int todo_total = (int)(range.y - range.x);
  PairRows& rows = s_rows[warp];
  int n_rows = 0, n_rec = 0;

  uint32_t last_contrib[2];
  bool inside[2];
  PairPix pix[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t py = wy0 + (lane >> 3) + 4 * k;
    inside[k] = px < (uint32_t)W && py < (uint32_t)H;
    PairPix& p = pix[k];
    p.ray = make_pixel_ray<false>((float)px, (float)py, W, H, vp.tanfovx, vp.tanfovy, vp.cx, vp.cy, c2w_s);
    const uint32_t pix_id = (uint32_t)W * py + px;
    p.T = inside[k] ? in.T[pix_id] : 0.f;
    last_contrib[k] = inside[k] ? in.n_contrib[pix_id] : 0u;
    p.gx = p.gy = p.gz = p.last_dL_dT = 0.f;
    if (inside[k]) {
      p.gx = in.dL_dcolor[0 * HW + pix_id];
      p.gy = in.dL_dcolor[1 * HW + pix_id];
      p.gz = in.dL_dcolor[2 * HW + pix_id];
      p.last_dL_dT = in.dL_dT[pix_id] + vp.bg * (p.gx + p.gy + p.gz);
    }
  }

  const uint32_t warp_lc = __reduce_max_sync(0xffffffffu, max(last_contrib[0], last_contrib[1]));
  const uint32_t quad_mask = __reduce_or_sync(
      0xffffffffu, (inside[0] ? (1u << pix[0].ray.quad) : 0u) | (inside[1] ? (1u << pix[1].ray.quad) : 0u));
  // Lane q holds, per pixel row k, the lanes whose pixel k is in the image
  // with ray quadrant q.
  uint32_t qlanes[2] = {0u, 0u};
  for (uint32_t qm = quad_mask; qm; qm &= qm - 1) {
    const uint32_t q = (uint32_t)(__ffs(qm) - 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t bk = __ballot_sync(0xffffffffu, inside[k] && pix[k].ray.quad == q);
      if ((uint32_t)lane == q) qlanes[k] = bk;
    }
  }

  const int rounds = (todo_total + SB - 1) / SB;
  for (int r = 0; r < rounds; ++r) {
    if (CFG::NW > 1) __syncthreads();
    else __syncwarp();
    const int base = r * SB;
    const int n_here = min(SB, todo_total - base);
    for (int i = tid; i < n_here; i += CFG::NT)
      stage_record<FAST, GRID>(s, i, vals[range.y - base - i - 1], va, pix[0].ray.ox, pix[0].ray.oy, pix[0].ray.oz);
    if (CFG::NW > 1) __syncthreads();
    else __syncwarp();

    for (int g = 0; g < CFG::GROUPS && g * 32 < n_here; ++g) {
      const int slot = g * 32 + lane;
      const uint32_t pos = (uint32_t)(todo_total - base - slot - 1);
      const bool hit = slot < n_here && pos < warp_lc && record_hits_block8(s, slot, wx0, wy0, quad_mask);
      // Each lane's candidate records of this group per pixel: lane j turns
      // record j's bbox into masks of the pixels it covers in the two 8x4
      // halves, restricted to the lanes of its ray quadrant, and a bit
      // transposition hands every lane its records; a record reaches pixel k
      // only while its position is below the pixel's contributor count.
      uint32_t cov[2] = {0u, 0u};
      uint32_t rec_quad = 0u;
      if (hit) {
        const uint4 b = s.box[slot];
        cov[0] = block_cover_mask(b, wx0, wy0);
        cov[1] = block_cover_mask(b, wx0, wy0 + 4u);
        rec_quad = b.w >> 16;
      }
      uint32_t mine[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        mine[k] = warp_transpose_bits(cov[k] & __shfl_sync(0xffffffffu, qlanes[k], (int)rec_quad), (uint32_t)lane);
        // slot j is in reach while todo_total - base - j - 1 < last_contrib[k]
        const int first = todo_total - base - (int)last_contrib[k] - g * 32;
        mine[k] &= first <= 0 ? 0xffffffffu : (first >= 32 ? 0u : ~((1u << first) - 1u));
      }
      const uint32_t m0 = __reduce_or_sync(0xffffffffu, mine[0]), m1 = __reduce_or_sync(0xffffffffu, mine[1]);
      if ((m0 | m1) == 0u) continue;  // no pixel of the warp takes any of them
      mine[0] = __brev(mine[0]);
      mine[1] = __brev(mine[1]);
      uint32_t m = __brev(m0 | m1);
      while (m) {
        const int bit = bfind(m);
        const int j = g * 32 + 31 - bit;
        const uint32_t mbit = 1u << bit;
        m ^= mbit;
        const PairRecord rec = load_record(s, j);
        float gp[12];
#pragma unroll
        for (int c = 0; c < 12; ++c) gp[c] = 0.f;
        bool contrib = false;
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (mine[k] & mbit) contrib |= pair_pixel_record<NS, FAST>(rec, pix[k], gp);
        const uint32_t act_mask = __ballot_sync(0xffffffffu, contrib);
        if (act_mask == 0u) continue;
        const int n_act = __popc(act_mask);
        if (n_rows + n_act > kPairRows || n_rec == 32) {
          flush_rows<true, GRID>(rows, n_rec, lane, out);
          n_rows = n_rec = 0;
        }
        if (contrib) store_row(rows.row[n_rows + __popc(act_mask & lanemask_lt())], gp);
        if (lane == 0)
          rows.recs[n_rec] =
              make_uint2((uint32_t)__float_as_int(rec.corner.w), (uint32_t)n_rows | ((uint32_t)n_act << 16));
        n_rows += n_act;
        ++n_rec;
      }
    }
  }
  if (n_rec > 0) flush_rows<true, GRID>(rows, n_rec, lane, out);
}

}  // namespace svr
