// Backward compositing of one tile: walks the tile's list back to
// front from tile_last, recovers transmittance by division and accumulates
// per-voxel gradients.
//
// Per-pixel arithmetic mirrors BACKWARD::renderCUDA (backward.cu:35-530):
// contributor skip (:246-248), recomputed quadrature with dI/dgeo
// (:295-323), T recovery (:333), colour / distortion / normal / depth /
// ascending / colour-concentration terms (:344-510) and the 12-float
// gradient pack (:515-522).  The reference issues 12 global atomics per
// contributing (pixel, voxel); here a warp's lanes write their gradients as rows
// into shared memory (GradRows), each record's rows are summed, and a record is
// flushed once per warp (16-byte vector reductions where the gradient rows are
// aligned).
#pragma once

#include "svr_render.cuh"

namespace svr {

struct BwdTileIn {
  const float* T;          // [H*W] final transmittance from the forward
  const uint32_t* n_contrib;
  const float* dL_dcolor;  // [3,H,W]
  const float* dL_ddepth;  // [3,H,W] or nullptr
  const float* dL_dnormal; // [3,H,W] or nullptr
  const float* dL_dT;      // [H*W]
  const float* gt_color;   // [3,H,W] or nullptr
  const float* out_depth;  // [3,H,W] or nullptr (distortion prefix sums)
  float lambda_R_concen, lambda_ascending, lambda_dist;
};

struct BwdTileOut {
  float* dL_dgeos;   // [P,8]
  float* dL_drgbs;   // [P,3] (this view), or [P,4] with RGB4 (xyz = dL/drgb, w = subdivision priority)
  float* subdiv;     // [P] (unused with RGB4)
  uint32_t* err;     // device error word
  int geo_vec4;      // dL_dgeos is 16-byte aligned: flush its rows with vector reductions
  // Grid-point densities: when key is set, a record's 8 corner gradients are
  // added into grid_grad[key[8 v + c]] instead of a dL_dgeos row.
  const int64_t* key = nullptr;
  float* grid_grad = nullptr;
};

// Four of a record's 12 summed gradients to global memory: q = 0, 1 the
// corner densities 4q .. 4q + 3 (a row of dL_dgeos, as one 16-byte reduction
// where the rows are aligned, or the grid points that the corners index), q = 2
// the colour and the subdivision priority.
template <bool RGB4, bool MAYBE_GRID>
__device__ __forceinline__ void flush_quad(const BwdTileOut& out, uint32_t vid, int q, const float4& v) {
  if (v.x == 0.f && v.y == 0.f && v.z == 0.f && v.w == 0.f) return;
  if (q == 2) {
    if (RGB4) {
      atomicAdd(reinterpret_cast<float4*>(out.dL_drgbs) + vid, v);
    } else {
      float* c = out.dL_drgbs + 3 * (size_t)vid;
      atomicAdd(c, v.x);
      atomicAdd(c + 1, v.y);
      atomicAdd(c + 2, v.z);
      atomicAdd(out.subdiv + vid, v.w);
    }
  } else if (MAYBE_GRID && out.key) {
    const int64_t* k = out.key + 8 * (size_t)vid + 4 * q;
    atomicAdd(out.grid_grad + k[0], v.x);
    atomicAdd(out.grid_grad + k[1], v.y);
    atomicAdd(out.grid_grad + k[2], v.z);
    atomicAdd(out.grid_grad + k[3], v.w);
  } else {
    float* g = out.dL_dgeos + 8 * (size_t)vid + 4 * q;
    if (RGB4 || out.geo_vec4) {
      atomicAdd(reinterpret_cast<float4*>(g), v);
    } else {
      atomicAdd(g, v.x);
      atomicAdd(g + 1, v.y);
      atomicAdd(g + 2, v.z);
      atomicAdd(g + 3, v.w);
    }
  }
}

// Gradient rows of one warp.  Every (record, pixel) pair of a run of records
// has a row of 12 values (8 corner densities, 3 colour, 1 subdivision
// priority), a record's rows next to each other in pixel order; the lanes
// fill them while each walks its own pixel's records, then add them up
// record by record.  64 rows (3.6 KB a warp): 128 leave the staging's gathers
// less of the L1 cache, 40 cut the runs too short (5.7 / 6.4 / 6.3 ms for 64 /
// 128 / 40 with 16 views of 2M voxels).
template <int ROWS_>
struct GradRows {
  static constexpr int kRows = ROWS_;
  static_assert(ROWS_ >= 32, "a record may take a row per lane");
  float4 row[ROWS_][3];
  uint2 pairs[32];  // by record of the group: lanes that take it, its first row
  uint2 recs[32];   // by place in the run: voxel id, first row | rows << 16
};
template <class CFG>
using TileRows = GradRows<64>;

// Sums the rows of the run's n_rec records and sends them off.  Lanes take
// (record, four of its values) and, while lanes are left over, a half or a
// quarter of its rows.
template <bool RGB4, bool MAYBE_GRID, class ROWS>
__device__ __forceinline__ void flush_rows(const ROWS& g, int n_rec, int lane, const BwdTileOut& out) {
  __syncwarp();
  const int fs = n_rec <= 2 ? 2 : (n_rec <= 5 ? 1 : 0);  // log2 of the lanes per (record, values)
  const int n = (3 * n_rec) << fs;
  for (int e0 = 0; e0 < n; e0 += 32) {
    const int e = e0 + lane;
    const int rq = min(e, n - 1) >> fs;
    const int r = rq / 3, q = rq - 3 * r;
    const uint2 rec = g.recs[r];
    const int i0 = (int)(rec.y & 0xFFFFu), i1 = i0 + (int)(rec.y >> 16);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = i0 + (e & ((1 << fs) - 1)); i < i1; i += 1 << fs) {
      const float4 x = g.row[i][q];
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    __syncwarp();
    for (int d = 1; d < (1 << fs); d <<= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
      v.z += __shfl_xor_sync(0xffffffffu, v.z, d);
      v.w += __shfl_xor_sync(0xffffffffu, v.w, d);
    }
    if (e < n && (e & ((1 << fs) - 1)) == 0)
      flush_quad<RGB4, MAYBE_GRID>(out, rec.x, q, v);
  }
  __syncwarp();
}

// Per-pixel state of the backward walk (the pixel's upstream gradients, its
// transmittance being recovered record by record, and the running sums).
struct BwdPix {
  float T, last_dL_dT;
  float gx, gy, gz, dL_dD, dNx, dNy, dNz, gtx, gty, gtz;
  float weight_R, weight_asc, weight_dist;
  float prefix_wm, suffix_wm, prefix_w, suffix_w;
};

template <bool DEPTH, bool DIST, bool NORMAL>
__device__ __forceinline__ BwdPix bwd_pixel_init(const ViewParams& vp, const BwdTileIn& in, const PixelRay& ray,
                                                 bool inside, uint32_t pix_id, float T_final) {
  const int W = vp.W, H = vp.H;
  const size_t HW = (size_t)H * W;
  BwdPix st;
  st.T = T_final;
  st.gx = 0.f; st.gy = 0.f; st.gz = 0.f; st.last_dL_dT = 0.f; st.dL_dD = 0.f;
  st.dNx = 0.f; st.dNy = 0.f; st.dNz = 0.f;
  if (inside) {
    st.gx = in.dL_dcolor[0 * HW + pix_id];
    st.gy = in.dL_dcolor[1 * HW + pix_id];
    st.gz = in.dL_dcolor[2 * HW + pix_id];
    const float dT = in.dL_dT[pix_id];
    st.last_dL_dT = dT + vp.bg * (st.gx + st.gy + st.gz);
    if (DEPTH) st.dL_dD = in.dL_ddepth[pix_id] * ray.rd_norm_inv;
    if (NORMAL) {
      st.dNx = in.dL_dnormal[0 * HW + pix_id];
      st.dNy = in.dL_dnormal[1 * HW + pix_id];
      st.dNz = in.dL_dnormal[2 * HW + pix_id];
    }
  }
  const float WH_inv = 1.f / ((float)(W * H));
  st.weight_R = in.lambda_R_concen * WH_inv;
  st.weight_asc = in.lambda_ascending * WH_inv;
  st.gtx = 0.f; st.gty = 0.f; st.gtz = 0.f;
  if (in.lambda_R_concen > 0 && inside) {
    st.gtx = in.gt_color[0 * HW + pix_id];
    st.gty = in.gt_color[1 * HW + pix_id];
    st.gtz = in.gt_color[2 * HW + pix_id];
  }
  st.weight_dist = in.lambda_dist * WH_inv;
  st.prefix_wm = 0.f; st.suffix_wm = 0.f; st.prefix_w = 0.f; st.suffix_w = 0.f;
  if (DIST && inside) {
    st.prefix_wm = in.out_depth[HW + pix_id];
    st.prefix_w = 1.f - T_final;
  }
  return st;
}

// One (pixel, staged record j) step of the backward walk, for a pixel inside
// the record's bbox with a matching quadrant: slab test, recomputed
// quadrature, T recovery and the 12 gradient values (8 density corners, 3
// colour, 1 subdivision priority) in gp.  Returns whether the record
// contributes (gp is left unset otherwise).
template <int SB, int NS, bool DEPTH, bool DIST, bool NORMAL, bool FAST>
__device__ __forceinline__ bool bwd_pixel_record(const FwdStage<SB>& s, int j, const PixelRay& ray,
                                                 const BwdTileIn& in, BwdPix& st, float gp[12]) {
  float& T = st.T;
  float& last_dL_dT = st.last_dL_dT;
  float& prefix_wm = st.prefix_wm;
  float& suffix_wm = st.suffix_wm;
  float& prefix_w = st.prefix_w;
  float& suffix_w = st.suffix_w;
  const float gx = st.gx, gy = st.gy, gz = st.gz, dL_dD = st.dL_dD;
  const float dNx = st.dNx, dNy = st.dNy, dNz = st.dNz, gtx = st.gtx, gty = st.gty, gtz = st.gtz;
  const float weight_R = st.weight_R, weight_asc = st.weight_asc, weight_dist = st.weight_dist;
  (void)dL_dD; (void)dNx; (void)dNy; (void)dNz; (void)weight_dist;
  (void)prefix_wm; (void)suffix_wm; (void)prefix_w; (void)suffix_w;
  bool contrib = false;
  // One sample, no depth terms: dL/dgeo is dL/d(density) times the corner
  // weights; the fast arithmetic splits it axis by axis instead of forming
  // the weights (the density itself is a polynomial there).
  constexpr bool kFoldScale = NS == 1 && !DEPTH;
  const float2 ab = octant_ray_box(s.rel[j], ray);
  const float a = ab.x, b = ab.y;
  {
    float geo[8];  // with the fast arithmetic: the density polynomial
    load_geo(s, j, geo);
    float dgeo[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) dgeo[c] = 0.f;
    float vol_int = 0.f;
    float dI_dgeo[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) dI_dgeo[c] = 0.f;
    float each_dI[NS][8];
    float w[8];
    float local_alpha[NS];
    const float4 cr = s.corner[j];
    const float vox_l_inv = cr.w;
    const float step_sz = (b - a) * (1.f / NS);
    const float stx = step_sz * ray.dx, sty = step_sz * ray.dy, stz = step_sz * ray.dz;
    const float t0 = a + 0.5f * step_sz;
    // Scalar here: with x and y packed, as the forward has it, this kernel took 883
    // us against 872 for one 1297x840 view (the same values either way).
    const float ptx = ray.ox + t0 * ray.dx, pty = ray.oy + t0 * ray.dy, ptz = ray.oz + t0 * ray.dz;
    float qx = (ptx - cr.x) * vox_l_inv;
    float qy = (pty - cr.y) * vox_l_inv;
    float qz = (ptz - cr.z) * vox_l_inv;
    const float qsx = stx * vox_l_inv, qsy = sty * vox_l_inv, qsz = stz * vox_l_inv;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
      if (!(FAST && kFoldScale)) trilinear_weights(qx, qy, qz, w);
      float d = 0.f;
      if (FAST) {
        d = trilinear_poly(make_float4(geo[0], geo[1], geo[2], geo[3]), make_float4(geo[4], geo[5], geo[6], geo[7]),
                           qx, qy, qz);
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) d += geo[c] * w[c];
      }
      float act, act_grad;
      density_act_and_grad_f<FAST>(d, act, act_grad);
      const float lvi = kStepScale * step_sz * act;
      vol_int += FAST ? act : lvi;
      if (DEPTH && NS > 1) local_alpha[k] = fminf(kMaxAlpha, 1.f - expf(-lvi));
      const float dd_dd = kStepScale * step_sz * act_grad;
      if (kFoldScale) {
        dI_dgeo[0] = dd_dd;
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float tmp = dd_dd * w[c];
          dI_dgeo[c] += tmp;
          if (DEPTH && NS > 1) each_dI[k][c] = tmp;
        }
      }
      if (k + 1 < NS) { qx = qx + qsx; qy = qy + qsy; qz = qz + qsz; }
    }
    const float exp_neg = FAST ? fast_transmittance(step_sz, vol_int) : expf(-vol_int);
    const float alpha = fminf(kMaxAlpha, 1.f - exp_neg);
    if (a <= b && !(alpha < kMinAlpha)) {
      contrib = true;
      T = div_f<FAST>(T, 1.f - alpha);
      const float pt_w = alpha * T;
      const float4 rgbv = s.rgb[j];
      float dL_dpt_w = gx * rgbv.x + gy * rgbv.y + gz * rgbv.z;
      if (DIST) {
        const float adist = contract_depth(a), bdist = contract_depth(b);
        const float now_m = 0.5f * (adist + bdist);
        const float now_wm = now_m * pt_w;
        prefix_wm -= now_wm;
        prefix_w -= pt_w;
        const float uni = 0.6666666f * pt_w * (bdist - adist);
        const float bi = 2.f * (now_m * (prefix_w - suffix_w) - (prefix_wm - suffix_wm));
        dL_dpt_w += weight_dist * (uni + bi);
        suffix_wm += now_wm;
        suffix_w += pt_w;
      }
      if (NORMAL) {
        float nx, ny, nz;
        field_normal(geo, nx, ny, nz);
        const float rl = safe_rnorm3(nx, ny, nz);
        const float sx = rl * nx, sy = rl * ny, sz = rl * nz;
        dL_dpt_w += dNx * sx + dNy * sy + dNz * sz;
        const float dsx = pt_w * dNx, dsy = pt_w * dNy, dsz = pt_w * dNz;
        const float dot_ = dsx * nx + dsy * ny + dsz * nz;
        const float lnx = rl * (dsx - dot_ * rl * sx);
        const float lny = rl * (dsy - dot_ * rl * sy);
        const float lnz = rl * (dsz - dot_ * rl * sz);
        dgeo[0] += -lnx - lny - lnz;
        dgeo[1] += -lnx - lny + lnz;
        dgeo[2] += -lnx + lny - lnz;
        dgeo[3] += -lnx + lny + lnz;
        dgeo[4] += +lnx - lny - lnz;
        dgeo[5] += +lnx - lny + lnz;
        dgeo[6] += +lnx + lny - lnz;
        dgeo[7] += +lnx + lny + lnz;
      }
      const float dL_dalpha = T * (dL_dpt_w - last_dL_dT);
      last_dL_dT += alpha * (dL_dpt_w - last_dL_dT);
      const float dL_dI = dL_dalpha * exp_neg;
      if (kFoldScale && FAST) {
        const float s1 = dL_dI * dI_dgeo[0];
        const float x1 = s1 * qx, x0 = s1 - x1;
        const float x0y1 = x0 * qy, x0y0 = x0 - x0y1;
        const float x1y1 = x1 * qy, x1y0 = x1 - x1y1;
        dgeo[1] = x0y0 * qz; dgeo[0] = x0y0 - dgeo[1];
        dgeo[3] = x0y1 * qz; dgeo[2] = x0y1 - dgeo[3];
        dgeo[5] = x1y0 * qz; dgeo[4] = x1y0 - dgeo[5];
        dgeo[7] = x1y1 * qz; dgeo[6] = x1y1 - dgeo[7];
      } else if (kFoldScale) {
        const float sI = dL_dI * dI_dgeo[0];
#pragma unroll
        for (int c = 0; c < 8; ++c) dgeo[c] += sI * w[c];
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) dgeo[c] += dL_dI * dI_dgeo[c];
      }
      if (DEPTH) {
        float dval;
        float dI[NS];
        if (NS == 3) {
          const float ss = 0.3333333f * (b - a);
          const float a0 = local_alpha[0], a1 = local_alpha[NS > 1 ? 1 : 0], a2 = local_alpha[NS > 2 ? 2 : 0];
          const float t0_ = a + 0.5f * ss, t1_ = a + 1.5f * ss, t2_ = a + 2.5f * ss;
          dval = a0 * t0_ + (1.f - a0) * a1 * t1_ + (1.f - a0) * (1.f - a1) * a2 * t2_;
          dI[0] = dL_dD * T * (t0_ + a1 * a2 * t2_ - a1 * t1_ - a2 * t2_) * (1.f - a0);
          dI[NS > 1 ? 1 : 0] = dL_dD * T * (t1_ + a0 * a2 * t2_ - a0 * t1_ - a2 * t2_) * (1.f - a1);
          dI[NS > 2 ? 2 : 0] = dL_dD * T * (t2_ + a0 * a1 * t2_ - a0 * t2_ - a1 * t2_) * (1.f - a2);
        } else if (NS == 2) {
          const float ss = 0.5f * (b - a);
          const float a0 = local_alpha[0], a1 = local_alpha[NS > 1 ? 1 : 0];
          const float t0_ = a + 0.5f * ss, t1_ = a + 1.5f * ss;
          dval = a0 * t0_ + (1.f - a0) * a1 * t1_;
          dI[0] = dL_dD * T * (t0_ - a1 * t1_) * (1.f - a0);
          dI[NS > 1 ? 1 : 0] = dL_dD * T * (t1_ - a0 * t1_) * (1.f - a1);
        } else {
          const float t0_ = 0.5f * (a + b);
          dval = alpha * t0_;
          dI[0] = dL_dD * T * t0_ * (1.f - alpha);
        }
        last_dL_dT += dL_dD * dval;
        if (NS == 3) {
#pragma unroll
          for (int c = 0; c < 8; ++c)
            dgeo[c] += dI[0] * each_dI[0][c] + dI[NS > 1 ? 1 : 0] * each_dI[NS > 1 ? 1 : 0][c] +
                       dI[NS > 2 ? 2 : 0] * each_dI[NS > 2 ? 2 : 0][c];
        } else if (NS == 2) {
#pragma unroll
          for (int c = 0; c < 8; ++c)
            dgeo[c] += dI[0] * each_dI[0][c] + dI[NS > 1 ? 1 : 0] * each_dI[NS > 1 ? 1 : 0][c];
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) dgeo[c] += dI[0] * dI_dgeo[c];
        }
      }
      if (!FAST && in.lambda_ascending > 0) {
        const float lo_x = cr.x, lo_y = cr.y, lo_z = cr.z;
        const float pax = ray.ox + a * ray.dx, pay = ray.oy + a * ray.dy, paz = ray.oz + a * ray.dz;
        const float pbx = ray.ox + b * ray.dx, pby = ray.oy + b * ray.dy, pbz = ray.oz + b * ray.dz;
        float wa[8], wb[8];
        trilinear_weights((pax - lo_x) * vox_l_inv, (pay - lo_y) * vox_l_inv, (paz - lo_z) * vox_l_inv, wa);
        trilinear_weights((pbx - lo_x) * vox_l_inv, (pby - lo_y) * vox_l_inv, (pbz - lo_z) * vox_l_inv, wb);
        float d_a = 0.f, d_b = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          d_a += geo[c] * wa[c];
          d_b += geo[c] * wb[c];
        }
        const float reg_w = weight_asc * pt_w * static_cast<float>(d_a > d_b);
#pragma unroll
        for (int c = 0; c < 8; ++c) dgeo[c] += reg_w * (wa[c] - wb[c]);
      }
      float drx = pt_w * gx, dry = pt_w * gy, drz = pt_w * gz;
      if (in.lambda_R_concen > 0) {
        const float sR = weight_R * pt_w * 2.0f;
        drx += sR * (rgbv.x - gtx);
        dry += sR * (rgbv.y - gty);
        drz += sR * (rgbv.z - gtz);
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) gp[c] = dgeo[c];
      gp[8] = drx; gp[9] = dry; gp[10] = drz;
      gp[11] = fabsf(dL_dalpha * alpha);
    }
  }
  return contrib;
}

// One tile, one pixel per thread, each warp an 8x4 block of its own.  Each lane
// walks its own pixel's records of a staged batch, as in the forward, so a warp
// takes as many iterations as its busiest pixel has records and not one per
// record that touches it; the 12 gradients of each pair go to the record's rows
// (GradRows), which are summed when the run of records that they have room
// for is through.  RGB4: the [P,4] colour-gradient layout, and 16-byte aligned
// density rows.
template <class CFG, int NS, bool DEPTH, bool DIST, bool NORMAL, bool FAST = false, bool RGB4 = false,
          bool MAYBE_GRID = false, bool SHARED_LIST = false>
__device__ __forceinline__ void render_tile_bwd(const ViewParams& vp, const float* __restrict__ c2w_s, int tile_x,
                                                int tile_y, uint2 range_raw, uint32_t tile_last,
                                                const uint32_t* __restrict__ vals, const VoxelArrays& va,
                                                const BwdTileIn& in, const BwdTileOut& out, FwdStage<CFG::SB>& s,
                                                TileRows<CFG>* s_rows /*[CFG::NW]*/,
                                                ListFilter<CFG>* s_list = nullptr) {
  constexpr int SB = CFG::SB;
  const int W = vp.W, H = vp.H;
  const int tid = threadIdx.x, lane = tid & 31;
  int lx, ly;
  tile_pixel_of<CFG>(tid, lx, ly);
  const uint32_t px = tile_x * CFG::TS + lx, py = tile_y * CFG::TS + ly;
  const uint32_t pix_id = (uint32_t)W * py + px;
  const bool inside = px < (uint32_t)W && py < (uint32_t)H;
  const PixelRay ray = make_pixel_ray<!RGB4>((float)px, (float)py, W, H, vp.tanfovx, vp.tanfovy, vp.cx, vp.cy, c2w_s);
  const int warp = tid >> 5;
  const uint32_t wx0 = tile_x * CFG::TS + (warp % CFG::MX) * 8, wy0 = tile_y * CFG::TS + (warp / CFG::MX) * 4;
  TileRows<CFG>& rows = s_rows[warp];

  // Range check (replaces the __trap at backward.cu:122-133).
  if (tile_last > range_raw.y || range_raw.x > tile_last) {
    if (tid == 0) atomicOr(out.err, SVR_DEVERR_RANGE);
    return;
  }
  const uint2 range = make_uint2(range_raw.x, tile_last);

  const float T_final = inside ? in.T[pix_id] : 0.f;
  const int todo_total = (int)(range.y - range.x);
  const uint32_t last_contrib = inside ? in.n_contrib[pix_id] : 0u;
  BwdPix st = bwd_pixel_init<DEPTH, DIST, NORMAL>(vp, in, ray, inside, pix_id, T_final);

  // Largest contributor count of this warp: records at or beyond it are skipped by every lane.
  const uint32_t warp_lc = __reduce_max_sync(0xffffffffu, last_contrib);
  const uint32_t quad_mask = __reduce_or_sync(0xffffffffu, inside ? (1u << ray.quad) : 0u);
  // Lane q holds the lanes whose pixel is in the image with ray quadrant q.
  uint32_t qlanes = 0u;
  for (uint32_t qm = quad_mask; qm; qm &= qm - 1) {
    const uint32_t q = (uint32_t)(__ffs(qm) - 1);
    const uint32_t bq = __ballot_sync(0xffffffffu, inside && ray.quad == q);
    if ((uint32_t)lane == q) qlanes = bq;
  }

  const int rounds = (todo_total + SB - 1) / SB;
  ListReader<CFG, true> list;
  if (SHARED_LIST) list.init(range, tile_x, tile_y, vals, va);
  for (int r = 0; SHARED_LIST || r < rounds; ++r) {
    __syncthreads();
    const int base = r * SB;                     // records [base, base+n_here) from the back
    const int n_here = SHARED_LIST ? list.round(*s_list, vals, va) : min(SB, todo_total - base);
    if (SHARED_LIST && n_here == 0) break;
    for (int i = tid; i < (SHARED_LIST ? SB : n_here); i += CFG::NT) {
      uint32_t val;
      if (SHARED_LIST) {
        // positions relative to range.x; 0 past the round, in reach of everyone and covering nothing
        if (i >= n_here) {
          s_list->pos[i] = 0u;
          continue;
        }
        const uint2 e = list.entry(*s_list, n_here, i);
        val = e.x;
        s_list->pos[i] = (uint32_t)(todo_total - 1) - e.y;
      } else {
        val = vals[range.y - base - i - 1];
      }
      stage_record<FAST, MAYBE_GRID>(s, i, val, va, ray.ox, ray.oy, ray.oz);
    }
    __syncthreads();

    // Position (relative to range.x) of staged slot j is todo_total - base - j - 1, or in s_list.
    for (int g = 0; g < CFG::GROUPS && g * 32 < n_here; ++g) {
      const int slot = g * 32 + lane;
      const uint32_t pos = SHARED_LIST ? s_list->pos[slot] : (uint32_t)(todo_total - base - slot - 1);
      const bool hit = slot < n_here && pos < warp_lc && record_hits_warp(s, slot, wx0, wy0, quad_mask);
      // This lane's candidate records of the group (pixel in the record's
      // bbox, matching quadrant, record within the contributor count): lane
      // j's block mask of record j, transposed across the warp.
      uint32_t covers = 0u, rec_quad = 0u;
      if (hit) {
        const uint4 b = s.box[slot];
        covers = block_cover_mask(b, wx0, wy0);
        rec_quad = b.w >> 16;
      }
      uint32_t mine = warp_transpose_bits(covers & __shfl_sync(0xffffffffu, qlanes, (int)rec_quad), (uint32_t)lane);
      if (SHARED_LIST) {
        // the first slot whose position is below this pixel's contributor
        // count (positions fall with the slot)
        int first = 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
          if (s_list->pos[g * 32 + first + d - 1] >= last_contrib) first += d;
        if (s_list->pos[g * 32 + first] >= last_contrib) ++first;
        mine &= first >= 32 ? 0u : ~((1u << first) - 1u);
      } else {
        // slot j is in reach while todo_total - base - j - 1 < last_contrib
        const int first = todo_total - base - (int)last_contrib - g * 32;
        mine &= first <= 0 ? 0xffffffffu : (first >= 32 ? 0u : ~((1u << first) - 1u));
      }
      // Back: lane j holds the lanes that take record j, and the records'
      // rows one after the other.
      const uint32_t takers = warp_transpose_bits(mine, (uint32_t)lane);
      const uint32_t n_takers = __popc(takers);
      uint32_t incl = n_takers;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
      }
      mine = __brev(mine);  // record j of the group is bit 31 - j: walked highest bit first
      uint32_t done_rows = 0u;
      const uint32_t all_rows = __shfl_sync(0xffffffffu, incl, 31);
      uint32_t left = 0xffffffffu;  // records not yet walked (bit j)
      while (done_rows < all_rows) {
        // the run of records whose rows fit
        const bool in_run = ((left >> lane) & 1u) && incl - done_rows <= (uint32_t)TileRows<CFG>::kRows;
        const uint32_t run = __ballot_sync(0xffffffffu, in_run);
        const uint32_t used = __ballot_sync(0xffffffffu, in_run && n_takers > 0u);
        const uint32_t first_row = incl - n_takers - done_rows;
        if (in_run) {
          rows.pairs[lane] = make_uint2(takers, first_row);
          if (n_takers > 0u)
            rows.recs[__popc(used & lanemask_lt())] = make_uint2((uint32_t)__float_as_int(s.rgb[slot].w), first_row | (n_takers << 16));
        }
        done_rows = __shfl_sync(0xffffffffu, incl, 31 - __clz((int)run));
        left &= ~run;
        __syncwarp();
        uint32_t walk = mine & __brev(run);
        while (walk) {
          const int bit = bfind(walk);
          walk ^= 1u << bit;
          const int jj = 31 - bit;
          float gp[12];
          if (!bwd_pixel_record<SB, NS, DEPTH, DIST, NORMAL, FAST>(s, g * 32 + jj, ray, in, st, gp)) {
#pragma unroll
            for (int c = 0; c < 12; ++c) gp[c] = 0.f;
          }
          const uint2 pr = rows.pairs[jj];
          float4* row = rows.row[pr.y + __popc(pr.x & lanemask_lt())];
          row[0] = make_float4(gp[0], gp[1], gp[2], gp[3]);
          row[1] = make_float4(gp[4], gp[5], gp[6], gp[7]);
          row[2] = make_float4(gp[8], gp[9], gp[10], gp[11]);
        }
        flush_rows<RGB4, MAYBE_GRID>(rows, __popc(used), lane, out);
      }
    }
  }
}

}  // namespace svr
