// Adjoint kernels of the FP32 path (sm_100a): the exact transposes of the
// forward stages, for gradients with respect to the raw readings and the
// filter taps. No counterpart in the reference, whose fct_wfbp has no
// backward pass; each kernel states the forward loop it transposes.
//
// None of them uses atomics: every output element is owned by one thread,
// which gathers the forward contributions that reach it (so results do not
// depend on scheduling).
#include "wfbp_internal.h"

#include <math.h>

#include <algorithm>

#include "bp_math.cuh"
#include "rebin_sample.cuh"

namespace {

// W(q) exactly as the forward backprojection (k_backproject.cu) evaluates it.
__device__ __forceinline__ float q_weight_fwd(float qh) {
  float t = __saturatef(fmaf(fabsf(qh), 2.5f, -1.5f));
  return fmaf(0.5f, __cosf(3.14159265f * t), 0.5f);
}

// ---------------------------------------------------------------------------
// backprojection adjoint
// ---------------------------------------------------------------------------
//
// Forward (k_bp, the reference-layout FP32 backprojection): for voxel
// (x, y, z) and half-turn angle t, with views j = t + k P/2,
//   vol += dtheta / sum_k W_k * sum_k W_k * bilinear(D_j; p_idx_j, q_idx_j).
// The gradient of one filtered sample D[j][r][c] is therefore
//   sum over voxels of g_vol * dtheta * W_j / sum_k W_k * hat(p_idx_j - c) * hat_row,
// where hat is the bilinear weight. k_bp_adjoint_band gathers it with the
// weights dtheta / sum_k W_k in a table; where no table fits,
// k_bp_adjoint_sums recomputes the sums.
constexpr int AD_CH = 128;

__device__ __forceinline__ float xcoord(const BPParams& p, int ix) {
  return ((float)ix - 0.5f * ((float)p.nx - 1.0f)) * p.fov / (float)p.nx + p.x0;
}
__device__ __forceinline__ float ycoord(const BPParams& p, int iy) {
  return ((float)iy - 0.5f * ((float)p.ny - 1.0f)) * p.fov / (float)p.ny + p.y0;
}

struct ViewGeo {
  float zt, asn, A, lt, inv, p_idx;  // asn = asin(p_hat / R), A = z_rot / 2 pi asn, lt = l_hat tan(cone), inv = 1 / lt
  bool valid_p;
};

__device__ __forceinline__ ViewGeo view_geo(const BPParams& p, float x, float y, float2 sc, float zt) {
  ViewGeo g;
  g.zt = zt;
  // roundings written out: a view's borderline samples must fall the same way
  // in every kernel, whatever the compiler hoists
  const float p_hat = fmaf(x, sc.x, -__fmul_rn(y, sc.y));
  // the forward's short forms (bp_math.cuh): hardware square root and
  // reciprocal, arcsine from its series
  const float l_hat = fmaf(-y, sc.x, fmaf(-x, sc.y, bp_sqrt(fmaf(-p_hat, p_hat, p.R2))));
  g.asn = bp_asin(p.rR * p_hat);
  g.A = p.zr2pi * g.asn;
  g.lt = l_hat * p.tanc;
  g.inv = bp_rcp(g.lt);
  g.p_idx = p.kp - fmaf(p_hat, p.ps, p.c0);
  const float pf = floorf(g.p_idx);
  g.valid_p = pf >= 0.0f && ceilf(g.p_idx) <= p.ncm2;
  return g;
}

// Q weight of view geometry g at slice z (0 where the forward skips it).
__device__ __forceinline__ float view_weight(const BPParams& p, const ViewGeo& g, float z, float* q_idx_out) {
  const float dz = z - g.zt;
  const float qh = __fmul_rn(fmaf(p.zr2pi, g.asn, dz), g.inv);
  const float q_idx = __fmul_rn(__fadd_rn(qh, 1.0f), p.hn);
  *q_idx_out = q_idx;
  const bool ok = g.valid_p && fabsf(dz) <= p.z_rot && q_idx >= 0.0f && q_idx <= p.nrm2;
  return ok ? q_weight_fwd(qh) : 0.0f;
}

// The views of one half-turn angle lie pi apart, so they cross the image along
// the same axis: p_hat = x sin - y cos changes faster along x when
// |sin| >= |cos|. That axis is the angle's inner axis u, the other v.
__device__ __forceinline__ bool inner_is_x(float2 sc) { return fabsf(sc.x) >= fabsf(sc.y); }

// Weights G[t - t0][s][v][u] = dtheta / sum_k W_k of half-turn angles t0 .. (0
// where no half turn contributes, as the forward's NaN voxel has no
// gradient). A thread takes one voxel column and 32 slices of one angle, lanes
// along u: it computes the column's geometry for the views whose cone reaches
// the slices and sums the weights of every slice in the forward's order. Bound by
// instruction issue (97.5 % of cycles; 16 rows, 256 x 256 x 26: 5.6 ms).
constexpr int AN_WARPS = 8;

__global__ void __launch_bounds__(AN_WARPS * 32)
k_bp_adjoint_scale(float* __restrict__ G, const float2* __restrict__ view_sc, const float* __restrict__ view_z,
                   const float* __restrict__ zslices, BPParams p, int t0, float reach, int nv_max) {
  extern __shared__ float2 s_geo[];  // [nv_max][threads] (inv, asn); then float [nv_max] table positions, [32] slices
  float2* geo = s_geo + threadIdx.x;
  float* zts = reinterpret_cast<float*>(s_geo + (size_t)AN_WARPS * nv_max * 32);
  float* zs = zts + nv_max;
  const int lane = threadIdx.x % 32;
  const int t = t0 + (int)blockIdx.y, s0 = blockIdx.z * 32, ns = min(32, p.nz - s0);
  if (threadIdx.x < 32) zs[threadIdx.x] = __ldg(zslices + s0 + min((int)threadIdx.x, ns - 1));
  __syncthreads();
  float zmn = zs[min(lane, ns - 1)], zmx = zmn;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    zmn = fminf(zmn, __shfl_xor_sync(0xffffffffu, zmn, o));
    zmx = fmaxf(zmx, __shfl_xor_sync(0xffffffffu, zmx, o));
  }
  const bool ux = inner_is_x(__ldg(view_sc + t));
  const int nu = ux ? p.nx : p.ny;
  const long plane = (long)p.nx * p.ny, col = (long)blockIdx.x * (AN_WARPS * 32) + threadIdx.x;
  const int u = (int)(col % nu), v = (int)(col / nu);
  const float x = xcoord(p, ux ? u : v), y = ycoord(p, ux ? v : u);
  const bool active = col < plane && !(x * x + y * y > p.fov_half2);
  int n = 0;
  for (int k = 0; k < p.K; k++) {
    const int j = t + k * p.P2;
    const float zt = __ldg(view_z + j);
    // beyond the cone's reach (or z_rot) of all these slices every weight is 0
    if (zt < zmn - reach || zt > zmx + reach || n >= nv_max) continue;
    const ViewGeo g = view_geo(p, x, y, __ldg(view_sc + j), zt);
    // an invalid column: no row coordinate
    geo[n * (AN_WARPS * 32)] = make_float2(g.inv, active && g.valid_p ? g.asn : __int_as_float(0x7fc00000));
    if (threadIdx.x == 0) zts[n] = zt;
    n++;
  }
  __syncthreads();
  if (col >= plane) return;
  float* out = G + ((size_t)blockIdx.y * p.nz + s0) * plane + col;
  for (int i = 0; i < ns; i++, out += plane) {
    const float z = zs[i];
    float aw = 0.0f;
    for (int a = 0; a < n; a++) {
      const float2 ga = geo[a * (AN_WARPS * 32)];
      const float dz = z - zts[a];
      const float qh = __fmul_rn(fmaf(p.zr2pi, ga.y, dz), ga.x);
      const float q_idx = __fmul_rn(__fadd_rn(qh, 1.0f), p.hn);
      const bool ok = fabsf(dz) <= p.z_rot && q_idx >= 0.0f && q_idx <= p.nrm2;
      aw += ok ? q_weight_fwd(qh) : 0.0f;
    }
    *out = aw > 0.0f ? p.dtheta * (1.0f / aw) : 0.0f;
  }
}

// Gather with the weight table. A CTA owns one view and a run of CH channels
// and visits the voxels whose p_idx lies in its channels (a band across the
// image) or in the channel before them (whose voxels share their sample with
// the run's first channel). Its warps take the image rows v in turn; lanes are
// VL consecutive voxels u of the row inside the band, times 32 / VL shares of
// the slices in the view's cone, which they walk together. A slice's
// g_vol dtheta / sum_k W_k W_j goes to the rows r and r + 1 around its row
// coordinate, weighted for the voxel's channel c (1 - frac(p_idx)) and for
// c + 1 (frac(p_idx)), into the warp's own window [row][channel] of (c, c + 1)
// sums in shared memory. Neighbouring voxels are p_step channels apart and
// the shares' slices a share's length: with p_step > 1 and shares of a few
// rows no two lanes write the same sums at a time, else lanes take turns. At
// the end the warps' windows are added in a fixed order: no atomics, nothing
// depends on scheduling. Weights and gradient are read along u in full lines,
// the next slice's before this one's arithmetic. Issue is the busiest unit (76 %
// of cycles at three CTAs per SM; 16 rows, 256 x 256 x 26: 9.5 ms, 13.1 before).
constexpr int AB_WARPS = 8;

__global__ void __launch_bounds__(AB_WARPS * 32, 3)
k_bp_adjoint_band(const float* __restrict__ gvol_x, const float* __restrict__ gvol_y, const float* __restrict__ G,
                  float* __restrict__ gD, const float2* __restrict__ view_sc, const float* __restrict__ view_z,
                  const float* __restrict__ zslices, BPParams p, float z0, float dzs, int t0, float reach, int CH) {
  extern __shared__ float2 s_win[];  // [AB_WARPS][nr][CH + 1] (sum for c, sum for c + 1); then float [nz] slices
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int tl = blockIdx.y / p.K, j = t0 + tl + (blockIdx.y % p.K) * p.P2;
  const int W = CH + 1, wsize = W * p.nr, c_base = blockIdx.x * CH - 1;  // channel of a window's first column
  float* s_z = reinterpret_cast<float*>(s_win + (size_t)AB_WARPS * wsize);
  const int win = warp * wsize;
  for (int e = threadIdx.x; e < AB_WARPS * wsize; e += AB_WARPS * 32) s_win[e] = make_float2(0.0f, 0.0f);
  for (int e = threadIdx.x; e < p.nz; e += AB_WARPS * 32) s_z[e] = __ldg(zslices + e);
  __syncthreads();

  const float zt = __ldg(view_z + j);
  const float za0 = s_z[0], za1 = s_z[p.nz - 1];
  if (!(zt < fminf(za0, za1) - reach || zt > fmaxf(za0, za1) + reach)) {  // else no slice is in the cone's reach
    const float2 sc = __ldg(view_sc + j);
    const bool ux = inner_is_x(__ldg(view_sc + t0 + tl));
    const int nu = ux ? p.nx : p.ny, nv = ux ? p.ny : p.nx;
    const size_t plane = (size_t)p.nx * p.ny;
    const float* Gt = G + (size_t)tl * p.nz * plane;
    const float* gv = ux ? gvol_x : gvol_y;
    // p_idx in [c_base, c_base + CH + 1) <=> p_hat in this interval (widened
    // by a rounding margin; the exact forward test below decides)
    const float ph_a = (p.kp - p.c0 - ((float)c_base + (float)(CH + 1))) / p.ps,
                ph_b = (p.kp - p.c0 - (float)c_base) / p.ps;
    const float marg = 0.02f / p.ps + 1e-3f * p.fov / (float)p.nx;
    const float plo = fminf(ph_a, ph_b) - marg, phi = fmaxf(ph_a, ph_b) + marg;
    const float su = p.fov / (float)nu, num = 0.5f * ((float)nu - 1.0f);
    // candidate ranges through reciprocals computed once: their rounding (a few
    // 1e-5 mm) stays far inside the margin
    const float r_sc = 1.0f / (ux ? sc.x : sc.y), r_s = 1.0f / su;
    const float r_dzs = dzs != 0.0f ? 1.0f / dzs : 0.0f, top_q = p.nrm2 / p.hn - 1.0f;
    // voxels a few lanes apart that are sure to lie in different channels
    const float p_step = p.ps * su * fabsf(ux ? sc.x : sc.y);
    // lanes per run of voxels: the split with the fewest instructions for the
    // band's width, a run costing its geometry (about 110) and 40 a slice
    int VL = 32;
    {
      const float width = fminf((float)W / p_step + 1.0f, (float)nu), slices = fminf((float)p.nr, (float)p.nz);
      float best = 3.0e38f;
      for (int l = 32; l >= 4; l >>= 1) {
        const float cost = ceilf(width / (float)l) * (110.0f + 40.0f * ceilf(slices * (float)l / 32.0f));
        if (cost < best) {
          best = cost;
          VL = l;
        }
      }
    }
    const int vl = lane & (VL - 1), share = lane / VL, shares = 32 / VL;
    const int v_turns = min((int)ceilf(fminf(1.001f / p_step, 64.0f)), VL), v_turn = vl % v_turns;
    const float r_hd = r_dzs / p.hn;

    for (int v = warp; v < nv; v += AB_WARPS) {
      const float cv = ux ? ycoord(p, v) : xcoord(p, v);
      float a, b;
      if (ux) {
        a = (plo + cv * sc.y) * r_sc - p.x0;
        b = (phi + cv * sc.y) * r_sc - p.x0;
      } else {
        a = (cv * sc.x - phi) * r_sc - p.y0;
        b = (cv * sc.x - plo) * r_sc - p.y0;
      }
      const int u_lo = max(0, (int)floorf(fminf(a, b) * r_s + num));
      const int u_hi = min(nu - 1, (int)ceilf(fmaxf(a, b) * r_s + num));
      for (int u0 = u_lo; u0 <= u_hi; u0 += VL) {
        const int u = u0 + vl;
        const float x = ux ? xcoord(p, u) : cv, y = ux ? cv : ycoord(p, u);
        const ViewGeo g = view_geo(p, x, y, sc, zt);
        const float pf = floorf(g.p_idx), wp = g.p_idx - pf, h0 = 1.0f - wp;
        const int c = (int)pf - c_base;
        const bool own = u <= u_hi && !(x * x + y * y > p.fov_half2) && g.valid_p && c >= 0 && c <= CH;
        // slices that can pass this view's tests: |z - zt| <= z_rot and q_idx in
        // [0, nr - 2], a z interval around zt - A (evenly spaced slices lie
        // within 1e-3 of a slice of z0 + s dzs)
        const float za = zt - g.A - g.lt, zb = zt - g.A + top_q * g.lt;
        const float zlo = fmaxf(fminf(za, zb), zt - p.z_rot), zhi = fminf(fmaxf(za, zb), zt + p.z_rot);
        int s_lo = 0, s_hi = p.nz - 1;
        if (dzs != 0.0f) {
          const float fa = (zlo - z0) * r_dzs, fb = (zhi - z0) * r_dzs;
          s_lo = max(0, (int)ceilf(fminf(fa, fb) - 0.01f));
          s_hi = min(p.nz - 1, (int)floorf(fmaxf(fa, fb) + 0.01f));
        }
        const bool use = own && !(zlo > zhi) && s_lo <= s_hi;
        // the lanes' slices together
        const int first = __reduce_min_sync(0xffffffffu, use ? s_lo : p.nz);
        const int last = __reduce_max_sync(0xffffffffu, use ? s_hi : -1);
        if (first > last) continue;
        // a share's slices; rows between the shares' slices at a time: len / rows_max
        const int len = (last - first + shares) / shares;
        const unsigned rows_max = __reduce_max_sync(0xffffffffu, __float_as_uint(use ? fabsf(g.lt * r_hd) : 0.0f));
        const bool apart = dzs != 0.0f && (float)len > 2.1f * __uint_as_float(rows_max);
        const int turns = apart ? v_turns : v_turns * shares, my_turn = apart ? v_turn : v_turn + v_turns * share;
        const int s_first = first + share * len;
        const float asn = use ? g.asn : __int_as_float(0x7fc00000);  // NaN: no slice passes the row test
        const float inv = g.inv;
        const size_t at = (size_t)min(s_first, last) * plane + (size_t)v * nu + min(u, nu - 1);
        const float *pw = Gt + at, *pg = gv + at;
        float w = __ldg(pw), gn = __ldg(pg);
        const int col = win + (use ? c : 0);
        for (int s = s_first; s < s_first + len; s++) {
          const bool in = s <= last;
          const float dz = s_z[min(s, last)] - zt, wc = in ? w : 0.0f, gc = gn;
          if (s < last) {
            pw += plane;
            pg += plane;
            w = __ldg(pw);
            gn = __ldg(pg);
          }
          const float qh = __fmul_rn(fmaf(p.zr2pi, asn, dz), inv);
          const float q = __fmul_rn(__fadd_rn(qh, 1.0f), p.hn);
          const bool ok = fabsf(dz) <= p.z_rot && q >= 0.0f && q <= p.nrm2 && wc != 0.0f;
          const float vv = gc * wc * q_weight_fwd(qh);  // g_vol dtheta / sum_k W_k (cuda_kernels.cuh:283) W_j
          const float qf = floorf(q), hi = vv * (q - qf), lo = vv - hi;
          const int at0 = col + (int)qf * W, at1 = at0 + W;
          auto add = [&](bool mine) {
            if (mine) {
              const float2 d = s_win[at0], e = s_win[at1];
              s_win[at0] = make_float2(fmaf(lo, h0, d.x), fmaf(lo, wp, d.y));
              s_win[at1] = make_float2(fmaf(hi, h0, e.x), fmaf(hi, wp, e.y));
            }
            __syncwarp();
          };
          if (turns == 1) {
            add(ok);
          } else {
            for (int k = 0; k < turns; k++) add(ok && my_turn == k);
          }
        }
        __syncwarp();  // other lanes have these channels next
      }
    }
  }
  __syncthreads();
  // channel c = its own sums + those that channel c - 1 has for it, over the windows in order
  float* out = gD + (size_t)j * p.nr * p.nch + blockIdx.x * CH;
  const int nc = min(CH, p.nch - (int)blockIdx.x * CH);
  for (int e = threadIdx.x; e < nc * p.nr; e += AB_WARPS * 32) {
    const int c = e % nc, r = e / nc;
    float own = 0.0f, next = 0.0f;
    for (int k = 0; k < AB_WARPS; k++) {
      own += s_win[(size_t)k * wsize + r * W + c + 1].x;
      next += s_win[(size_t)k * wsize + r * W + c].y;
    }
    out[(size_t)r * p.nch + c] = own + next;
  }
}

// Gather without a table: a CTA owns one view and AD_CH - 1 channels; thread c
// walks the voxels of its channel (as above), recomputes sum_k W_k of
// every (voxel, slice) from the forward's expressions in the forward's order,
// and adds the row contributions to two accumulators of its own in shared
// memory, for channel c and for channel c + 1. At the end channel c = own(c) +
// next(c - 1), in that order; the CTA's first thread only supplies
// next(c0 - 1) for its neighbour.
__global__ void __launch_bounds__(AD_CH, 8)
k_bp_adjoint_sums(const float* __restrict__ gvol, float* __restrict__ gD, const float2* __restrict__ view_sc,
                  const float* __restrict__ view_z, const float* __restrict__ zslices, BPParams p, float z0,
                  float dzs) {
  extern __shared__ float2 acc2[];  // [nr][AD_CH]: (own channel, next channel) of thread cl
  const int j = blockIdx.y;
  const int cl = threadIdx.x;
  const int c = blockIdx.x * (AD_CH - 1) - 1 + cl;  // channels c0 - 1 .. c0 + AD_CH - 2
  for (int r = 0; r < p.nr; r++) acc2[r * AD_CH + cl] = make_float2(0.0f, 0.0f);

  const int t = j % p.P2, kj = j / p.P2;
  if (kj < p.K && c >= 0 && c < p.nch) {
    const float2 sc = __ldg(view_sc + j);
    const float zt = __ldg(view_z + j);
    // p_idx in [c, c + 1) <=> p_hat in this interval (widened by a rounding
    // margin; the exact forward test below decides)
    const float ph_a = (p.kp - p.c0 - ((float)c + 1.0f)) / p.ps, ph_b = (p.kp - p.c0 - (float)c) / p.ps;
    const float marg = 0.02f / p.ps + 1e-3f * p.fov / (float)p.nx;
    const float plo = fminf(ph_a, ph_b) - marg, phi = fmaxf(ph_a, ph_b) + marg;
    const float sx = p.fov / (float)p.nx, sy = p.fov / (float)p.ny;
    const float nxm = 0.5f * ((float)p.nx - 1.0f), nym = 0.5f * ((float)p.ny - 1.0f);
    const bool along_y = fabsf(sc.x) >= fabsf(sc.y);  // p_hat = x sin - y cos: solve for x per row y
    const int n_outer = along_y ? p.ny : p.nx;
    // the candidate range of each row through reciprocals computed once: their
    // rounding (a few 1e-5 mm) stays far inside the margin, and the exact
    // channel test below decides which voxels the thread owns
    const float r_sc = 1.0f / (along_y ? sc.x : sc.y), r_sx = 1.0f / sx, r_sy = 1.0f / sy;
    for (int o = 0; o < n_outer; o++) {
      int i_lo, i_hi;
      if (along_y) {
        const float y = ycoord(p, o);
        float xa = (plo + y * sc.y) * r_sc, xb = (phi + y * sc.y) * r_sc;
        if (xa > xb) { const float tt = xa; xa = xb; xb = tt; }
        i_lo = max(0, (int)floorf((xa - p.x0) * r_sx + nxm));
        i_hi = min(p.nx - 1, (int)ceilf((xb - p.x0) * r_sx + nxm));
      } else {
        const float x = xcoord(p, o);
        float ya = (x * sc.x - phi) * r_sc, yb = (x * sc.x - plo) * r_sc;
        if (ya > yb) { const float tt = ya; ya = yb; yb = tt; }
        i_lo = max(0, (int)floorf((ya - p.y0) * r_sy + nym));
        i_hi = min(p.ny - 1, (int)ceilf((yb - p.y0) * r_sy + nym));
      }
      for (int in = i_lo; in <= i_hi; in++) {
        const int ix = along_y ? in : o, iy = along_y ? o : in;
        const float x = xcoord(p, ix), y = ycoord(p, iy);
        if (x * x + y * y > p.fov_half2) continue;  // cuda_kernels.cuh:220
        {
          // the channel test first (three FMAs), the square root, arcsine
          // and division of the geometry only for the voxel that passes it
          const float ph = x * sc.x - y * sc.y;
          if ((int)floorf(p.kp - (ph * p.ps + p.c0)) != c) continue;
        }
        const ViewGeo g = view_geo(p, x, y, sc, zt);
        if (!g.valid_p) continue;
        const float pf = floorf(g.p_idx), wp = g.p_idx - pf;
        if ((int)pf != c) continue;
        const float h0 = 1.0f - wp;  // channel c; channel c + 1 gets wp
        // slices that can pass this view's tests: |z - zt| <= z_rot and
        // q_idx in [0, nr-2], a z interval around zt - A
        const float za = zt - g.A - g.lt, zb = zt - g.A + (p.nrm2 / p.hn - 1.0f) * g.lt;
        const float zlo = fmaxf(fminf(za, zb), zt - p.z_rot), zhi = fminf(fmaxf(za, zb), zt + p.z_rot);
        if (zlo > zhi) continue;
        int s_lo, s_hi;
        if (p.nz == 1 || dzs == 0.0f) {
          s_lo = 0;
          s_hi = p.nz - 1;
        } else {
          float fa = (zlo - z0) / dzs, fb = (zhi - z0) / dzs;
          if (fa > fb) { const float tt = fa; fa = fb; fb = tt; }
          s_lo = max(0, (int)floorf(fa) - 1);
          s_hi = min(p.nz - 1, (int)ceilf(fb) + 1);
        }
        for (int s = s_lo; s <= s_hi; s++) {
          const float z = __ldg(zslices + s);
          float q_idx;
          const float Wj = view_weight(p, g, z, &q_idx);
          if (Wj == 0.0f) continue;
          const float gv = __ldg(gvol + ((size_t)s * p.ny + iy) * p.nx + ix);
          if (gv == 0.0f) continue;
          // sum of the weights of all half turns, in the forward's order
          float aw = 0.0f;
          for (int k = 0; k < p.K; k++) {
            const int jj = t + k * p.P2;
            if (jj == j) {
              aw += Wj;
              continue;
            }
            const float ztk = __ldg(view_z + jj);
            if (!(fabsf(z - ztk) <= p.z_rot)) continue;
            const ViewGeo gk = view_geo(p, x, y, __ldg(view_sc + jj), ztk);
            float qk;
            aw += view_weight(p, gk, z, &qk);
          }
          const float scaled = gv * (p.dtheta * (1.0f / aw));  // cuda_kernels.cuh:283
          const float sw = scaled * Wj;
          const float c0v = sw * h0, c1v = sw * wp;
          const float qf = floorf(q_idx), wq = q_idx - qf;
          const int r = min(max((int)qf, 0), p.nr - 2);
          float2* a0 = acc2 + r * AD_CH + cl;
          float2 v0 = a0[0], v1 = a0[AD_CH];
          v0.x += c0v * (1.0f - wq);
          v0.y += c1v * (1.0f - wq);
          v1.x += c0v * wq;
          v1.y += c1v * wq;
          a0[0] = v0;
          a0[AD_CH] = v1;
        }
      }
    }
  }
  __syncthreads();
  if (cl >= 1 && c < p.nch) {
    float* out = gD + (size_t)j * p.nr * p.nch + c;
    for (int r = 0; r < p.nr; r++) out[(size_t)r * p.nch] = acc2[r * AD_CH + cl].x + acc2[r * AD_CH + cl - 1].y;
  }
}

// out[s][x][y] = in[s][y][x], 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256)
k_transpose_slices(const float* __restrict__ in, float* __restrict__ out, int nx, int ny) {
  __shared__ float tile[32][33];
  const size_t slice = (size_t)blockIdx.z * nx * ny;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32, tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  for (int i = ty; i < 32; i += 8)
    if (x0 + tx < nx && y0 + i < ny) tile[i][tx] = __ldg(in + slice + (size_t)(y0 + i) * nx + x0 + tx);
  __syncthreads();
  for (int i = ty; i < 32; i += 8)
    if (x0 + i < nx && y0 + tx < ny) out[slice + (size_t)(x0 + i) * ny + y0 + tx] = tile[tx][i];
}

// ---------------------------------------------------------------------------
// thickening adjoint
// ---------------------------------------------------------------------------
// Forward: vol[r] = sum_n w_rn vol_n / ws_r over the CSR of requested slice r.
// Transposed CSR (built on the host): native slice n lists (r, w_rn / ws_r).
__global__ void k_thicken_adjoint(const float* __restrict__ gvol, float* __restrict__ gvn, const int* __restrict__ off,
                                  const int* __restrict__ ridx, const float* __restrict__ w, int nxy, int nz) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)nxy * nz) return;
  const int n = (int)(i / nxy);
  const long px = i % nxy;
  float acc = 0.0f;
  for (int e = off[n]; e < off[n + 1]; e++) acc = fmaf(w[e], gvol[(size_t)ridx[e] * nxy + px], acc);
  gvn[i] = acc;
}

// ---------------------------------------------------------------------------
// rebin adjoint
// ---------------------------------------------------------------------------
// Forward (rebin_sample, k_stages.cu): output sample (v, i, c) is the
// bilinear texel sample of raw row nr-1-i at sheet column bidx[c] and sheet
// view aidx(v, c), clamp addressing, sheet column x <- raw channel nch-1-x.
// Column lists: sheet column x receives weight wx from channel c when one of
// c's two clamped column taps is x (both taps, when they clamp to the same
// column). Built once per context by k_rebin_adj_cols.
__global__ void k_rebin_adj_cols(const float* __restrict__ bidx_t, int nch, int q8, int* __restrict__ cnt,
                                 int* __restrict__ cidx, float* __restrict__ cw, int maxl, int* __restrict__ err) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= nch) return;
  int n = 0;
  // bidx is monotone in c with slope >= 1, so the channels reaching x lie near x
  for (int c = 0; c < nch; c++) {
    const float b = bidx_t[c];
    if (isnan(b)) continue;
    const float xb = (b + 0.5f) - 0.5f;
    const float fx = floorf(xb);
    float ax = xb - fx;
    if (q8) ax = rintf(ax * 256.0f) * (1.0f / 256.0f);
    const int x0 = min(max((int)fx, 0), nch - 1), x1 = min(max((int)fx + 1, 0), nch - 1);
    float wgt = 0.0f;
    if (x0 == x) wgt += 1.0f - ax;
    if (x1 == x) wgt += ax;
    if (x0 != x && x1 != x) continue;
    if (n == maxl) {
      atomicOr(err, WFBP_ERRBIT_ADJ_LIST);
      break;
    }
    cidx[x * maxl + n] = c;
    cw[x * maxl + n] = wgt;
    n++;
  }
  cnt[x] = n;
}

// Weight with which sheet view y enters output view v's sample of channel
// (fan angle beta): the transposed row taps of rebin_sample.
__device__ __forceinline__ float rebin_view_weight(int v, int y, float beta, float dth, int V, int q8, int voff) {
  const float theta = (float)(v + voff) * dth;
  const float alpha = theta - beta;
  const float aidx = alpha / dth;
  const float yb = (aidx + 0.5f) - 0.5f;
  const float fy = floorf(yb);
  float ay = yb - fy;
  if (q8) ay = rintf(ay * 256.0f) * (1.0f / 256.0f);
  const int y0 = min(max((int)fy - voff, 0), V - 1), y1 = min(max((int)fy + 1 - voff, 0), V - 1);
  float w = 0.0f;
  if (y0 == y) w += 1.0f - ay;
  if (y1 == y) w += ay;
  return w;
}

// One thread per raw channel of a reading and RA_ROWS of its detector rows: the
// view weights of a channel do not depend on the row, so they are computed
// once, and the rows' independent loads hide each other's latency (a thread
// per sample spent its time on the weights: 16 rows of 672 channels 1.03 ms,
// now 0.37; 64 rows of 888 channels, 2460 readings, 3.66 ms, now 1.00, of
// which moving its 1.1 GB takes 0.17). Lanes are consecutive raw channels,
// whose sources are consecutive channels.
constexpr int RA_ROWS = 8, RA_CH = 128;

__global__ void __launch_bounds__(RA_CH)
k_rebin_adjoint(const float* __restrict__ gR, float* __restrict__ graw, const float* __restrict__ beta_t,
                const int* __restrict__ cnt, const int* __restrict__ cidx, const float* __restrict__ cw, int maxl,
                RebinParams p) {
  const int y = blockIdx.x, xr = blockIdx.y * RA_CH + threadIdx.x, i0 = blockIdx.z * RA_ROWS;
  if (xr >= p.nch) return;
  const int x = p.nch - 1 - xr;  // sheet column
  const int rows = min(RA_ROWS, p.nr - i0);  // sheet rows i0 .. of the output
  float acc[RA_ROWS];
#pragma unroll
  for (int k = 0; k < RA_ROWS; k++) acc[k] = 0.0f;
  const int n = cnt[x];
  for (int e = 0; e < n; e++) {
    const int c = cidx[x * maxl + e];
    const float wx = cw[x * maxl + e];
    const float beta = __ldg(beta_t + c);
    const float sh = beta / p.dth;  // aidx ~ v - sh
    int v_lo = (int)floorf((float)y + sh) - 2, v_hi = (int)ceilf((float)y + sh) + 2;
    if (y == 0) v_lo = 0;            // every view whose taps clamp to the first reading
    if (y == p.V - 1) v_hi = p.V - 1;  // ... or to the last
    if (y == 0) v_hi = max(v_hi, (int)ceilf(sh) + 2);
    if (y == p.V - 1) v_lo = min(v_lo, (int)floorf((float)(p.V - 1) + sh) - 2);
    v_lo = max(v_lo, 0);
    v_hi = min(v_hi, p.V - 1);
    float sum[RA_ROWS];
#pragma unroll
    for (int k = 0; k < RA_ROWS; k++) sum[k] = 0.0f;
    for (int v = v_lo; v <= v_hi; v++) {
      const float wy = rebin_view_weight(v, y, beta, p.dth, p.V, p.q8, p.voff);
      if (wy == 0.0f) continue;
      const float* g = gR + ((size_t)v * p.nr + i0) * p.nch + c;
#pragma unroll
      for (int k = 0; k < RA_ROWS; k++)
        if (k < rows) sum[k] = fmaf(wy, __ldg(g + (size_t)k * p.nch), sum[k]);
    }
#pragma unroll
    for (int k = 0; k < RA_ROWS; k++) acc[k] = fmaf(wx, sum[k], acc[k]);
  }
  // sheet row i is raw row nr - 1 - i
  float* out = graw + ((size_t)y * p.nr + (p.nr - 1 - i0)) * p.nch + xr;
#pragma unroll
  for (int k = 0; k < RA_ROWS; k++)
    if (k < rows) out[-(ptrdiff_t)k * p.nch] = acc[k];
}

// ---------------------------------------------------------------------------
// filter-tap gradient, with the rebinned rows recomputed on the fly
// ---------------------------------------------------------------------------
// Forward: y[n] = sum_m h[|n - m|] x[m] over the nch channels of each row.
// dL/dh[0] = sum_rows sum_n g[n] x[n]; dL/dh[d] = sum_rows sum_n g[n] (x[n-d] + x[n+d]).
// A CTA takes TG_ROWS rows and recomputes their rebinned samples x from the
// raw readings into shared memory (nothing of the rebinned array is stored).
// Thread (tap group, row) correlates its row for TG_TAPS consecutive taps d0..
// d0+3: one gradient load and two sliding-window loads of x feed 8 FMAs per
// channel. The rows of a CTA (8 consecutive lanes) are summed with shuffles
// in a fixed order, and the per-CTA partial sums by k_taps_reduce, so the
// result does not depend on scheduling.
constexpr int TG_ROWS = 8;
constexpr int TG_TAPS = 4;
constexpr int TG_THREADS = 128;  // 16 tap groups x 8 rows

__global__ void __launch_bounds__(TG_THREADS)
k_taps_grad(const float* __restrict__ raw, const float* __restrict__ gY, const float* __restrict__ beta_t,
            const float* __restrict__ bidx_t, RebinParams p, int ntaps, float* __restrict__ partial) {
  extern __shared__ float sm[];
  const int ns = p.nch | 1;               // odd row stride: the 8 rows of a warp fall in different banks
  float* xs = sm;                         // [TG_ROWS][ns]
  float* gs = sm + TG_ROWS * ns;          // [TG_ROWS][ns]
  const long m0 = (long)blockIdx.x * TG_ROWS;
  const long M = (long)p.V * p.nr;
  const int rows = (int)min((long)TG_ROWS, M - m0);
  for (int e = threadIdx.x; e < TG_ROWS * p.nch; e += TG_THREADS) {
    const int rr = e / p.nch, c = e % p.nch;
    const long m = m0 + rr;
    float xv = 0.0f, gv = 0.0f;  // rows past the end contribute nothing
    if (rr < rows) {
      const int v = (int)(m / p.nr), i = (int)(m % p.nr);
      xv = wfbp_rebin_sample(raw, p, __ldg(bidx_t + c), __ldg(beta_t + c), v, i);
      gv = __ldg(gY + m * p.nch + c);
    }
    xs[rr * ns + c] = xv;
    gs[rr * ns + c] = gv;
  }
  __syncthreads();
  const int rr = threadIdx.x % TG_ROWS;
  const float* xr = xs + rr * ns;
  const float* gr = gs + rr * ns;
  const int ngroups = (ntaps + TG_TAPS - 1) / TG_TAPS;
  // every lane of a warp runs the same number of group iterations (the shuffles below)
  for (int g0 = 0; g0 < ngroups; g0 += TG_THREADS / TG_ROWS) {
    const int gi = g0 + threadIdx.x / TG_ROWS;
    const int d0 = gi * TG_TAPS;
    float af[TG_TAPS], ab[TG_TAPS], wf[TG_TAPS], wb[TG_TAPS];
#pragma unroll
    for (int k = 0; k < TG_TAPS; k++) {
      af[k] = ab[k] = 0.0f;
      wf[k] = 0.0f;  // wf[k] = x[n - d0 - k]
      const int jb = d0 + k;
      wb[k] = jb < p.nch ? xr[jb] : 0.0f;  // wb[k] = x[n + d0 + k]
    }
    if (gi < ngroups) {
      for (int n = 0; n < p.nch; n++) {
        const float g = gr[n];
        // slide the forward window: wf[k] = x[n - d0 - k]
#pragma unroll
        for (int k = TG_TAPS - 1; k > 0; k--) wf[k] = wf[k - 1];
        wf[0] = n - d0 >= 0 ? xr[n - d0] : 0.0f;
#pragma unroll
        for (int k = 0; k < TG_TAPS; k++) {
          af[k] = fmaf(g, wf[k], af[k]);
          ab[k] = fmaf(g, wb[k], ab[k]);
        }
        // slide the backward window to n + 1: wb[k] = x[n + 1 + d0 + k]
#pragma unroll
        for (int k = 0; k < TG_TAPS - 1; k++) wb[k] = wb[k + 1];
        const int jb = n + 1 + d0 + TG_TAPS - 1;
        wb[TG_TAPS - 1] = jb < p.nch ? xr[jb] : 0.0f;
      }
    }
#pragma unroll
    for (int k = 0; k < TG_TAPS; k++) {
      // dL/dh[0] counts the product once, dL/dh[d > 0] both neighbours
      float v = d0 + k == 0 ? af[k] : af[k] + ab[k];
#pragma unroll
      for (int o = TG_ROWS / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (rr == 0 && gi < ngroups && d0 + k < ntaps) partial[(size_t)blockIdx.x * ntaps + d0 + k] = v;
    }
  }
}

// One CTA per tap: thread i sums partials i, i + TR_THREADS, ... in double,
// then a tree over the threads in a fixed order (deterministic).
constexpr int TR_THREADS = 256;

__global__ void __launch_bounds__(TR_THREADS)
k_taps_reduce(const float* __restrict__ partial, int nblk, int ntaps, float* __restrict__ out) {
  __shared__ double red[TR_THREADS];
  const int d = blockIdx.x;
  double acc = 0.0;
  for (int b = threadIdx.x; b < nblk; b += TR_THREADS) acc += (double)partial[(size_t)b * ntaps + d];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = TR_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[d] = (float)red[0];
}

}  // namespace

namespace {
// Channels of a CTA: the windows of all its warps together at most 60 KB, so
// that three CTAs share an SM (up to 64 rows; taller detectors take 12
// channels and fewer CTAs).
int band_channels(int nr) { return std::max(12, std::min(63, 60 * 1024 / (AB_WARPS * 8 * nr) - 1)); }

size_t band_smem(int nr, int nz) {
  return sizeof(float2) * (size_t)AB_WARPS * (band_channels(nr) + 1) * nr + sizeof(float) * (size_t)nz;
}

size_t scale_smem(int nv_max) {
  return (size_t)nv_max * (AN_WARPS * 32 * sizeof(float2) + sizeof(float)) + 32 * sizeof(float);
}
}  // namespace

bool bp_adjoint_table_ok(const BPParams& p, int nv_max) {
  return band_smem(p.nr, p.nz) <= 200 * 1024 && scale_smem(nv_max) <= 200 * 1024;
}

cudaError_t launch_bp_adjoint(const float* gvol, float* gD, const float2* sc, const float* vz, const float* zs,
                              const BPParams& p, float z0, float dzs, float* scale_table, int table_angles,
                              bool fill_table, float* gvol_t, float reach, int nv_max, cudaStream_t s) {
  cudaError_t e;
  if (!scale_table) {
    dim3 grid((unsigned)((p.nch + AD_CH - 2) / (AD_CH - 1)), (unsigned)p.V);
    const size_t smem = (size_t)p.nr * AD_CH * sizeof(float2);
    if (smem > 48 * 1024 && (e = cudaFuncSetAttribute(k_bp_adjoint_sums, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      (int)smem)) != cudaSuccess)
      return e;
    k_bp_adjoint_sums<<<grid, AD_CH, smem, s>>>(gvol, gD, sc, vz, zs, p, z0, dzs);
    return cudaGetLastError();
  }
  // the gradient volume with the voxels of a column next to each other, for the angles whose inner axis is y
  const dim3 tg((unsigned)((p.nx + 31) / 32), (unsigned)((p.ny + 31) / 32), (unsigned)p.nz);
  k_transpose_slices<<<tg, 256, 0, s>>>(gvol, gvol_t, p.nx, p.ny);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // the views the forward never reads
  const int used = p.K * p.P2;
  const size_t view = (size_t)p.nr * p.nch;
  if (used < p.V && (e = cudaMemsetAsync(gD + used * view, 0, sizeof(float) * view * (p.V - used), s)) != cudaSuccess)
    return e;
  const size_t an_smem = scale_smem(nv_max), ab_smem = band_smem(p.nr, p.nz);
  if ((e = cudaFuncSetAttribute(k_bp_adjoint_scale, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)an_smem)) !=
          cudaSuccess ||
      (e = cudaFuncSetAttribute(k_bp_adjoint_band, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ab_smem)) !=
          cudaSuccess)
    return e;
  const int ch = band_channels(p.nr);
  // one group of the table's angles after another, in launches that a grid's y takes
  const int most = std::max(1, 65535 / std::max(p.K, 1));
  for (int g0 = 0; g0 < p.P2; g0 += table_angles)
    for (int t0 = g0; t0 < std::min(p.P2, g0 + table_angles); t0 += most) {
      const int nt = std::min(most, std::min(p.P2, g0 + table_angles) - t0);
      float* G = scale_table + (size_t)(t0 - g0) * p.nz * p.nx * p.ny;
      if (fill_table) {
        const dim3 g((unsigned)(((long)p.nx * p.ny + AN_WARPS * 32 - 1) / (AN_WARPS * 32)), (unsigned)nt,
                     (unsigned)((p.nz + 31) / 32));
        k_bp_adjoint_scale<<<g, AN_WARPS * 32, an_smem, s>>>(G, sc, vz, zs, p, t0, reach, nv_max);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
      }
      const dim3 g((unsigned)((p.nch + ch - 1) / ch), (unsigned)(nt * p.K));
      k_bp_adjoint_band<<<g, AB_WARPS * 32, ab_smem, s>>>(gvol, gvol_t, G, gD, sc, vz, zs, p, z0, dzs, t0, reach, ch);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
  return cudaSuccess;
}

cudaError_t launch_thicken_adjoint(const float* gvol, float* gvn, const int* off, const int* ridx, const float* w,
                                   int nxy, int nz, cudaStream_t s) {
  const long n = (long)nxy * nz;
  k_thicken_adjoint<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(gvol, gvn, off, ridx, w, nxy, nz);
  return cudaGetLastError();
}

cudaError_t launch_rebin_adj_cols(const float* bidx, int nch, int q8, int* cnt, int* cidx, float* cw, int maxl,
                                  int* err, cudaStream_t s) {
  k_rebin_adj_cols<<<(nch + 127) / 128, 128, 0, s>>>(bidx, nch, q8, cnt, cidx, cw, maxl, err);
  return cudaGetLastError();
}

cudaError_t launch_rebin_adjoint(const float* gR, float* graw, const float* beta, const int* cnt, const int* cidx,
                                 const float* cw, int maxl, const RebinParams& p, cudaStream_t s) {
  const dim3 g((unsigned)p.V, (unsigned)((p.nch + RA_CH - 1) / RA_CH), (unsigned)((p.nr + RA_ROWS - 1) / RA_ROWS));
  k_rebin_adjoint<<<g, RA_CH, 0, s>>>(gR, graw, beta, cnt, cidx, cw, maxl, p);
  return cudaGetLastError();
}

int taps_grad_blocks(const RebinParams& p) { return (int)(((long)p.V * p.nr + TG_ROWS - 1) / TG_ROWS); }

cudaError_t launch_taps_gradient(const float* raw, const float* gY, const float* beta, const float* bidx,
                                 const RebinParams& p, int ntaps, float* partial, float* out, cudaStream_t s) {
  const int nblk = taps_grad_blocks(p);
  const size_t smem = (size_t)2 * TG_ROWS * (p.nch | 1) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_taps_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  k_taps_grad<<<nblk, TG_THREADS, smem, s>>>(raw, gY, beta, bidx, p, ntaps, partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_taps_reduce<<<ntaps, TR_THREADS, 0, s>>>(partial, nblk, ntaps, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// self-test of the bounded waits
// ---------------------------------------------------------------------------
#include "wait.cuh"

namespace {
// Waits on an mbarrier that nothing ever arrives at, with a limit of
// limit_ns; when the wait gives up (as it must) the error word is set to
// WFBP_ERR_TIMEOUT, exactly as a stalled pipeline in the production kernels
// reports itself.
__global__ void k_selftest_wait(int* err, unsigned long long limit_ns) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(&bar)), "r"(1));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0 && !wfbp_mbar_wait(&bar, 0, limit_ns)) atomicExch(err, WFBP_ERR_TIMEOUT);
}
}  // namespace

cudaError_t launch_selftest_wait(int* err, unsigned long long limit_ns, cudaStream_t s) {
  k_selftest_wait<<<1, 32, 0, s>>>(err, limit_ns);
  return cudaGetLastError();
}
