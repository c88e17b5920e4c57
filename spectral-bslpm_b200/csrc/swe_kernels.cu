// Shallow-water (SWE v2) velocity kernels, sm_100a: the two-field sources and
// upward pass, and the proxy interactions of swe_vel_panel_interaction_2
// (src/fmm_interactions/swe_vel_impl.hpp:80-147):
//
//   u(x) += 1/(4 pi) [ -S_vor (x cross y')/(1 - x.y' + eps)
//                      + S_div (y - x (x.y))/(1 - x.y + eps) ]
//
// with y' the displaced, re-projected source proxy and y the fixed one.  Both
// denominators are computed as |y - x|^2/2 + eps (|x| = |y| = 1), the
// rotational part as x cross sum g (y' - x), and the divergent part as the
// tangential projection (I - x x^T) of sum g2 (y - x), which equals
// sum g2 (y - x (x.y)) for |x| = 1.  Sources (double4, 32 B per proxy):
//   src  = (y'_x, y'_y, y'_z, S_vor),   src2 = (y_x, y_y, y_z, S_div).
// Every kernel is owner-computes (no atomics) and deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "../../include/sbslpm.h"
#include "device_common.cuh"
#include "list32.cuh"
#include "list64.cuh"
#include "swe_kernels.cuh"

namespace sbslpm {
namespace {

using namespace dev;

constexpr int kWarps = 4;

// ---------------------------------------------------------------------------
// Sources.

// Strengths of leaf point i (relative index) at a stage: swe_apply_tendencies_2
// (src/swe_time_step_2.cpp:390-414) folded into base_pots
// (src/fmm_funcs_impl.hpp:17-34): w_vor = area (1 + dts div) (vor + dts tv),
// w_div = area (div + dts td).
__device__ __forceinline__ void leaf_strengths(long i, long ln, int stage, double dts, const double* tprev,
                                               const double* vors, const double* divs, const double* area,
                                               double& wv, double& wd) {
  const double a = area[i], vor = vors[i], div = divs[i];
  if (stage == 0) {
    wv = a * vor;
    wd = a * div;
  } else {
    const double dvor = vor + dts * tprev[i];
    const double ddiv = div + dts * tprev[ln + i];
    wv = (a * (1.0 + dts * div)) * dvor;
    wd = a * ddiv;
  }
}

// Positions of the non-leaf proxies of both fields (swe_disp_interp_2,
// src/swe_time_step_2.cpp:436-476, identical to the BVE form): the vorticity
// sources displaced by the interpolated leaf velocity, the divergence sources
// at the fixed proxies.  Positions only; the subtrees write the strengths.
template <int N1>
__device__ __forceinline__ void swe_nonleaf_source(const StepGeom& g, const SweGeom& sw, long i, int stage, double dtd,
                                                   const double* __restrict__ vprev, double4* __restrict__ src,
                                                   double4* __restrict__ src2, int mixed) {
  const int q = N1 > 0 ? N1 * N1 : g.q;
  const long pn = (long)g.panels * q;
  const double x0 = g.px[i], y0 = g.px[pn + i], z0 = g.px[2 * pn + i];
  double px, py, pz;
  nonleaf_position<N1 * N1>(g, i, stage, dtd, vprev, px, py, pz);
  src[i].x = px;
  src[i].y = py;
  src[i].z = pz;
  src2[i].x = x0;
  src2[i].y = y0;
  src2[i].z = z0;
  if (mixed) {
    const double* c = g.pd_centre + 4 * (i / q);
    store_packed_xyz(g.srcf, q, i / q, (int)(i % q), (float)((px - c[0]) * kPackScale),
                     (float)((py - c[1]) * kPackScale), (float)((pz - c[2]) * kPackScale));
    store_packed_xyz(sw.srcf2, q, i / q, (int)(i % q), (float)((x0 - c[0]) * kPackScale),
                     (float)((y0 - c[1]) * kPackScale), (float)((z0 - c[2]) * kPackScale));
  }
}

// Fused upward pass over one subtree (the SWE form of k_upward_subtree): leaf
// sources of both fields when the subtree reaches the leaves, both strengths
// anterpolated level by level (upward_pass, src/fmm_funcs.cpp:341-355), and
// the packed float sources in mixed precision; the blocks past `roots` of the
// first launch place the non-leaf proxies.
constexpr int kTreeThreads = 1024;

template <int N1>
__global__ void __launch_bounds__(kTreeThreads)
    k_swe_upward_subtree(StepGeom g, SweGeom sw, int roots, int chunk, int r, int D, int stage, double dtd, double dts,
                         const double* __restrict__ vprev, const double* __restrict__ tprev,
                         const double* __restrict__ vors, const double* __restrict__ divs,
                         const double* __restrict__ area, double4* __restrict__ src, double4* __restrict__ src2,
                         int mixed) {
  const int n1 = N1 > 0 ? N1 : g.degree + 1, q = N1 > 0 ? N1 * N1 : g.q;
  if ((int)blockIdx.x >= roots) {
    const long i = ((long)blockIdx.x - roots) * chunk + threadIdx.x;
    if ((int)threadIdx.x < chunk && i < (long)g.offset * q) swe_nonleaf_source<N1>(g, sw, i, stage, dtd, vprev, src, src2, mixed);
    return;
  }
  extern __shared__ double sh[];  // 2 fields x levels r..r+D, then 2 x 4^D q scratch
  const int root_rel = blockIdx.x;
  const bool leaves_here = (r + D == g.levels - 1);
  const long ln = (long)g.leaves * q, pn = (long)g.panels * q;
  const int per_field = q * (((1 << (2 * (D + 1))) - 1) / 3);
  auto lvl = [&](int f, int k) { return sh + f * per_field + q * (((1 << (2 * k)) - 1) / 3); };
  double* scratch = sh + 2 * per_field;
  const int sstride = (1 << (2 * D)) * q;

  {
    const int first = subtree_first(r, root_rel, D), npts = (1 << (2 * D)) * q;
    for (int t = threadIdx.x; t < npts; t += blockDim.x) {
      const long o = (long)first * q + t;
      double wv, wd;
      if (leaves_here) {
        const long i = o - (long)g.offset * q;
        leaf_strengths(i, ln, stage, dts, tprev, vors, divs, area, wv, wd);
        const double x0 = g.px[o], y0 = g.px[pn + o], z0 = g.px[2 * pn + o];
        double px = x0, py = y0, pz = z0;
        src2[o] = make_double4(x0, y0, z0, wd);
        if (stage > 0) {
          px += dtd * vprev[i];
          py += dtd * vprev[ln + i];
          pz += dtd * vprev[2 * ln + i];
        }
        project_to_sphere(px, py, pz);
        src[o] = make_double4(px, py, pz, wv);
        if (mixed) {
          const double* c = g.pd_centre + 4 * (o / q);
          store_packed(g.srcf, q, o / q, t % q, c, px, py, pz, wv);
          store_packed(sw.srcf2, q, o / q, t % q, c, x0, y0, z0, wd);
        }
      } else {
        wv = src[o].w;
        wd = src2[o].w;
      }
      lvl(0, D)[t] = wv;
      lvl(1, D)[t] = wd;
    }
  }
  __syncthreads();
  for (int k = D - 1; k >= 0; k--) {
    const int np = 1 << (2 * k), first = subtree_first(r, root_rel, k);
    for (int t = threadIdx.x; t < 2 * 4 * np * q; t += blockDim.x) {  // T[f][cc][i][b]
      const int f = t >= 4 * np * q, tt = t - f * 4 * np * q;
      const int cc = tt / q, rem = tt % q, i = rem / n1, b = rem % n1;
      const double* ly = g.child_1d + ((cc & 3) >= 2 ? n1 * n1 : 0);
      const double* sc = lvl(f, k + 1) + cc * q + i * n1;
      double acc = 0;
#pragma unroll
      for (int j = 0; j < (N1 > 0 ? N1 : n1); j++) acc = fma(__ldg(ly + j * n1 + b), sc[j], acc);
      scratch[f * sstride + tt] = acc;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 2 * np * q; t += blockDim.x) {  // S[f][p][a][b]
      const int f = t >= np * q, tt = t - f * np * q;
      const int p = tt / q, rem = tt % q, a = rem / n1, b = rem % n1;
      double acc = 0;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const double* lx = g.child_1d + ((c == 1 || c == 2) ? n1 * n1 : 0);
        const double* tc = scratch + f * sstride + (4 * p + c) * q + b;
#pragma unroll
        for (int i = 0; i < (N1 > 0 ? N1 : n1); i++) acc = fma(__ldg(lx + i * n1 + a), tc[i * n1], acc);
      }
      lvl(f, k)[tt] = acc;
      const long o = (long)first * q + tt;
      if (f == 0) src[o].w = acc;
      else src2[o].w = acc;
      if (mixed) {
        store_packed_w(f == 0 ? g.srcf : sw.srcf2, q, o / q, rem, (float)acc);
      }
    }
    __syncthreads();
  }
}

// Direct velocity: leaf sources of both fields (no tree).
__global__ void k_swe_leaf_sources(StepGeom g, SweGeom sw, int stage, double dtd, double dts,
                                   const double* __restrict__ vprev, const double* __restrict__ tprev,
                                   const double* __restrict__ vors, const double* __restrict__ divs,
                                   const double* __restrict__ area, double4* __restrict__ src,
                                   double4* __restrict__ src2, int mixed) {
  const long ln = (long)g.leaves * g.q, pn = (long)g.panels * g.q;
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= ln) return;
  const long o = (long)g.offset * g.q + i;
  double wv, wd;
  leaf_strengths(i, ln, stage, dts, tprev, vors, divs, area, wv, wd);
  double px = g.px[o], py = g.px[pn + o], pz = g.px[2 * pn + o];
  src2[o] = make_double4(px, py, pz, wd);
  const double* c = g.pd_centre + 4 * (o / g.q);
  const int j = (int)(o % g.q);
  if (mixed) store_packed(sw.srcf2, g.q, o / g.q, j, c, px, py, pz, wd);
  if (stage > 0) {
    px += dtd * vprev[i];
    py += dtd * vprev[ln + i];
    pz += dtd * vprev[2 * ln + i];
  }
  project_to_sphere(px, py, pz);
  src[o] = make_double4(px, py, pz, wv);
  if (mixed) store_packed(g.srcf, g.q, o / g.q, j, c, px, py, pz, wv);
}

// Piecewise API: sources from explicit displacements (swe_vel_panel_interaction_2
// displaces every proxy, src/fmm_interactions/swe_vel_impl.hpp:124-128) and strengths.
__global__ void k_swe_sources_from_disp(StepGeom g, SweGeom sw, const double* __restrict__ dx,
                                        const double* __restrict__ dy, const double* __restrict__ dz,
                                        const double* __restrict__ sv, const double* __restrict__ sd,
                                        double4* __restrict__ src, double4* __restrict__ src2, int mixed) {
  const long pn = (long)g.panels * g.q;
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= pn) return;
  const double x0 = g.px[i], y0 = g.px[pn + i], z0 = g.px[2 * pn + i];
  double px = x0 + dx[i], py = y0 + dy[i], pz = z0 + dz[i];
  project_to_sphere(px, py, pz);
  src[i] = make_double4(px, py, pz, sv[i]);
  src2[i] = make_double4(x0, y0, z0, sd[i]);
  if (mixed) {
    const double* c = g.pd_centre + 4 * (i / g.q);
    const int j = (int)(i % g.q);
    store_packed(g.srcf, g.q, i / g.q, j, c, px, py, pz, sv[i]);
    store_packed(sw.srcf2, g.q, i / g.q, j, c, x0, y0, z0, sd[i]);
  }
}

// ---------------------------------------------------------------------------
// Interactions: q <= 25 by list64.cuh and list32.cuh below; larger q by one
// warp per target panel, each lane owning ceil(q/32) target nodes.  A source
// panel's q proxies of both fields are staged in shared memory and every lane
// sweeps them (mixed: two proxies per paired float32 instruction, each panel's
// two interleaved float32 halves added before the float64 conversion).
// ALL_LEAVES: every leaf against every leaf, source leaves split into
// gridDim.y groups whose partials are reduced in order afterwards.

// u = K x cross A - K (B - x (x.B)); K = -1/(4 pi), or scaled by sqrt(2)
// for the packed float sums.
__device__ __forceinline__ void swe_epilogue(double K, double tx, double ty, double tz, double ax, double ay,
                                             double az, double bx, double by, double bz, double& ux, double& uy,
                                             double& uz) {
  const double tb = tx * bx + ty * by + tz * bz;
  ux = K * (ty * az - tz * ay) - K * (bx - tx * tb);
  uy = K * (tz * ax - tx * az) - K * (by - ty * tb);
  uz = K * (tx * ay - ty * ax) - K * (bz - tz * tb);
}

template <int Q, bool ALL_LEAVES, bool GUARD, bool MIXED>
__global__ void __launch_bounds__(32 * kWarps)
    k_swe_interact(StepGeom g, SweGeom sw, const double4* __restrict__ src, const double4* __restrict__ src2,
                   double* __restrict__ out, long out_stride) {
  constexpr int TPL = (Q + 31) / 32;
  using Src = typename std::conditional<MIXED, float4, double4>::type;
  // mixed: the Q proxies as ceil(Q/2) source pairs of two float4
  // (x0,x1,y0,y1),(z0,z1,w0,w1), an odd Q closing on a zero-strength source
  // at the panel's centre (which adds exactly zero)
  constexpr int HQ = (Q + 1) / 2, kRow = row_of(Q);
  __shared__ Src stage[kWarps][2][MIXED ? 2 * HQ : Q];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tp_first = ALL_LEAVES ? g.offset : 0;
  const int tp_count = ALL_LEAVES ? g.leaves : g.panels;
  const int tix = blockIdx.x * kWarps + warp;
  if (tix >= tp_count) return;
  const int t = tp_first + tix;
  const long pn = (long)g.panels * g.q;
  int e0, e1;
  if (ALL_LEAVES) {
    const int per = (g.leaves + gridDim.y - 1) / gridDim.y;
    e0 = blockIdx.y * per;
    e1 = min(g.leaves, e0 + per);
  } else {
    e0 = g.tgt_start[t];
    e1 = g.tgt_start[t + 1];
  }
  auto source_of = [&](int e) { return ALL_LEAVES ? g.offset + e : __ldg(g.src_panel + e); };
  const Src* s1 = nullptr;
  const Src* s2 = nullptr;
  if constexpr (MIXED) {
    s1 = g.srcf;
    s2 = sw.srcf2;
  } else {
    s1 = src;
    s2 = src2;
  }
  const double* ct = g.pd_centre + 4 * (long)t;
  const float eps32 = (float)g.eps;
  const double deps2 = twice_eps(g.eps);
  constexpr double K = MIXED ? kBiotSavartPacked : kBiotSavartTwice;

  double tx[TPL], ty[TPL], tz[TPL], ax[TPL], ay[TPL], az[TPL], bx[TPL], by[TPL], bz[TPL];
  float dtx[TPL], dty[TPL], dtz[TPL];
#pragma unroll
  for (int r = 0; r < TPL; r++) {
    const int j = lane + 32 * r;
    const long o = (long)t * Q + (j < Q ? j : 0);
    tx[r] = g.px[o];
    ty[r] = g.px[pn + o];
    tz[r] = g.px[2 * pn + o];
    if (MIXED) {
      dtx[r] = (float)((tx[r] - ct[0]) * kPackScale);
      dty[r] = (float)((ty[r] - ct[1]) * kPackScale);
      dtz[r] = (float)((tz[r] - ct[2]) * kPackScale);
    }
    ax[r] = ay[r] = az[r] = bx[r] = by[r] = bz[r] = 0;
  }
  constexpr int PER = MIXED ? HQ : Q;  // staging items per source panel: proxies (float64) or source pairs (mixed)
  for (int e = e0; e < e1; e++) {
    const int sp = source_of(e);
    for (int k = lane; k < PER; k += 32) {
      if constexpr (MIXED) {
        const long b = (long)sp * Q + 2 * k;
        const bool two = 2 * k + 1 < Q;
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 a0 = s1[b], a1 = two ? s1[b + 1] : none, c0 = s2[b], c1 = two ? s2[b + 1] : none;
        stage[warp][0][2 * k] = make_float4(a0.x, a1.x, a0.y, a1.y);
        stage[warp][0][2 * k + 1] = make_float4(a0.z, a1.z, a0.w, a1.w);
        stage[warp][1][2 * k] = make_float4(c0.x, c1.x, c0.y, c1.y);
        stage[warp][1][2 * k + 1] = make_float4(c0.z, c1.z, c0.w, c1.w);
      } else {
        stage[warp][0][k] = s1[(long)sp * Q + k];
        stage[warp][1][k] = s2[(long)sp * Q + k];
      }
    }
    __syncwarp();
    {
      const Src* st1 = stage[warp][0];
      const Src* st2 = stage[warp][1];
      if constexpr (MIXED) {
        const double* cs = g.pd_centre + 4 * (long)sp;
        const float c0 = (float)((cs[0] - ct[0]) * kPackScale), c1 = (float)((cs[1] - ct[1]) * kPackScale),
                    c2 = (float)((cs[2] - ct[2]) * kPackScale);
        const float2 eps2 = make_float2(eps32, eps32);
        float2 fa[TPL][3], fb[TPL][3], b0[TPL], b1[TPL], b2[TPL];
#pragma unroll
        for (int r = 0; r < TPL; r++) {
          b0[r] = make_float2(c0 - dtx[r], c0 - dtx[r]);
          b1[r] = make_float2(c1 - dty[r], c1 - dty[r]);
          b2[r] = make_float2(c2 - dtz[r], c2 - dtz[r]);
          fa[r][0] = fa[r][1] = fa[r][2] = fb[r][0] = fb[r][1] = fb[r][2] = make_float2(0.f, 0.f);
        }
#pragma unroll 4
        for (int k = 0; k < HQ; k++) {
          const float4 A = st1[2 * k], B = st1[2 * k + 1], C = st2[2 * k], D = st2[2 * k + 1];
#pragma unroll
          for (int r = 0; r < TPL; r++) {
            pair32x2<GUARD>(b0[r], b1[r], b2[r], make_float2(A.x, A.y), make_float2(A.z, A.w),
                            make_float2(B.x, B.y), make_float2(B.z, B.w), eps2, fa[r][0], fa[r][1], fa[r][2]);
            pair32x2<GUARD>(b0[r], b1[r], b2[r], make_float2(C.x, C.y), make_float2(C.z, C.w),
                            make_float2(D.x, D.y), make_float2(D.z, D.w), eps2, fb[r][0], fb[r][1], fb[r][2]);
          }
        }
#pragma unroll
        for (int r = 0; r < TPL; r++) {
          ax[r] += (double)(fa[r][0].x + fa[r][0].y);
          ay[r] += (double)(fa[r][1].x + fa[r][1].y);
          az[r] += (double)(fa[r][2].x + fa[r][2].y);
          bx[r] += (double)(fb[r][0].x + fb[r][0].y);
          by[r] += (double)(fb[r][1].x + fb[r][1].y);
          bz[r] += (double)(fb[r][2].x + fb[r][2].y);
        }
      } else {
#pragma unroll kRow
        for (int k = 0; k < Q; k++) {
          const double4 v1 = st1[k], v2 = st2[k];
          pairs64<GUARD>(tx, ty, tz, v1.x, v1.y, v1.z, v1.w, deps2, ax, ay, az);
          pairs64<GUARD>(tx, ty, tz, v2.x, v2.y, v2.z, v2.w, deps2, bx, by, bz);
        }
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int r = 0; r < TPL; r++) {
    const int j = lane + 32 * r;
    if (j >= Q) continue;
    double ux, uy, uz;
    const long ot = (long)t * Q + j;  // the target's position again: not held in registers across the sweep
    swe_epilogue(K, g.px[ot], g.px[pn + ot], g.px[2 * pn + ot], ax[r], ay[r], az[r], bx[r], by[r], bz[r], ux, uy,
                 uz);
    const long o = ALL_LEAVES ? (long)blockIdx.y * 3 * out_stride + (long)tix * Q + j : (long)t * Q + j;
    const long s = ALL_LEAVES ? out_stride : pn;
    out[o] = ux;
    out[s + o] = uy;
    out[2 * s + o] = uz;
  }
}

// Float64, q <= 25: both fields by list64.cuh.
template <int Q, int WPT, bool ALL_LEAVES, bool GUARD>
__global__ void __launch_bounds__(32 * ListShape<Q, 2>::NW)
    k_swe_interact64(StepGeom g, const double4* __restrict__ src, const double4* __restrict__ src2,
                     double* __restrict__ out, long out_stride) {
  using W = ListShape<Q, 2>;
  __shared__ __align__(16) double2 tiles[W::NW * W::WARP];
  const long pn = (long)g.panels * Q;
  list64_sweep<Q, 2, WPT, ALL_LEAVES, GUARD>(
      g, src, src2, tiles, [&](int t, int tix, int j, const double* a) {
        const long i = (long)t * Q + j;
        double ux, uy, uz;
        swe_epilogue(kBiotSavartTwice, g.px[i], g.px[pn + i], g.px[2 * pn + i], a[0], a[1], a[2], a[3], a[4], a[5],
                     ux, uy, uz);
        const long o = ALL_LEAVES ? (long)blockIdx.y * 3 * out_stride + (long)tix * Q + j : i;
        const long s = ALL_LEAVES ? out_stride : pn;
        out[o] = ux;
        out[s + o] = uy;
        out[2 * s + o] = uz;
      });
}

// Mixed precision, q <= 25: both fields by list32.cuh.
template <int Q, int WPT, bool ALL_LEAVES, bool GUARD>
__global__ void __launch_bounds__(32 * ListShape32<Q, 2>::NW)
    k_swe_interact32(StepGeom g, SweGeom sw, double* __restrict__ out, long out_stride) {
  using W = ListShape32<Q, 2>;
  __shared__ __align__(16) double shared[W::NW * ((W::WARP + 1) & ~1)];
  const long pn = (long)g.panels * Q;
  list32_sweep<Q, 2, WPT, ALL_LEAVES, GUARD>(
      g, g.srcf, sw.srcf2, shared, [&](int t, int tix, int j, const double* a) {
        const long i = (long)t * Q + j;
        double ux, uy, uz;
        swe_epilogue(kBiotSavartPacked, g.px[i], g.px[pn + i], g.px[2 * pn + i], a[0], a[1], a[2], a[3], a[4], a[5],
                     ux, uy, uz);
        const long o = ALL_LEAVES ? (long)blockIdx.y * 3 * out_stride + (long)tix * Q + j : i;
        const long s = ALL_LEAVES ? out_stride : pn;
        out[o] = ux;
        out[s + o] = uy;
        out[2 * s + o] = uz;
      });
}

__global__ void k_swe_reduce(const double* __restrict__ partial, int groups, long n, long gstride,
                             double* __restrict__ out) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0;
  for (int k = 0; k < groups; k++) s += partial[k * gstride + i];
  out[i] = s;
}

template <int Q, bool GUARD>
void swe_interact_qg(const StepGeom& g, const SweGeom& s, int precision, const double4* src, const double4* src2,
                     double* out, bool all_leaves, int groups, long out_stride, cudaStream_t st) {
  const int tp = all_leaves ? g.leaves : g.panels;
  dim3 grid(blocks_for(tp, kWarps), all_leaves ? groups : 1);
  const bool mixed = precision == SBSLPM_MIXED;
#define SB_SWE_K(AL, MX) \
  SB_LAUNCH((k_swe_interact<Q, AL, GUARD, MX>), grid, 32 * kWarps, 0, st, g, s, src, src2, out, out_stride)
  if constexpr (Q <= 32) {
    if (mixed) {
      constexpr int NW = ListShape32<Q, 2>::NW, threads = 32 * NW;
      const int wpt = dev::list_warps<Q, 2, true>(tp);
      if (all_leaves)
        SB_LAUNCH((k_swe_interact32<Q, 1, true, GUARD>), dim3(blocks_for(tp, NW), groups), threads, 0, st, g, s, out,
                  out_stride);
      else if (wpt == NW)
        SB_LAUNCH((k_swe_interact32<Q, NW, false, GUARD>), tp, threads, 0, st, g, s, out, out_stride);
      else if (wpt == 2)
        SB_LAUNCH((k_swe_interact32<Q, 2, false, GUARD>), blocks_for(tp, NW / 2), threads, 0, st, g, s, out, out_stride);
      else
        SB_LAUNCH((k_swe_interact32<Q, 1, false, GUARD>), blocks_for(tp, NW), threads, 0, st, g, s, out, out_stride);
      return;
    }
    constexpr int NW = ListShape<Q, 2>::NW, threads = 32 * NW;
    const int wpt = dev::list_warps<Q, 2, false>(tp);
    if (all_leaves)
      SB_LAUNCH((k_swe_interact64<Q, 1, true, GUARD>), dim3(blocks_for(tp, NW), groups), threads, 0, st, g, src, src2,
                out, out_stride);
    else if (wpt == NW)
      SB_LAUNCH((k_swe_interact64<Q, NW, false, GUARD>), tp, threads, 0, st, g, src, src2, out, out_stride);
    else if (wpt == 2)
      SB_LAUNCH((k_swe_interact64<Q, 2, false, GUARD>), blocks_for(tp, NW / 2), threads, 0, st, g, src, src2, out,
                out_stride);
    else
      SB_LAUNCH((k_swe_interact64<Q, 1, false, GUARD>), blocks_for(tp, NW), threads, 0, st, g, src, src2, out,
                out_stride);
  } else {
    if (all_leaves && mixed) SB_SWE_K(true, true);
    else if (all_leaves) SB_SWE_K(true, false);
    else if (mixed) SB_SWE_K(false, true);
    else SB_SWE_K(false, false);
  }
#undef SB_SWE_K
}

void swe_interact_dispatch(const StepGeom& g, const SweGeom& s, int precision, const double4* src,
                           const double4* src2, double* out, bool all_leaves, int groups, long out_stride,
                           cudaStream_t st) {
#define SB_SQ(Q)                                                                                   \
  case Q:                                                                                          \
    if (g.eps > 0) swe_interact_qg<Q, false>(g, s, precision, src, src2, out, all_leaves, groups, out_stride, st); \
    else swe_interact_qg<Q, true>(g, s, precision, src, src2, out, all_leaves, groups, out_stride, st);            \
    break;
  switch (g.q) {
    SB_SQ(1) SB_SQ(4) SB_SQ(9) SB_SQ(16) SB_SQ(25) SB_SQ(36) SB_SQ(49) SB_SQ(64) SB_SQ(81) SB_SQ(100) SB_SQ(121)
  }
#undef SB_SQ
}

size_t swe_subtree_smem(int q, int D) {
  return (size_t)q * 2 * 8 * ((((1L << (2 * (D + 1))) - 1) / 3) + (1L << (2 * D)));
}

template <int N1>
void swe_upward(const StepGeom& g, const SweGeom& s, int stage, double dtd, double dts, const double* vprev,
                const double* tprev, const double* vors, const double* divs, const double* area, double4* src,
                double4* src2, bool mixed, cudaStream_t st) {
  static std::atomic<unsigned long long> attr{0};
  raise_smem_once(attr, 200 * 1024, k_swe_upward_subtree<N1>);
  const int Dmax = g.q <= 25 ? 3 : 1;
  int r = g.levels - 1;
  bool first = true;
  do {
    const int D = r < Dmax ? r : Dmax, root = r - D, roots = 6 << (2 * root);
    const unsigned threads = std::min((unsigned)kTreeThreads, (unsigned)(((g.q << (2 * D)) + 31) / 32 * 32));
    const long points = first ? (long)g.offset * g.q : 0;
    const int chunk = nonleaf_chunk(points, threads);
    const unsigned extra = blocks_for(points, chunk);
    SB_LAUNCH(k_swe_upward_subtree<N1>, roots + extra, threads, swe_subtree_smem(g.q, D), st, g, s, roots, chunk, root, D,
              stage, dtd, dts, vprev, tprev, vors, divs, area, src, src2, mixed ? 1 : 0);
    r = root;
    first = false;
  } while (r > 0);
}

}  // namespace

void launch_swe_upward(const StepGeom& g, const SweGeom& s, int stage, double dtd, double dts, const double* vprev,
                       const double* tprev, const double*, const double*, const double*, const double* vors,
                       const double* divs, const double* area, double4* src, double4* src2, bool mixed,
                       cudaStream_t st) {
  // the degrees in use; the general form serves the others (5.4 us a launch at degree 5, levels 3)
  switch (g.degree) {
    case 2: swe_upward<3>(g, s, stage, dtd, dts, vprev, tprev, vors, divs, area, src, src2, mixed, st); break;
    case 3: swe_upward<4>(g, s, stage, dtd, dts, vprev, tprev, vors, divs, area, src, src2, mixed, st); break;
    case 4: swe_upward<5>(g, s, stage, dtd, dts, vprev, tprev, vors, divs, area, src, src2, mixed, st); break;
    default: swe_upward<0>(g, s, stage, dtd, dts, vprev, tprev, vors, divs, area, src, src2, mixed, st); break;
  }
}

void launch_swe_leaf_sources(const StepGeom& g, const SweGeom& s, int stage, double dtd, double dts,
                             const double* vprev, const double* tprev, const double* vors, const double* divs,
                             const double* area, double4* src, double4* src2, bool mixed, cudaStream_t st) {
  const long ln = (long)g.leaves * g.q;
  SB_LAUNCH(k_swe_leaf_sources, blocks_for(ln, 256), 256, 0, st, g, s, stage, dtd, dts, vprev, tprev, vors, divs,
            area, src, src2, mixed ? 1 : 0);
}

void launch_swe_interactions(const StepGeom& g, const SweGeom& s, int precision, const double4* src,
                             const double4* src2, double* tgt, cudaStream_t st) {
  swe_interact_dispatch(g, s, precision, src, src2, tgt, false, 1, 0, st);
}

void launch_swe_direct(const StepGeom& g, const SweGeom& s, int precision, const double4* src, const double4* src2,
                       double* vout, double* partial, int groups, cudaStream_t st) {
  const long n = (long)g.leaves * g.q;
  swe_interact_dispatch(g, s, precision, src, src2, partial, true, groups, n, st);
  SB_LAUNCH(k_swe_reduce, blocks_for(3 * n, 256), 256, 0, st, partial, groups, 3 * n, 3 * n, vout);
}

void launch_swe_sources_from_disp(const StepGeom& g, const SweGeom& s, const double* dx, const double* dy,
                                  const double* dz, const double* s_vor, const double* s_div, double4* src,
                                  double4* src2, bool mixed, cudaStream_t st) {
  const long pn = (long)g.panels * g.q;
  SB_LAUNCH(k_swe_sources_from_disp, blocks_for(pn, 256), 256, 0, st, g, s, dx, dy, dz, s_vor, s_div, src, src2,
            mixed ? 1 : 0);
}

}  // namespace sbslpm
