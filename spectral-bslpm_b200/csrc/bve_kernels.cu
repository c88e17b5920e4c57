// Device kernels of the BVE backward semi-Lagrangian step, sm_100a.
//
// Data layout in HBM (all row-major, [panel][q] as in the reference):
//   src   : double4 [panels*q]  displaced source position (x, y, z) and
//           strength w = area * vorticity (leaves) or its anterpolation
//           (non-leaf proxies).  32 B per proxy point, one load per pair block.
//   srcf  : float4  [panels][packed_stride(q)]  mixed precision: position
//           relative to the panel centre (float) and strength (float), up to
//           25 sources two by two (store_packed_xyz).
//   tgt   : double  [3][panels*q] proxy-target velocities.
//   v_k   : double  [3][leaves*q] stage velocities (x, y, z blocks).
// Every kernel is owner-computes (no atomics), so results are deterministic.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <initializer_list>
#include <type_traits>

#include "../../include/sbslpm.h"
#include "bve_kernels.cuh"
#include "device_common.cuh"
#include "list32.cuh"
#include "list64.cuh"

namespace sbslpm {

std::atomic<long>& launch_counter() {
  static std::atomic<long> n{0};
  return n;
}

namespace {

using namespace dev;


// ---------------------------------------------------------------------------
// Source preparation.

// Leaves (bve_disp_update, src/bve_time_step.cpp:69-105, with the forcing
// copy of src/forcing_funcs.cpp:93-95 and base_pots, src/fmm_funcs_impl.hpp:17-34):
// stage 0: strength area*vor at proj(proxy); stage s > 0: disp = dt_s v,
// strength area*(vor + 2 Omega z - 2 Omega z'), z' from proj(x + v dt_s),
// position proj(proxy + disp).
__global__ void k_leaf_sources(StepGeom g, int stage, double dt_s, const double* __restrict__ vprev,
                               const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, const double* __restrict__ vors,
                               const double* __restrict__ area, double4* __restrict__ src,
                               double* __restrict__ keep) {
  long n = (long)g.leaves * g.q;
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (keep) keep[i] = vors[i];
  long pn = (long)g.panels * g.q;
  long o = (long)g.offset * g.q + i;
  double px = g.px[o], py = g.px[pn + o], pz = g.px[2 * pn + o];
  double w;
  if (stage == 0) {
    w = area[i] * (g.force ? vors[i] + g.force[i] : vors[i]);
  } else {
    double vx = vprev[i], vy = vprev[n + i], vz = vprev[2 * n + i];
    double xx = x[i] + vx * dt_s, yy = y[i] + vy * dt_s, zz = z[i] + vz * dt_s;
    project_to_sphere(xx, yy, zz);
    double dvor = vors[i] + 2 * g.omega * z[i] - 2 * g.omega * zz;
    w = area[i] * (g.force ? dvor + g.force[i] : dvor);
    px += dt_s * vx;
    py += dt_s * vy;
    pz += dt_s * vz;
  }
  project_to_sphere(px, py, pz);
  src[o] = make_double4(px, py, pz, w);
}

// Piecewise API: sources from explicit displacements and strengths
// (the inputs of bve_vel_interactions).
__global__ void k_sources_from_disp(StepGeom g, const double* __restrict__ dx, const double* __restrict__ dy,
                                    const double* __restrict__ dz, const double* __restrict__ s,
                                    double4* __restrict__ src) {
  long pn = (long)g.panels * g.q;
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= pn) return;
  double px = g.px[i] + dx[i], py = g.px[pn + i] + dy[i], pz = g.px[2 * pn + i] + dz[i];
  project_to_sphere(px, py, pz);
  src[i] = make_double4(px, py, pz, s[i]);
}

__global__ void k_copy_strength(StepGeom g, const double4* __restrict__ src, double* __restrict__ out) {
  long pn = (long)g.panels * g.q;
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= pn) return;
  out[i] = src[i].w;
}

// ---------------------------------------------------------------------------
// Tree passes (upward_pass / downward_pass_3, src/fmm_funcs.cpp:341-392;
// child_to_parent / parent_to_child_3, src/fmm_funcs_impl.hpp:36-172).
// The BLI basis of parent node (a,b) at child c's node (i,j) is the product
// Lx_c[i][a] Ly_c[j][b] of one-dimensional bases, and the uniform quadtree has
// only two of them: child_1d[h][i][a] for the child in the upper (h = 0) or
// lower (h = 1) half of its parent.  The passes contract one direction at a
// time:
//   upward:   T[c][i][b] = sum_j Ly_c[j][b] S_c[i][j];  S[a][b] = sum_c sum_i Lx_c[i][a] T[c][i][b]
//   downward: U[c][a][j] = sum_b Ly_c[j][b] T[a][b];    T_c[i][j] += sum_a Lx_c[i][a] U[c][a][j]
//
// One CTA owns the subtree of depth D below one panel of level r and keeps
// the strengths (upward) or target values (downward) of all its levels in
// shared memory, so a pass over the whole tree takes ceil((L-1)/3) launches.
// The passes are bound by latency (a chain of short phases between barriers):
// the node count n1 is a template argument (index arithmetic without
// divisions, contractions unrolled) and a CTA has a thread per point of its
// widest level where it can.
//
// Upward, mode 0 (the step): when the subtree reaches the leaves, the leaf
// sources are computed here (bve_disp_update, src/bve_time_step.cpp:69-105,
// with the forcing copy and base_pots folded in) and, at stage 0, the
// vorticity is copied to `keep` for the remap; strengths are anterpolated
// level by level; in mixed precision the packed float4 sources are written.
// The displaced positions of the non-leaf proxies (bve_disp_interp,
// src/bve_time_step.cpp:107-160, leaf row and BLI basis precomputed on the
// host) come from the blocks past `roots` of the first launch, a thread per
// point, beside the subtrees: they write the positions only, the subtrees the
// strengths only.  Levels 5, degree 3, us per stage: positions 7.0, passes up
// 13.1 and down 11.7 before; 7.9 and 8.3 now.
// Mode 1 (sbslpm_upward_pass): leaf strengths area * pots, positions untouched.
// Mode 2 (treecode): leaf strengths already anterpolated into src, fixed
// proxy positions untouched, mixed packing as in mode 0.

template <int N1>
__device__ __forceinline__ void nonleaf_source(const StepGeom& g, long i, int stage, double dt_s,
                                               const double* __restrict__ vprev, double4* __restrict__ src,
                                               int mixed) {
  const int q = N1 > 0 ? N1 * N1 : g.q;
  double px, py, pz;
  nonleaf_position<N1 * N1>(g, i, stage, dt_s, vprev, px, py, pz);
  src[i].x = px;
  src[i].y = py;
  src[i].z = pz;
  if (mixed) {
    const double* c = g.pd_centre + 4 * (i / q);
    store_packed_xyz(g.srcf, q, i / q, (int)(i % q), (float)((px - c[0]) * kPackScale),
                     (float)((py - c[1]) * kPackScale), (float)((pz - c[2]) * kPackScale));
  }
}

template <int N1>
__device__ __forceinline__ void upward_subtree_body(const StepGeom& g, int root_rel, int r, int D, int mode,
                                                    int stage, double dt_s, const double* __restrict__ vprev,
                                                    const double* __restrict__ x, const double* __restrict__ y,
                                                    const double* __restrict__ z, const double* __restrict__ vors,
                                                    const double* __restrict__ area, double4* __restrict__ src,
                                                    int mixed, double* __restrict__ keep) {
  extern __shared__ double sh[];  // strengths of levels r..r+D (level k at q*(4^k-1)/3), then scratch
  const int n1 = N1 > 0 ? N1 : g.degree + 1, q = N1 > 0 ? N1 * N1 : g.q;
  const bool leaves_here = (r + D == g.levels - 1);
  const long ln = (long)g.leaves * q, pn = (long)g.panels * q;
  auto lvl = [&](int k) { return sh + q * (((1 << (2 * k)) - 1) / 3); };

  // bottom level of the subtree: leaf sources, or strengths computed by the previous launch
  {
    const int first = subtree_first(r, root_rel, D), npts = (1 << (2 * D)) * q;
    double* bot = lvl(D);
    for (int t = threadIdx.x; t < npts; t += blockDim.x) {
      const long o = (long)first * q + t;
      if (leaves_here && mode != 2) {
        const long i = o - (long)g.offset * q;
        double w;
        if (mode == 1) {
          w = area[i] * vors[i];
          src[o].w = w;
        } else {
          double px = g.px[o], py = g.px[pn + o], pz = g.px[2 * pn + o];
          const double vor = vors[i];
          if (keep) keep[i] = vor;
          if (stage == 0) {
            w = area[i] * (g.force ? vor + g.force[i] : vor);
          } else {
            double vx = vprev[i], vy = vprev[ln + i], vz = vprev[2 * ln + i];
            double xx = x[i] + vx * dt_s, yy = y[i] + vy * dt_s, zz = z[i] + vz * dt_s;
            project_to_sphere(xx, yy, zz);
            double dvor = vor + 2 * g.omega * z[i] - 2 * g.omega * zz;
            w = area[i] * (g.force ? dvor + g.force[i] : dvor);
            px += dt_s * vx;
            py += dt_s * vy;
            pz += dt_s * vz;
          }
          project_to_sphere(px, py, pz);
          src[o] = make_double4(px, py, pz, w);
          if (mixed) store_packed(g.srcf, q, o / q, t % q, g.pd_centre + 4 * (o / q), px, py, pz, w);
        }
        bot[t] = w;
      } else {
        const double4 v = src[o];
        bot[t] = v.w;
        if (mixed && leaves_here)
          store_packed(g.srcf, q, o / q, t % q, g.pd_centre + 4 * (o / q), v.x, v.y, v.z, v.w);
      }
    }
  }
  __syncthreads();
  // anterpolation, deepest parents first, one direction at a time
  double* scratch = sh + q * (((1 << (2 * (D + 1))) - 1) / 3);
  for (int k = D - 1; k >= 0; k--) {
    const double* ch = lvl(k + 1);
    double* pa = lvl(k);
    const int np = 1 << (2 * k), first = subtree_first(r, root_rel, k);
    for (int t = threadIdx.x; t < 4 * np * q; t += blockDim.x) {  // T[cc][i][b]
      const int cc = t / q, rem = t % q, i = rem / n1, b = rem % n1;
      const double* ly = g.child_1d + ((cc & 3) >= 2 ? n1 * n1 : 0);
      const double* sc = ch + cc * q + i * n1;
      double acc = 0;
#pragma unroll
      for (int j = 0; j < (N1 > 0 ? N1 : n1); j++) acc = fma(__ldg(ly + j * n1 + b), sc[j], acc);
      scratch[t] = acc;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < np * q; t += blockDim.x) {  // S[p][a][b]
      const int p = t / q, rem = t % q, a = rem / n1, b = rem % n1;
      double acc = 0;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const double* lx = g.child_1d + ((c == 1 || c == 2) ? n1 * n1 : 0);
        const double* tc = scratch + (4 * p + c) * q + b;
#pragma unroll
        for (int i = 0; i < (N1 > 0 ? N1 : n1); i++) acc = fma(__ldg(lx + i * n1 + a), tc[i * n1], acc);
      }
      pa[t] = acc;
      const long o = (long)first * q + t;
      if (mixed && mode == 2) {
        const double4 v = src[o];
        store_packed(g.srcf, q, o / q, rem, g.pd_centre + 4 * (o / q), v.x, v.y, v.z, acc);
      } else if (mixed && mode == 0) {
        store_packed_w(g.srcf, q, o / q, rem, (float)acc);
      }
      src[o].w = acc;
    }
    __syncthreads();
  }
}

constexpr int kTreeThreads = 1024;

template <int N1>
__global__ void __launch_bounds__(kTreeThreads)
    k_upward_subtree(StepGeom g, int roots, int chunk, int r, int D, int mode, int stage, double dt_s,
                     const double* __restrict__ vprev, const double* __restrict__ x, const double* __restrict__ y,
                     const double* __restrict__ z, const double* __restrict__ vors, const double* __restrict__ area,
                     double4* __restrict__ src, int mixed, double* __restrict__ keep) {
  if ((int)blockIdx.x >= roots) {
    const long i = ((long)blockIdx.x - roots) * chunk + threadIdx.x;
    if ((int)threadIdx.x < chunk && i < (long)g.offset * (N1 > 0 ? N1 * N1 : g.q)) nonleaf_source<N1>(g, i, stage, dt_s, vprev, src, mixed);
    return;
  }
  upward_subtree_body<N1>(g, blockIdx.x, r, D, mode, stage, dt_s, vprev, x, y, z, vors, area, src, mixed, keep);
}

// Batched treecode members (mode 2): member blockIdx.z.
__global__ void k_upward_subtree_batch(const BatchMember* __restrict__ mem, int r, int D, int mixed) {
  const StepGeom g = mem[blockIdx.z].fg;
  upward_subtree_body<0>(g, blockIdx.x, r, D, 2, 0, 0.0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                         mem[blockIdx.z].fsrc, mixed, nullptr);
}

// Downward: the root's targets are final; children of levels r+1..r+D get
// own + interpolated parent values.  Leaves go to leaf_out when given (the
// stage velocity), intermediate levels stay in shared memory, and the
// deepest non-leaf level is written back for the next launch.
template <int N1>
__device__ __forceinline__ void downward_subtree_body(const StepGeom& g, int root_rel, int r, int D,
                                                      double* __restrict__ tgt, double* __restrict__ leaf_out) {
  extern __shared__ double sh[];  // 3 fields x levels r..r+D, then 3 x 4^D q scratch
  const int n1 = N1 > 0 ? N1 : g.degree + 1, q = N1 > 0 ? N1 * N1 : g.q;
  const long pn = (long)g.panels * q, ln = (long)g.leaves * q;
  const int per_field = q * (((1 << (2 * (D + 1))) - 1) / 3);
  auto lvl = [&](int f, int k) { return sh + f * per_field + q * (((1 << (2 * k)) - 1) / 3); };
  double* scratch = sh + 3 * per_field;
  const int sstride = (1 << (2 * D)) * q;
  {
    const int first = subtree_first(r, root_rel, 0);
    for (int t = threadIdx.x; t < q; t += blockDim.x)
      for (int f = 0; f < 3; f++) lvl(f, 0)[t] = tgt[f * pn + (long)first * q + t];
  }
  __syncthreads();
  for (int k = 1; k <= D; k++) {
    const int level = r + k, npts = (1 << (2 * k)) * q, first = subtree_first(r, root_rel, k);
    const bool is_leaf = (level == g.levels - 1);
    for (int t = threadIdx.x; t < npts; t += blockDim.x) {  // U[cc][a][j]
      const int cc = t / q, rem = t % q, a = rem / n1, j = rem % n1;
      const double* ly = g.child_1d + ((cc & 3) >= 2 ? n1 * n1 : 0) + j * n1;
      const int pp = cc >> 2;
      const double *p0 = lvl(0, k - 1) + pp * q + a * n1, *p1 = lvl(1, k - 1) + pp * q + a * n1,
                   *p2 = lvl(2, k - 1) + pp * q + a * n1;
      double u0 = 0, u1 = 0, u2 = 0;
#pragma unroll
      for (int b = 0; b < (N1 > 0 ? N1 : n1); b++) {
        const double l = __ldg(ly + b);
        u0 = fma(l, p0[b], u0);
        u1 = fma(l, p1[b], u1);
        u2 = fma(l, p2[b], u2);
      }
      scratch[t] = u0;
      scratch[sstride + t] = u1;
      scratch[2 * sstride + t] = u2;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < npts; t += blockDim.x) {  // T_c[i][j] += sum_a Lx[i][a] U[a][j]
      const int cc = t / q, rem = t % q, i = rem / n1, j = rem % n1, c = cc & 3;
      const double* lx = g.child_1d + ((c == 1 || c == 2) ? n1 * n1 : 0) + i * n1;
      const double* u = scratch + cc * q + j;
      double a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
      for (int a = 0; a < (N1 > 0 ? N1 : n1); a++) {
        const double l = __ldg(lx + a);
        a0 = fma(l, u[a * n1], a0);
        a1 = fma(l, u[sstride + a * n1], a1);
        a2 = fma(l, u[2 * sstride + a * n1], a2);
      }
      const long o = (long)first * q + t;
      a0 += tgt[o];
      a1 += tgt[pn + o];
      a2 += tgt[2 * pn + o];
      lvl(0, k)[t] = a0;
      lvl(1, k)[t] = a1;
      lvl(2, k)[t] = a2;
      if (is_leaf && leaf_out != nullptr) {
        const long lo = o - (long)g.offset * q;
        leaf_out[lo] = a0;
        leaf_out[ln + lo] = a1;
        leaf_out[2 * ln + lo] = a2;
      } else if (k == D || is_leaf || leaf_out == nullptr) {
        tgt[o] = a0;
        tgt[pn + o] = a1;
        tgt[2 * pn + o] = a2;
      }
    }
    __syncthreads();
  }
}

template <int N1>
__global__ void __launch_bounds__(kTreeThreads)
    k_downward_subtree(StepGeom g, int r, int D, double* __restrict__ tgt, double* __restrict__ leaf_out) {
  downward_subtree_body<N1>(g, blockIdx.x, r, D, tgt, leaf_out);
}

__global__ void k_downward_subtree_batch(const BatchMember* __restrict__ mem, int r, int D) {
  const StepGeom g = mem[blockIdx.z].fg;
  downward_subtree_body<0>(g, blockIdx.x, r, D, mem[blockIdx.z].ftgt, nullptr);
}

// ---------------------------------------------------------------------------
// Interactions (bve_vel_panel_interaction, src/fmm_interactions/bve_vel_impl.hpp:85-122).
//
// Panels of up to 25 points by list64.cuh and list32.cuh (a warp or more per
// target panel, its lists split over the lanes); larger ones by four warps per
// target panel (interact_wide_body).  Partial sums are combined in a fixed
// order, so the result is deterministic.
//
// Direct velocity: in float64, and mixed for panels of few points, the
// stand-alone direct sum's kernel over the leaf points; else every leaf against
// every leaf (ALL_LEAVES), the source leaves split into gridDim.y groups whose
// partials k_reduce_groups sums in order.

// Float64, q <= 25 (list64.cuh).
template <int Q, int WPT, bool GUARD>
__global__ void __launch_bounds__(32 * ListShape<Q, 1>::NW)
    k_interact64(StepGeom g, const double4* __restrict__ src, double* __restrict__ out) {
  using W = ListShape<Q, 1>;
  __shared__ __align__(16) double2 tiles[W::NW * W::WARP];
  const long pn = (long)g.panels * Q;
  list64_sweep<Q, 1, WPT, false, GUARD>(g, src, nullptr, tiles, [&](int t, int, int j, const double* a) {
    const long i = (long)t * Q + j;
    const double x = g.px[i], y = g.px[pn + i], z = g.px[2 * pn + i];
    out[i] = kBiotSavartTwice * (y * a[2] - z * a[1]);
    out[pn + i] = kBiotSavartTwice * (z * a[0] - x * a[2]);
    out[2 * pn + i] = kBiotSavartTwice * (x * a[1] - y * a[0]);
  });
}

// Mixed precision: positions relative to panel centres in float, pair
// arithmetic in float32, per-source-panel partial sums in float32 added into
// float64 accumulators.  For q <= 32 the two float32 halves of a panel's sum
// are added in float32 before the conversion: with 16 sources per panel the
// float64 conversions would otherwise load the MUFU/conversion pipe more than
// the reciprocals do.
__global__ void k_pack_mixed(StepGeom g, const double4* __restrict__ src, float4* __restrict__ srcf) {
  long pn = (long)g.panels * g.q;
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= pn) return;
  const double4 s = src[i];
  store_packed(srcf, g.q, i / g.q, (int)(i % g.q), g.pd_centre + 4 * (i / g.q), s.x, s.y, s.z, s.w);
}

// Mixed precision, q <= 25 (list32.cuh).
template <int Q, int WPT, bool ALL_LEAVES, bool GUARD>
__global__ void __launch_bounds__(32 * ListShape32<Q, 1>::NW)
    k_interact32(StepGeom g, const float4* __restrict__ srcf, double* __restrict__ out, long out_stride) {
  using W = ListShape32<Q, 1>;
  __shared__ __align__(16) double shared[W::NW * ((W::WARP + 1) & ~1)];
  const long pn = (long)g.panels * Q;
  list32_sweep<Q, 1, WPT, ALL_LEAVES, GUARD>(
      g, srcf, nullptr, shared, [&](int t, int tix, int j, const double* a) {
        const long i = (long)t * Q + j;
        const double x = g.px[i], y = g.px[pn + i], z = g.px[2 * pn + i];
        const long o = ALL_LEAVES ? (long)blockIdx.y * 3 * out_stride + (long)tix * Q + j : i;
        const long s = ALL_LEAVES ? out_stride : pn;
        out[o] = kBiotSavartPacked * (y * a[2] - z * a[1]);
        out[s + o] = kBiotSavartPacked * (z * a[0] - x * a[2]);
        out[2 * s + o] = kBiotSavartPacked * (x * a[1] - y * a[0]);
      });
}

// Wide panels (q > 32, e.g. 81 treecode proxies): one CTA of four warps per
// target panel; the warps take every fourth source panel, each lane owns
// ceil(q/32) target nodes, and the four partial sums are added in warp order
// (deterministic).  MIXED: float32 pairs on packed sources (kPackScale),
// per-source-panel float32 sums added into float64.
template <int Q, bool ALL_LEAVES, bool GUARD, bool MIXED>
__device__ __forceinline__ void interact_wide_body(const StepGeom& g, int tix, int gy, int ngy,
                                                   const double4* __restrict__ src, const float4* __restrict__ srcf,
                                                   double* __restrict__ out, long out_stride) {
  constexpr int TPL = (Q + 31) / 32, NW = 4, Q2 = (Q + 1) / 2, kRow = row_of(Q);
  using Src = typename std::conditional<MIXED, float4, double4>::type;
  // MIXED: sources staged two at a time, transposed, (x0,x1,y0,y1),(z0,z1,w0,w1)
  __shared__ Src stage[NW][MIXED ? 2 * Q2 : Q];
  __shared__ double red[NW][3][Q];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = (ALL_LEAVES ? g.offset : 0) + tix;
  const long pn = (long)g.panels * g.q;
  int e0, e1;
  if (ALL_LEAVES) {
    int per = (g.leaves + ngy - 1) / ngy;
    e0 = gy * per;
    e1 = min(g.leaves, e0 + per);
  } else {
    e0 = g.tgt_start[t];
    e1 = g.tgt_start[t + 1];
  }
  const double* ct = g.pd_centre + 4 * (long)t;
  const double ctx = ct[0], cty = ct[1], ctz = ct[2];
  double tx[TPL], ty[TPL], tz[TPL], ax[TPL], ay[TPL], az[TPL];
  float dtx[TPL], dty[TPL], dtz[TPL];
#pragma unroll
  for (int r = 0; r < TPL; r++) {
    int j = lane + 32 * r;
    long o = (long)t * Q + (j < Q ? j : 0);
    tx[r] = g.px[o];
    ty[r] = g.px[pn + o];
    tz[r] = g.px[2 * pn + o];
    dtx[r] = (float)((tx[r] - ctx) * kPackScale);
    dty[r] = (float)((ty[r] - cty) * kPackScale);
    dtz[r] = (float)((tz[r] - ctz) * kPackScale);
    ax[r] = ay[r] = az[r] = 0;
  }
  const float feps = (float)g.eps;
  const double eps2 = twice_eps(g.eps);
  for (int e = e0 + warp; e < e1; e += NW) {
    const int sp = ALL_LEAVES ? g.offset + e : __ldg(g.src_panel + e);
    const long sb = (long)sp * Q;
    if constexpr (MIXED) {
      for (int k2 = lane; k2 < Q2; k2 += 32) {
        const float4 s0 = srcf[sb + 2 * k2];
        const float4 s1 = (2 * k2 + 1 < Q) ? srcf[sb + 2 * k2 + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
        stage[warp][2 * k2] = make_float4(s0.x, s1.x, s0.y, s1.y);
        stage[warp][2 * k2 + 1] = make_float4(s0.z, s1.z, s0.w, s1.w);
      }
    } else {
      for (int k = lane; k < Q; k += 32) stage[warp][k] = src[sb + k];
    }
    __syncwarp();
    if constexpr (MIXED) {
      const double* cs = g.pd_centre + 4 * (long)sp;
      const float bx0 = (float)((cs[0] - ctx) * kPackScale), by0 = (float)((cs[1] - cty) * kPackScale),
                  bz0 = (float)((cs[2] - ctz) * kPackScale);
      const float2 eps2 = make_float2(feps, feps);
      float2 fx[TPL], fy[TPL], fz[TPL], bx[TPL], by[TPL], bz[TPL];
#pragma unroll
      for (int r = 0; r < TPL; r++) {
        fx[r] = fy[r] = fz[r] = make_float2(0.f, 0.f);
        const float b0 = bx0 - dtx[r], b1 = by0 - dty[r], b2 = bz0 - dtz[r];
        bx[r] = make_float2(b0, b0);
        by[r] = make_float2(b1, b1);
        bz[r] = make_float2(b2, b2);
      }
#pragma unroll 3
      for (int k2 = 0; k2 < Q2; k2++) {
        const float4 A = stage[warp][2 * k2], B = stage[warp][2 * k2 + 1];
        const float2 sx = make_float2(A.x, A.y), sy = make_float2(A.z, A.w), sz = make_float2(B.x, B.y),
                     sw = make_float2(B.z, B.w);
#pragma unroll
        for (int r = 0; r < TPL; r++)
          pair32x2<GUARD>(bx[r], by[r], bz[r], sx, sy, sz, sw, eps2, fx[r], fy[r], fz[r]);
      }
#pragma unroll
      for (int r = 0; r < TPL; r++) {
        ax[r] += (double)fx[r].x + (double)fx[r].y;
        ay[r] += (double)fy[r].x + (double)fy[r].y;
        az[r] += (double)fz[r].x + (double)fz[r].y;
      }
    } else {
#pragma unroll kRow
      for (int k = 0; k < Q; k++) {
        const double4 s = stage[warp][k];
        pairs64<GUARD>(tx, ty, tz, s.x, s.y, s.z, s.w, eps2, ax, ay, az);
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int r = 0; r < TPL; r++) {
    int j = lane + 32 * r;
    if (j < Q) {
      red[warp][0][j] = ax[r];
      red[warp][1][j] = ay[r];
      red[warp][2][j] = az[r];
    }
  }
  __syncthreads();
  const double cb = MIXED ? kBiotSavartPacked : kBiotSavartTwice;
  for (int j = threadIdx.x; j < Q; j += blockDim.x) {
    double sx = red[0][0][j], sy = red[0][1][j], sz = red[0][2][j];
    for (int w = 1; w < NW; w++) {
      sx += red[w][0][j];
      sy += red[w][1][j];
      sz += red[w][2][j];
    }
    long o = (long)t * Q + j;
    const double px = g.px[o], py = g.px[pn + o], pz = g.px[2 * pn + o];
    long oo = ALL_LEAVES ? (long)gy * 3 * out_stride + (long)tix * Q + j : o;
    long st = ALL_LEAVES ? out_stride : pn;
    out[oo] = cb * (py * sz - pz * sy);
    out[st + oo] = cb * (pz * sx - px * sz);
    out[2 * st + oo] = cb * (px * sy - py * sx);
  }
}

template <int Q, bool ALL_LEAVES, bool GUARD, bool MIXED>
__global__ void __launch_bounds__(128) k_interact_wide(StepGeom g, const double4* __restrict__ src,
                                                       const float4* __restrict__ srcf, double* __restrict__ out,
                                                       long out_stride) {
  interact_wide_body<Q, ALL_LEAVES, GUARD, MIXED>(g, blockIdx.x, blockIdx.y, gridDim.y, src, srcf, out, out_stride);
}

// Batched treecode members with q = Q: member idx[blockIdx.z], well-separated pairs.
template <int Q, bool GUARD, bool MIXED>
__global__ void __launch_bounds__(128) k_interact_wide_batch(const BatchMember* __restrict__ mem,
                                                             const int* __restrict__ idx) {
  const BatchMember& m = mem[idx[blockIdx.z]];
  const StepGeom g = m.fg;
  interact_wide_body<Q, false, GUARD, MIXED>(g, blockIdx.x, 0, 1, m.fsrc, g.srcf, m.ftgt, 0);
}

// Sum of per-group partials (group gi at partial + gi * gstride) in group order.
__global__ void k_reduce_groups(const double* __restrict__ partial, int groups, long n, long gstride,
                                double* __restrict__ out) {
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a = 0;
  for (int gi = 0; gi < groups; gi++) a += partial[(long)gi * gstride + i];
  out[i] = a;
}

// ---------------------------------------------------------------------------
// Departure points and remap.
//
// bve_find_departure_points (src/bve_time_step.cpp:172-309): backward RK4
// with k1 = v3 at x, k2 = v2 at proj(x - dt/2 k1), k3 = v1 at
// proj(x - dt/2 k2), k4 = v0 at proj(x - dt k3), and the re-projected
// combination.  bve_departure_to_target (src/bve_time_step.cpp:15-67):
// new vorticity = BLI(vor)(dep) + 2 Omega dep_z - 2 Omega z, tracers by BLI.
// mode bit 1: compute departure points (else read dep); bit 2: remap (else
// write dep).  The locations use locate_basis_rcp (one division per
// direction of the barycentric basis, reciprocals in the projections): the
// kernel is bound by float64 division and atan latency, not by its 136 bytes
// of traffic per particle.

// Whether a build with two values per load exists: rows of an even q of at most
// 16 values.  From 36 values on, the loads of a row that the compiler keeps in
// flight spill 1.5 to 5.6 KB of registers (degree 7, 393,216 particles: 388 us
// with them, 176 with one value per load at the same register bound).
constexpr bool depart_vec(int D) { return D <= 3 && (D + 1) * (D + 1) % 2 == 0; }

// VEC: the gathered fields are read two values at a time (rows on 16-byte
// boundaries).
template <int D, bool VEC>
__device__ __forceinline__ void gather_velocity(const Basis<D>& b, const double* __restrict__ v, long n, double& x,
                                                double& y, double& z) {
  if constexpr (VEC) {
    x = gather_vec<D>(b, v);
    y = gather_vec<D>(b, v + n);
    z = gather_vec<D>(b, v + 2 * n);
  } else {
    gather3<D>(b, v, n, x, y, z);
  }
}

template <int D, bool VEC>
__device__ __forceinline__ void depart_remap_body(const StepGeom& g, const BliTable& tab, long o,
                                                  const double* __restrict__ x, const double* __restrict__ y,
                                                  const double* __restrict__ z, const double* __restrict__ v0,
                                                  const double* __restrict__ v1, const double* __restrict__ v2,
                                                  const double* __restrict__ v3, double dt, double* __restrict__ dep,
                                                  const double* __restrict__ vors, const double* __restrict__ tracers,
                                                  int T, double* __restrict__ new_vors,
                                                  double* __restrict__ new_tracers, int mode) {
  const long n = (long)g.leaves * g.q;
  unsigned err = 0;
  Basis<D> b;
  double dx, dy, dz;
  if (mode & 1) {
    const double x0 = x[o], y0 = y[o], z0 = z[o];
    const double k1x = v3[o], k1y = v3[n + o], k1z = v3[2 * n + o];
    double xx = x0 - 0.5 * dt * k1x, yy = y0 - 0.5 * dt * k1y, zz = z0 - 0.5 * dt * k1z;
    project_to_sphere_rcp(xx, yy, zz);
    locate_basis_rcp<D>(g, tab, xx, yy, zz, b, err);
    double k2x, k2y, k2z;
    gather_velocity<D, VEC>(b, v2, n, k2x, k2y, k2z);
    xx = x0 - 0.5 * dt * k2x, yy = y0 - 0.5 * dt * k2y, zz = z0 - 0.5 * dt * k2z;
    project_to_sphere_rcp(xx, yy, zz);
    locate_basis_rcp<D>(g, tab, xx, yy, zz, b, err);
    double k3x, k3y, k3z;
    gather_velocity<D, VEC>(b, v1, n, k3x, k3y, k3z);
    xx = x0 - dt * k3x, yy = y0 - dt * k3y, zz = z0 - dt * k3z;
    project_to_sphere_rcp(xx, yy, zz);
    locate_basis_rcp<D>(g, tab, xx, yy, zz, b, err);
    double k4x, k4y, k4z;
    gather_velocity<D, VEC>(b, v0, n, k4x, k4y, k4z);
    xx = x0 - 1.0 / 6.0 * dt * k1x, yy = y0 - 1.0 / 6.0 * dt * k1y, zz = z0 - 1.0 / 6.0 * dt * k1z;
    project_to_sphere_rcp(xx, yy, zz);
    xx -= -1.0 / 3.0 * dt * k2x, yy -= -1.0 / 3.0 * dt * k2y, zz -= -1.0 / 3.0 * dt * k2z;
    project_to_sphere_rcp(xx, yy, zz);
    xx -= -1.0 / 3.0 * dt * k3x, yy -= -1.0 / 3.0 * dt * k3y, zz -= -1.0 / 3.0 * dt * k3z;
    project_to_sphere_rcp(xx, yy, zz);
    xx -= -1.0 / 6.0 * dt * k4x, yy -= -1.0 / 6.0 * dt * k4y, zz -= -1.0 / 6.0 * dt * k4z;
    project_to_sphere_rcp(xx, yy, zz);
    dx = xx;
    dy = yy;
    dz = zz;
    if (!(mode & 2)) {
      dep[o] = dx;
      dep[n + o] = dy;
      dep[2 * n + o] = dz;
    }
  } else {
    dx = dep[o];
    dy = dep[n + o];
    dz = dep[2 * n + o];
  }
  if (mode & 2) {
    locate_basis_rcp<D>(g, tab, dx, dy, dz, b, err);
    double vor;
    if constexpr (VEC) vor = gather_vec<D>(b, vors);
    else vor = gather<D>(b, vors);
    for (int k = 0; k < T; k++) new_tracers[o * T + k] = gather<D>(b, tracers, T, k);
    vor += 2 * g.omega * dz;
    new_vors[o] = vor - 2 * g.omega * z[o];
  }
  flag(g.err, err);
}

// Blocks of 128 threads per SM, which bound the registers of a thread.  The
// chain of four locate -> gather rounds per particle is latency-bound: up to
// degree 3, 64 registers (eight blocks) where the grid fills the SMs that
// often, and a grid of at most four blocks per SM has the registers to keep a
// round's loads in flight; above, the basis and the row's values need them at
// any size.  us per launch at 8 / 6 / 4 / 3 blocks, degree 4 at 153,600
// particles 48 / 42 / 33 / 35, 5 at 221,184 50 / 45 / 49 / 55, 6 at 301,056 95 /
// 104 / 84 / 97, 7 at 98,304 54 / 51 / 58 / 49, 9 at 153,600 111 / 100 / 88 /
// 80, 10 at 185,856 181 / 161 / 124 / 126; degree 3 at 393,216 65 / 69 / 74 /
// -.  Before (a descent per location, eight blocks throughout): degree 3 at
// 393,216 72 us, 4 42, 5 58, 6 90, 7 51, 9 118, 10 173.
constexpr int depart_blocks(int D, bool few) { return D > 6 ? 3 : D > 3 ? 4 : few ? 4 : 8; }

template <int D, int MODE, bool VEC, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) k_depart_remap(StepGeom g, BliTable tab, const double* __restrict__ x, const double* __restrict__ y,
                               const double* __restrict__ z, const double* __restrict__ v0,
                               const double* __restrict__ v1, const double* __restrict__ v2,
                               const double* __restrict__ v3, double dt, double* __restrict__ dep,
                               const double* __restrict__ vors, const double* __restrict__ tracers, int T,
                               double* __restrict__ new_vors, double* __restrict__ new_tracers,
                               VelocityOut out) {
  const long o = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const long n = (long)g.leaves * g.q;
  if (o >= n) return;
  if (out.x) {
    out.x[o] = v0[o];
    out.y[o] = v0[n + o];
    out.z[o] = v0[2 * n + o];
  }
  depart_remap_body<D, VEC>(g, tab, o, x, y, z, v0, v1, v2, v3, dt, dep, vors, tracers, T, new_vors, new_tracers, MODE);
}

// Batched members on one particle grid (member blockIdx.y): departure and
// remap in one pass (mode 3), stage velocities v_k + m * 3n, vorticity + m * n.
template <int D, bool VEC, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) k_depart_remap_batch(StepGeom g, BliTable tab, const double* __restrict__ x,
                                     const double* __restrict__ y, const double* __restrict__ z,
                                     const double* __restrict__ v0, const double* __restrict__ v1,
                                     const double* __restrict__ v2, const double* __restrict__ v3, double dt,
                                     const double* __restrict__ vors, double* __restrict__ new_vors) {
  const long n = (long)g.leaves * g.q;
  const long o = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (o >= n) return;
  const long m = blockIdx.y, vo = m * 3 * n, so = m * n;
  depart_remap_body<D, VEC>(g, tab, o, x, y, z, v0 + vo, v1 + vo, v2 + vo, v3 + vo, dt, nullptr, vors + so, nullptr, 0,
                       new_vors + so, nullptr, 3);
}

// ---------------------------------------------------------------------------
// Stand-alone direct sums over arbitrary points.  A cluster of blocks (one to
// kDirectRanks) owns a tile of targets; its blocks, and the warps (float64) or
// 64-thread groups (mixed) within a block, split the sources, and the partial
// sums are added in a fixed order over shared memory and distributed shared
// memory.  Nothing goes through device memory: with partial sums there, a call
// of 10,007 x 24,577 points spent 450 of its 790 us allocating and freeing
// them, and three more launches adding them.

constexpr int kDirectThreads = 256, kDirectRanks = 8;
constexpr int kInvLapThreads = 128;

// Adds the partial sums red[parts][3][TB] of the cluster's blocks, part by
// part and rank by rank, and writes u = cb x cross a for the targets.
template <int TB>
__device__ __forceinline__ void direct_reduce(const double* red, double* bsum, int parts, long nt,
                                              const double* __restrict__ tx, const double* __restrict__ ty,
                                              const double* __restrict__ tz, double cb, double* __restrict__ ux,
                                              double* __restrict__ uy, double* __restrict__ uz) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  __syncthreads();
  for (int k = threadIdx.x; k < 3 * TB; k += blockDim.x) {
    double a = red[k];
    for (int p = 1; p < parts; p++) a += red[p * 3 * TB + k];
    bsum[k] = a;
  }
  cl.sync();
  const int ranks = gridDim.y, share = TB / ranks;  // each rank finishes its share of the targets
  for (int j = threadIdx.x; j < share; j += blockDim.x) {
    const int k = blockIdx.y * share + j;
    const long i = (long)blockIdx.x * TB + k;
    if (i < nt) {
      double a[3] = {0, 0, 0};
      for (int r = 0; r < ranks; r++) {
        const double* b = cl.map_shared_rank(bsum, r);
#pragma unroll
        for (int c = 0; c < 3; c++) a[c] += b[c * TB + k];
      }
      const double x = tx[i], y = ty[i], z = tz[i];
      ux[i] = cb * (y * a[2] - z * a[1]);
      uy[i] = cb * (z * a[0] - x * a[2]);
      uz[i] = cb * (x * a[1] - y * a[0]);
    }
  }
  cl.sync();  // the blocks' sums stay until every rank has read them
}

// Where eps is at least kPlainEps and a tile's strengths are at most
// kPlainStrength in magnitude, a pair's g is finite and a coincident pair adds
// g * 0; any other tile (infinite strengths and NaN among them) takes the
// guarded pairs, which leave a coincident pair out whatever its g.
constexpr double kPlainEps = 1e-100, kPlainStrength = 1e200;

// float64: two targets per lane (64 per block), each warp sweeping its own
// `per` sources 32 at a time through its own tile, the next 32 loaded during
// the current ones.  The loop over a whole tile knows its length (1 x 300,000:
// 494 us against 535 with one loop for every length).  GUARD: eps below kPlainEps (negative or NaN among them).
constexpr int kDirectTile64 = 64;
constexpr size_t direct_smem64(int parts) { return sizeof(double) * (parts * (128 + 3 * kDirectTile64) + 3 * kDirectTile64); }

// The sources of a direct sum: four arrays of a caller, or a grid's sources.
struct SourceArrays {
  const double *x, *y, *z, *w;
  __device__ __forceinline__ void get(long k, double2& a, double2& b) const {
    a = make_double2(__ldg(x + k), __ldg(y + k));
    b = make_double2(__ldg(z + k), __ldg(w + k));
  }
};
struct SourceRecords {
  const double4* s;
  __device__ __forceinline__ void get(long k, double2& a, double2& b) const {
    const double2* p = reinterpret_cast<const double2*>(s + k);
    a = __ldg(p);
    b = __ldg(p + 1);
  }
};

template <bool GUARD, class Sources>
__global__ void __launch_bounds__(kDirectThreads, 4)
    k_direct_bve64(long nt, const double* __restrict__ tx, const double* __restrict__ ty,
                   const double* __restrict__ tz, long ns, Sources sources, long per, double eps,
                   double* __restrict__ ux, double* __restrict__ uy, double* __restrict__ uz) {
  constexpr int TPT = 2, TB = 32 * TPT;
  static_assert(TB == kDirectTile64, "direct_smem64");
  extern __shared__ __align__(16) double dsh[];  // a tile of 32 sources per warp, partial sums, the block's sums
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, parts = blockDim.x >> 5;
  double2* tile = reinterpret_cast<double2*>(dsh) + warp * 64;
  double* red = dsh + parts * 128;
  double x[TPT], y[TPT], z[TPT], ax[TPT], ay[TPT], az[TPT];
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    const long i = min(nt - 1, (long)blockIdx.x * TB + lane + 32 * r);
    x[r] = tx[i];
    y[r] = ty[i];
    z[r] = tz[i];
    ax[r] = ay[r] = az[r] = 0;
  }
  const double eps2 = twice_eps(eps);
  const long s0 = (blockIdx.y * parts + warp) * per, s1 = min(ns, s0 + per);
  double2 a = make_double2(0, 0), b = a;
  auto load = [&](long k) {
    if (k < s1) sources.get(k, a, b);
  };
  load(s0 + lane);
  for (long k = s0; k < s1; k += 32) {
    __syncwarp();
    tile[2 * lane] = a;
    tile[2 * lane + 1] = b;
    __syncwarp();
    const bool plain = !GUARD && __all_sync(0xffffffffu, fabs(b.y) <= kPlainStrength);
    load(k + 32 + lane);
    const int cnt = (int)min(32L, s1 - k);
    if (plain && cnt == 32) {
#pragma unroll 8
      for (int m = 0; m < 32; m++) {
        const double2 p = tile[2 * m], q = tile[2 * m + 1];
        pairs64<false>(x, y, z, p.x, p.y, q.x, q.y, eps2, ax, ay, az);
      }
    } else if (plain) {
#pragma unroll 1
      for (int m = 0; m < cnt; m++) {
        const double2 p = tile[2 * m], q = tile[2 * m + 1];
        pairs64<false>(x, y, z, p.x, p.y, q.x, q.y, eps2, ax, ay, az);
      }
    } else {
#pragma unroll 1
      for (int m = 0; m < cnt; m++) {
        const double2 p = tile[2 * m], q = tile[2 * m + 1];
        pairs64<true>(x, y, z, p.x, p.y, q.x, q.y, eps2, ax, ay, az);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    double* p = red + warp * 3 * TB + lane + 32 * r;
    p[0] = ax[r];
    p[TB] = ay[r];
    p[2 * TB] = az[r];
  }
  direct_reduce<TB>(red, red + parts * 3 * TB, parts, nt, tx, ty, tz, kBiotSavartTwice, ux, uy, uz);
}

// Mixed: 128 targets per block, two per thread (the paired float32
// instructions take one source against both), groups of 64 threads walking
// shares of the source tiles; both tiles are measured relative to their first
// point (in float64), so float32 carries only the small in-tile offsets.  The
// sources are cut into `groups`, each into tiles of 128 from its first source
// on; a tile is summed in float32, the tiles in float64.
constexpr int kDirectTile32 = 128, kDirectPart32 = 64;
constexpr size_t direct_smem32(int parts) {
  return parts * (sizeof(float4) + 3 * sizeof(double)) * kDirectTile32 + 3 * sizeof(double) * kDirectTile32;
}

__global__ void __launch_bounds__(kDirectThreads)
    k_direct_bve32(long nt, const double* __restrict__ tx, const double* __restrict__ ty,
                   const double* __restrict__ tz, long ns, const double* __restrict__ sx,
                   const double* __restrict__ sy, const double* __restrict__ sz, const double* __restrict__ sw,
                   int groups, double eps, double* __restrict__ ux, double* __restrict__ uy, double* __restrict__ uz) {
  constexpr int TB = kDirectTile32, NT = kDirectPart32;
  extern __shared__ __align__(16) double dsh[];  // a source tile per part, partial sums, the block's sums
  const int part = threadIdx.x / NT, th = threadIdx.x % NT, parts = blockDim.x / NT;
  float4* tile = reinterpret_cast<float4*>(dsh) + part * TB;
  double* red = dsh + parts * 2 * TB;
  const long i0 = blockIdx.x * (long)TB;
  const double tcx = tx[i0], tcy = ty[i0], tcz = tz[i0];
  float dtx[2], dty[2], dtz[2];
  double ax[2] = {0, 0}, ay[2] = {0, 0}, az[2] = {0, 0};
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const long i = i0 + th + NT * r;
    dtx[r] = i < nt ? (float)((tx[i] - tcx) * kPackScale) : 0.f;
    dty[r] = i < nt ? (float)((ty[i] - tcy) * kPackScale) : 0.f;
    dtz[r] = i < nt ? (float)((tz[i] - tcz) * kPackScale) : 0.f;
  }
  const float feps = (float)eps;
  const float2 eps2 = make_float2(feps, feps);
  // tile u of the sources: number u % tiles of group u / tiles (the last groups may be short or empty)
  const long per = (ns + groups - 1) / groups, tiles = (per + TB - 1) / TB, units = groups * tiles;
  const long p0 = blockIdx.y * parts + part, shares = (long)gridDim.y * parts;
  const long u0 = units * p0 / shares, u1 = units * (p0 + 1) / shares;
  long s0 = u0 / tiles * per, b = s0 + u0 % tiles * TB;
  for (long u = u0; u < u1; u++, b += TB) {
    if (b >= s0 + per) s0 += per, b = s0;
    const long s1 = min(ns, s0 + per);
    if (b >= s1) continue;
    const double scx = sx[b], scy = sy[b], scz = sz[b];
    const int cnt = (int)min((long)TB, s1 - b);
    asm volatile("bar.sync %0, %1;" : : "r"(1 + part), "n"(NT) : "memory");
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int m = th + NT * r;
      const long k = b + m;
      if (m < cnt)
        tile[m] = make_float4((float)((sx[k] - scx) * kPackScale), (float)((sy[k] - scy) * kPackScale),
                              (float)((sz[k] - scz) * kPackScale), (float)sw[k]);
    }
    asm volatile("bar.sync %0, %1;" : : "r"(1 + part), "n"(NT) : "memory");
    const float cx = (float)((scx - tcx) * kPackScale), cy = (float)((scy - tcy) * kPackScale),
                cz = (float)((scz - tcz) * kPackScale);
    const float2 bx = make_float2(cx - dtx[0], cx - dtx[1]), by = make_float2(cy - dty[0], cy - dty[1]),
                 bz = make_float2(cz - dtz[0], cz - dtz[1]);
    float2 fx = make_float2(0.f, 0.f), fy = fx, fz = fx;
#pragma unroll 8
    for (int m = 0; m < cnt; m++) {
      const float4 v = tile[m];
      pair32x2<true>(bx, by, bz, make_float2(v.x, v.x), make_float2(v.y, v.y), make_float2(v.z, v.z),
                     make_float2(v.w, v.w), eps2, fx, fy, fz);
    }
    ax[0] += fx.x;
    ay[0] += fy.x;
    az[0] += fz.x;
    ax[1] += fx.y;
    ay[1] += fy.y;
    az[1] += fz.y;
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    double* p = red + part * 3 * TB + th + NT * r;
    p[0] = ax[r];
    p[TB] = ay[r];
    p[2 * TB] = az[r];
  }
  direct_reduce<TB>(red, red + parts * 3 * TB, parts, nt, tx, ty, tz, kBiotSavartPacked, ux, uy, uz);
}

// inv_lap (src/direct_sum_impl.hpp:20-27): soln_i += sum_{j != i}
// -1/(4 pi) log(1 - x_i.x_j) area_j pots_j.
__global__ void __launch_bounds__(kInvLapThreads)
    k_inv_lap(long n, const double* __restrict__ x, const double* __restrict__ y, const double* __restrict__ z,
              const double* __restrict__ area, const double* __restrict__ pots, double* __restrict__ soln) {
  __shared__ double4 tile[kInvLapThreads];
  long i = blockIdx.x * (long)kInvLapThreads + threadIdx.x;
  double xi = 0, yi = 0, zi = 0;
  if (i < n) {
    xi = x[i];
    yi = y[i];
    zi = z[i];
  }
  double acc = 0;
  for (long b = 0; b < n; b += kInvLapThreads) {
    long k = b + threadIdx.x;
    tile[threadIdx.x] = k < n ? make_double4(x[k], y[k], z[k], area[k] * pots[k]) : make_double4(0, 0, 0, 0);
    __syncthreads();
    int cnt = (int)min((long)kInvLapThreads, n - b);
    for (int m = 0; m < cnt; m++) {
      if (b + m == i) continue;
      double4 s = tile[m];
      double dp = xi * s.x + yi * s.y + zi * s.z;
      acc += -0.07957747154594767 * log(1 - dp) * s.w;
    }
    __syncthreads();
  }
  if (i < n) soln[i] += acc;
}

// The forcing of bve_ssw_forcing (type 1) / bve_ssw_forcing_2 (type 2),
// src/forcing_funcs.cpp:6-80: one thread per leaf panel walking its points
// in order as the reference's functor does, so that bcomp carries over from
// the panel's previous point where lat <= 0 (the reference sets it only for
// lat > 0).  force = 0.6 omega a b cos(lon) (type 1) or 1.2 omega a b
// cos(2 lon) (type 2), added to the vorticity by the source kernels.
__global__ void k_ssw_forcing(int leaves, int q, int type, double omega, const double* __restrict__ time,
                              const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, double* __restrict__ force) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= leaves) return;
  const double t = *time, Tp = 4.0, Tf = 4.0 + 11.0, theta1 = kPi / 3.0;
  double acomp, bcomp = 0;
  if (t / 86400.0 < Tp) acomp = 0.5 * (1.0 - cos(kPi * (t / 86400.0) / Tp));
  else if (t / 86400.0 < Tf - Tp) acomp = 1.0;
  else if (t / 86400.0 < Tf) acomp = 0.5 * (1.0 - cos(kPi + kPi * ((t / 86400.0) - Tf + Tp) / Tp));
  else acomp = 0.0;
  for (int j = 0; j < q; j++) {
    const long o = (long)i * q + j;
    const double xx = x[o], yy = y[o], zz = z[o];
    // xyz_to_latlon, src/general_utils_impl.hpp:230-235
    const double lat = kPi / 2.0 - atan2(sqrt(xx * xx + yy * yy), zz), lon = atan2(yy, xx);
    if (lat > 0) {
      const double tt = tan(theta1), tl = tan(lat);
      const double ccomp = (tt * tt) / (tl * tl);
      bcomp = ccomp * exp(1.0 - ccomp);
    }
    force[o] = type == 1 ? 0.6 * omega * acomp * bcomp * cos(lon) : 1.2 * omega * acomp * bcomp * cos(2.0 * lon);
  }
}

__global__ void k_time_advance(double* time, double dt) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *time += dt;
}

}  // namespace

// ---------------------------------------------------------------------------
// Launch wrappers.

using dev::blocks_for;

void launch_leaf_sources(const StepGeom& g, int stage, double dt_s, const double* vprev, const double* x,
                         const double* y, const double* z, const double* vors, const double* area, double4* src,
                         cudaStream_t st, double* keep) {
  long n = (long)g.leaves * g.q;
  SB_LAUNCH(k_leaf_sources, blocks_for(n, 256), 256, 0, st, g, stage, dt_s, vprev, x, y, z, vors, area, src, keep);
}

void launch_sources_from_disp(const StepGeom& g, const double* dx, const double* dy, const double* dz,
                              const double* s, double4* src, cudaStream_t st) {
  long n = (long)g.panels * g.q;
  SB_LAUNCH(k_sources_from_disp, blocks_for(n, 256), 256, 0, st, g, dx, dy, dz, s, src);
}

void launch_copy_strength(const StepGeom& g, const double4* src, double* out, cudaStream_t st) {
  long n = (long)g.panels * g.q;
  SB_LAUNCH(k_copy_strength, blocks_for(n, 256), 256, 0, st, g, src, out);
}

// Subtree depth per launch: three levels (85 panels) for small q, one level
// for large q so that a pass has enough CTAs; shared memory holds the levels
// plus one scratch level.
static int subtree_depth(int q) { return q <= 25 ? 3 : 1; }

static size_t subtree_smem(int q, int fields, int D) {
  return (size_t)q * fields * 8 * ((((1L << (2 * (D + 1))) - 1) / 3) + (1L << (2 * D)));
}

// A thread per point of a subtree's bottom level, up to kTreeThreads.
static unsigned subtree_threads(int q, int D) {
  return std::min((unsigned)kTreeThreads, (unsigned)(((q << (2 * D)) + 31) / 32 * 32));
}

// f(std::integral_constant<int, N1>) for the node count per direction, 0 where
// no kernel is built for it.
template <class F>
static void with_n1(int degree, F f) {
  switch (degree + 1) {
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    case 9: f(std::integral_constant<int, 9>()); break;
    case 10: f(std::integral_constant<int, 10>()); break;
    case 11: f(std::integral_constant<int, 11>()); break;
    default: f(std::integral_constant<int, 0>()); break;
  }
}

void launch_upward_fused(const StepGeom& g, int mode, int stage, double dt_s, const double* vprev, const double* x,
                         const double* y, const double* z, const double* vors, const double* area, double4* src,
                         bool mixed, cudaStream_t st, double* keep) {
  with_n1(g.degree, [&](auto n1) {
    static std::atomic<unsigned long long> attr{0};
    raise_smem_once(attr, 164 * 1024, k_upward_subtree<n1.value>);
    const int Dmax = subtree_depth(g.q);
    int r = g.levels - 1;  // the bottom of the next subtree
    bool first = true;
    while (first || r > 0) {
      const int D = r < Dmax ? r : Dmax, root = r - D, roots = 6 << (2 * root);
      const unsigned threads = subtree_threads(g.q, D);
      // the non-leaf proxies' positions beside the first launch's subtrees
      const long points = first && mode == 0 ? (long)g.offset * g.q : 0;
      const int chunk = nonleaf_chunk(points, threads);
      const unsigned extra = blocks_for(points, chunk);
      SB_LAUNCH(k_upward_subtree<n1.value>, roots + extra, threads, subtree_smem(g.q, 1, D), st, g, roots, chunk, root, D,
                mode, stage, dt_s, vprev, x, y, z, vors, area, src, mixed ? 1 : 0, keep);
      r = root;
      first = false;
    }
  });
}

void launch_upward_batch(const BatchMember* mem, int members, int levels, int qmax, bool mixed, cudaStream_t st) {
  static std::atomic<unsigned long long> attr{0};
  raise_smem_once(attr, 164 * 1024, k_upward_subtree_batch);
  const int Dmax = subtree_depth(qmax);
  int r = levels - 1;
  do {
    const int D = r < Dmax ? r : Dmax;
    const int root = r - D;
    SB_LAUNCH(k_upward_subtree_batch, dim3((unsigned)(6 << (2 * root)), 1, (unsigned)members), 256,
              subtree_smem(qmax, 1, D), st, mem, root, D, mixed ? 1 : 0);
    r = root;
  } while (r > 0);
}

void launch_downward_batch(const BatchMember* mem, int members, int levels, int qmax, cudaStream_t st) {
  static std::atomic<unsigned long long> attr{0};
  raise_smem_once(attr, 164 * 1024, k_downward_subtree_batch);
  const int Dmax = subtree_depth(qmax);
  int r = 0;
  while (r < levels - 1) {
    const int D = (levels - 1 - r) < Dmax ? (levels - 1 - r) : Dmax;
    SB_LAUNCH(k_downward_subtree_batch, dim3((unsigned)(6 << (2 * r)), 1, (unsigned)members), 256,
              subtree_smem(qmax, 3, D), st, mem, r, D);
    r += D;
  }
}

void launch_cc_batch(const BatchMember* mem, const int* idx, int count, int q, int tree_panels, double eps,
                     int precision, cudaStream_t st) {
  if (count <= 0) return;
  const dim3 grid((unsigned)tree_panels, 1, (unsigned)count);
  const bool mixed = precision == SBSLPM_MIXED, guard = !(eps > 0);
#define SB_CCB(Q)                                                                                              \
  case Q:                                                                                                      \
    if (mixed) {                                                                                               \
      if (guard) SB_LAUNCH((k_interact_wide_batch<Q, true, true>), grid, 128, 0, st, mem, idx);                \
      else SB_LAUNCH((k_interact_wide_batch<Q, false, true>), grid, 128, 0, st, mem, idx);                     \
    } else {                                                                                                   \
      if (guard) SB_LAUNCH((k_interact_wide_batch<Q, true, false>), grid, 128, 0, st, mem, idx);               \
      else SB_LAUNCH((k_interact_wide_batch<Q, false, false>), grid, 128, 0, st, mem, idx);                    \
    }                                                                                                          \
    break;
  switch (q) {
    SB_CCB(36) SB_CCB(49) SB_CCB(64) SB_CCB(81) SB_CCB(100) SB_CCB(121)
  }
#undef SB_CCB
}

void launch_downward_fused(const StepGeom& g, double* tgt, double* leaf_out, cudaStream_t st) {
  with_n1(g.degree, [&](auto n1) {
    static std::atomic<unsigned long long> attr{0};
    raise_smem_once(attr, 164 * 1024, k_downward_subtree<n1.value>);
    const int Dmax = subtree_depth(g.q);
    int r = 0;
    while (r < g.levels - 1) {
      const int D = (g.levels - 1 - r) < Dmax ? (g.levels - 1 - r) : Dmax;
      SB_LAUNCH(k_downward_subtree<n1.value>, (unsigned)(6 << (2 * r)), subtree_threads(g.q, D),
                subtree_smem(g.q, 3, D), st, g, r, D, tgt, leaf_out);
      r += D;
    }
  });
}

namespace {
template <int Q, bool GUARD>
void interact_qg(const StepGeom& g, int precision, const double4* src, double* out, cudaStream_t st, bool pack) {
  const int tp = g.panels;
  if (precision == SBSLPM_MIXED && pack)
    SB_LAUNCH(k_pack_mixed, blocks_for((long)g.panels * g.q, 256), 256, 0, st, g, src, g.srcf);
  if constexpr (Q > 32) {
    if (precision == SBSLPM_MIXED)
      SB_LAUNCH((k_interact_wide<Q, false, GUARD, true>), tp, 128, 0, st, g, src, g.srcf, out, 0L);
    else
      SB_LAUNCH((k_interact_wide<Q, false, GUARD, false>), tp, 128, 0, st, g, src, g.srcf, out, 0L);
  } else if (precision == SBSLPM_MIXED) {
    constexpr int NW = dev::ListShape32<Q, 1>::NW, threads = 32 * NW;
    const int wpt = dev::list_warps<Q, 1, true>(tp);
    if (wpt == NW)
      SB_LAUNCH((k_interact32<Q, NW, false, GUARD>), tp, threads, 0, st, g, g.srcf, out, 0L);
    else if (wpt == 2)
      SB_LAUNCH((k_interact32<Q, 2, false, GUARD>), blocks_for(tp, NW / 2), threads, 0, st, g, g.srcf, out, 0L);
    else
      SB_LAUNCH((k_interact32<Q, 1, false, GUARD>), blocks_for(tp, NW), threads, 0, st, g, g.srcf, out, 0L);
  } else {
    constexpr int NW = dev::ListShape<Q, 1>::NW, threads = 32 * NW;
    const int wpt = dev::list_warps<Q, 1, false>(tp);
    if (wpt == NW)
      SB_LAUNCH((k_interact64<Q, NW, GUARD>), tp, threads, 0, st, g, src, out);
    else if (wpt == 2)
      SB_LAUNCH((k_interact64<Q, 2, GUARD>), blocks_for(tp, NW / 2), threads, 0, st, g, src, out);
    else
      SB_LAUNCH((k_interact64<Q, 1, GUARD>), blocks_for(tp, NW), threads, 0, st, g, src, out);
  }
}

// Every leaf against every leaf, mixed precision, `groups` groups of source
// leaves whose partial sums go to out [group][3][leaves*q].
template <int Q, bool GUARD>
void leaves_qg(const StepGeom& g, double* out, int groups, cudaStream_t st) {
  const long n = (long)g.leaves * Q;
  if constexpr (Q > 32) {
    SB_LAUNCH((k_interact_wide<Q, true, GUARD, true>), dim3((unsigned)g.leaves, groups), 128, 0, st, g, nullptr, g.srcf,
              out, n);
  } else {
    constexpr int NW = dev::ListShape32<Q, 1>::NW;
    SB_LAUNCH((k_interact32<Q, 1, true, GUARD>), dim3(blocks_for(g.leaves, NW), groups), 32 * NW, 0, st, g, g.srcf, out,
              n);
  }
}

// The coincident-point guard is compiled in only when kernel_eps = 0.
void interact_dispatch(const StepGeom& g, int precision, const double4* src, double* out, cudaStream_t st,
                       bool pack) {
#define SB_IQ(Q)                                                             \
  case Q:                                                                    \
    if (g.eps > 0) interact_qg<Q, false>(g, precision, src, out, st, pack);  \
    else interact_qg<Q, true>(g, precision, src, out, st, pack);             \
    break;
  switch (g.q) {
    SB_IQ(1) SB_IQ(4) SB_IQ(9) SB_IQ(16) SB_IQ(25) SB_IQ(36) SB_IQ(49) SB_IQ(64) SB_IQ(81) SB_IQ(100) SB_IQ(121)
  }
#undef SB_IQ
}

void leaves_dispatch(const StepGeom& g, double* out, int groups, cudaStream_t st) {
#define SB_LQ(Q)                                                 \
  case Q:                                                        \
    if (g.eps > 0) leaves_qg<Q, false>(g, out, groups, st);      \
    else leaves_qg<Q, true>(g, out, groups, st);                 \
    break;
  switch (g.q) {
    SB_LQ(16) SB_LQ(25) SB_LQ(36) SB_LQ(49) SB_LQ(64) SB_LQ(81) SB_LQ(100) SB_LQ(121)
  }
#undef SB_LQ
}

// Independent FMA chains (8 per thread) so the pipe, not latency, limits throughput.
__global__ void k_fma_probe32(int iters, float* out) {
  float a[8];
  for (int k = 0; k < 8; k++) a[k] = threadIdx.x * 1e-7f + k;
  const float m = 0.999999f, c = 1e-7f;
  for (int i = 0; i < iters; i++)
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = fmaf(a[k], m, c);
  float s = 0;
  for (int k = 0; k < 8; k++) s += a[k];
  if (s == 12345.678f) out[0] = s;  // keeps the chains live
}
__global__ void k_fma_probe64(int iters, double* out) {
  double a[8];
  for (int k = 0; k < 8; k++) a[k] = threadIdx.x * 1e-7 + k;
  const double m = 0.999999, c = 1e-7;
  for (int i = 0; i < iters; i++)
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = fma(a[k], m, c);
  double s = 0;
  for (int k = 0; k < 8; k++) s += a[k];
  if (s == 12345.678) out[0] = s;
}
}  // namespace

void launch_interactions(const StepGeom& g, int precision, const double4* src, double* tgt, bool accumulate,
                         cudaStream_t st) {
  interact_dispatch(g, precision, src, tgt, st, true);
}

void launch_interactions_only(const StepGeom& g, int precision, const double4* src, double* tgt, cudaStream_t st) {
  interact_dispatch(g, precision, src, tgt, st, false);
}

void launch_pack_mixed(const StepGeom& g, const double4* src, cudaStream_t st) {
  long pn = (long)g.panels * g.q;
  SB_LAUNCH(k_pack_mixed, blocks_for(pn, 256), 256, 0, st, g, src, g.srcf);
}

void launch_fma_probe(int kind, int blocks, int iters, float* out32, double* out64, cudaStream_t st) {
  if (kind == 0)
    SB_LAUNCH(k_fma_probe32, blocks, 256, 0, st, iters, out32);
  else
    SB_LAUNCH(k_fma_probe64, blocks, 256, 0, st, iters, out64);
}

static bool aligned16(std::initializer_list<const double*> ps) {
  for (const double* p : ps)
    if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
  return true;
}

// f(std::integral_constant<int, degree>).
template <class F>
static void with_degree(int degree, F f) {
  switch (degree) {
#define SB_DEGREE(D)                            \
  case D:                                       \
    f(std::integral_constant<int, D>());        \
    break;
    SB_DEGREE(0) SB_DEGREE(1) SB_DEGREE(2) SB_DEGREE(3) SB_DEGREE(4) SB_DEGREE(5) SB_DEGREE(6) SB_DEGREE(7)
    SB_DEGREE(8) SB_DEGREE(9) SB_DEGREE(10)
#undef SB_DEGREE
  }
}

void launch_depart_remap(const StepGeom& g, const BliTable* tab, const double* x, const double* y, const double* z,
                         const double* v0, const double* v1, const double* v2, const double* v3, double dt,
                         double* dep, const double* vors, const double* tracers, int T, double* new_vors,
                         double* new_tracers, int mode, cudaStream_t st, VelocityOut vel) {
  long n = (long)g.leaves * g.q;
  const unsigned grid = blocks_for(n, 128);
  const bool vec = aligned16({v0, v1, v2, vors}) && n % 2 == 0, few = grid <= 4 * 148;
  with_degree(g.degree, [&](auto d) {
    constexpr int D = d.value;
    auto launch = [&](auto m, auto v, auto f) {
      SB_LAUNCH((k_depart_remap<D, m.value, v.value, depart_blocks(D, f.value)>), grid, 128, 0, st, g, *tab, x, y, z, v0,
                v1, v2, v3, dt, dep, vors, tracers, T, new_vors, new_tracers, vel);
    };
    auto sized = [&](auto m, auto v) {
      if (few) launch(m, v, std::true_type());
      else launch(m, v, std::false_type());
    };
    auto loads = [&](auto m) {
      if (depart_vec(D) && vec) sized(m, std::bool_constant<depart_vec(D)>());
      else sized(m, std::false_type());
    };
    if (mode == 1) loads(std::integral_constant<int, 1>());
    else if (mode == 2) loads(std::integral_constant<int, 2>());
    else loads(std::integral_constant<int, 3>());
  });
}

void launch_depart_remap_batch(const StepGeom& g, const BliTable* tab, int members, const double* x,
                               const double* y, const double* z, const double* v0, const double* v1,
                               const double* v2, const double* v3, double dt, const double* vors, double* new_vors,
                               cudaStream_t st) {
  const long n = (long)g.leaves * g.q;
  const dim3 grid(blocks_for(n, 128), (unsigned)members);
  const bool vec = aligned16({v0, v1, v2, vors}) && n % 2 == 0, few = (long)grid.x * members <= 4 * 148;
  with_degree(g.degree, [&](auto d) {
    constexpr int D = d.value;
    auto launch = [&](auto v, auto f) {
      SB_LAUNCH((k_depart_remap_batch<D, v.value, depart_blocks(D, f.value)>), grid, 128, 0, st, g, *tab, x, y, z, v0,
                v1, v2, v3, dt, vors, new_vors);
    };
    auto sized = [&](auto v) {
      if (few) launch(v, std::true_type());
      else launch(v, std::false_type());
    };
    if (depart_vec(D) && vec) sized(std::bool_constant<depart_vec(D)>());
    else sized(std::false_type());
  });
}

// Source groups of the mixed direct sum (a group's tiles start at its own
// first source): enough groups for a few blocks per SM, none below 1,024
// sources, 64 at most.
int direct_groups(long nt, long ns) {
  const long tblocks = (nt + 127) / 128;
  const long want = (4L * 148 * 8 + tblocks - 1) / tblocks, maxg = (ns + 1023) / 1024;
  const long gsel = want < maxg ? want : maxg;
  return (int)(gsel < 1 ? 1 : (gsel > 64 ? 64 : gsel));
}

// Shares of the sources per tile of targets, a power of two: as many as give
// the GPU `want` parts (warps or 64-thread groups) in all, none without a
// source tile of its own, kDirectRanks blocks of max_parts at most; a block
// takes them before the cluster does.  Few targets need all 64 shares to reach
// every SM, many targets none, and a share without sources only waits and is
// added: us per call with eight full blocks for every tile of targets and by
// this rule, 10,007 x 24,577 points 260 / 256 (float64), 191 / 165 (mixed);
// 100,000 x 12,000 1,106 / 1,116, 1,984 / 682; 600,000 x 33 756 / 64, 418 / 62;
// 2,000,000 x 3,000 5,695 / 5,220, 42,200 / 2,660.
struct DirectShape {
  unsigned parts, ranks;
};
static DirectShape direct_shape(long target_tiles, long source_tiles, long want, unsigned max_parts) {
  unsigned shares = 1;
  while (shares < kDirectRanks * max_parts && shares < source_tiles && target_tiles * shares < want) shares *= 2;
  const unsigned parts = std::min(shares, max_parts);
  return {parts, shares / parts};
}

constexpr long kDirectWaves = 16L * 148;  // of 32 warps (float64) or 16 64-thread groups per SM

template <class Sources>
static void launch_direct64(long nt, const double* tx, const double* ty, const double* tz, long ns,
                            const Sources& sources, double eps, double* ux, double* uy, double* uz, cudaStream_t st) {
  const unsigned blocks = blocks_for(nt, kDirectTile64);
  const DirectShape d = direct_shape(blocks, (ns + 31) / 32, 32 * kDirectWaves, kDirectThreads / 32);
  const long per = (ns + d.parts * d.ranks - 1) / (d.parts * d.ranks);  // sources of a warp
  launch_cluster(eps >= kPlainEps ? k_direct_bve64<false, Sources> : k_direct_bve64<true, Sources>, blocks, d.ranks,
                 32 * d.parts, direct_smem64(d.parts), st, nt, tx, ty, tz, ns, sources, per, eps, ux, uy, uz);
}

void launch_direct_bve(long nt, const double* tx, const double* ty, const double* tz, long ns, const double* sx,
                       const double* sy, const double* sz, const double* s, double eps, int precision, int groups,
                       double* ux, double* uy, double* uz, cudaStream_t st) {
  if (precision == SBSLPM_MIXED) {
    const unsigned blocks = blocks_for(nt, kDirectTile32);
    const long per = (ns + groups - 1) / groups, units = groups * ((per + kDirectTile32 - 1) / kDirectTile32);
    const DirectShape d = direct_shape(blocks, units, 16 * kDirectWaves, kDirectThreads / kDirectPart32);
    launch_cluster(k_direct_bve32, blocks, d.ranks, d.parts * kDirectPart32, direct_smem32(d.parts), st, nt, tx, ty, tz,
                   ns, sx, sy, sz, s, groups, eps, ux, uy, uz);
    return;
  }
  launch_direct64(nt, tx, ty, tz, ns, SourceArrays{sx, sy, sz, s}, eps, ux, uy, uz, st);
}

// Source groups of a grid's direct sum by panels: blocks of four warps for
// about 10 per SM and six groups at least (short last rounds on large grids),
// each a whole number of a warp's source splits (its rounds are then full).  us
// of a step's sums with 64 * 148 / leaves groups and with this rule: shallow
// water at levels 3, 9 points a panel 77 / 37, 16 74 / 44, 25 189 / 83
// (float64), 70 / 34, 60 / 35, 84 / 57 (mixed); mixed velocity, 16 points at
// levels 5 1,183 / 1,183, levels 6 19,160 / 17,290.
int direct_leaf_groups(int leaves, int q) {
  const int most = 64;
  if (q > 25) return std::max(1, std::min(most, 148 * 64 / leaves));
  const int splits = q <= 1 ? ListShape<1, 1>::S : q <= 4 ? ListShape<4, 1>::S : q <= 9 ? ListShape<9, 1>::S
                     : q <= 16 ? ListShape<16, 1>::S : ListShape<25, 1>::S;
  const int want = std::max(6, std::min(most, 148 * 40 / leaves)), per = (leaves + want - 1) / want;
  const int full = (per + splits - 1) / splits * splits;
  return (leaves + full - 1) / full;
}

// The grid's direct velocity.  In float64, and mixed up to nine points a panel,
// as a direct sum over points (mixed pairs need a panel's common centre, which
// costs more than they save on few points); else by panels, in source groups.
// us per step by panels, one target per lane / by points, float64 at levels 5, 4
// points a panel 471 / 185, levels 4, 9 points 132 / 96, 49 points 1,865 / 1,323.
void launch_direct_leaves(const StepGeom& g, int precision, const double4* src, double* vout, double* partial,
                          int groups, cudaStream_t st) {
  const long n = (long)g.leaves * g.q, pn = (long)g.panels * g.q, off = (long)g.offset * g.q;
  if (precision != SBSLPM_MIXED || g.q <= 9) {
    launch_direct64(n, g.px + off, g.px + pn + off, g.px + 2 * pn + off, n, SourceRecords{src + off}, g.eps, vout,
                    vout + n, vout + 2 * n, st);
    return;
  }
  launch_pack_mixed(g, src, st);
  leaves_dispatch(g, partial, groups, st);
  SB_LAUNCH(k_reduce_groups, blocks_for(3 * n, 256), 256, 0, st, partial, groups, 3 * n, 3 * n, vout);
}

void launch_ssw_forcing(int leaves, int q, int type, double omega, const double* time, const double* x,
                        const double* y, const double* z, double* force, cudaStream_t st) {
  SB_LAUNCH(k_ssw_forcing, blocks_for(leaves, 128), 128, 0, st, leaves, q, type, omega, time, x, y, z, force);
}

void launch_time_advance(double* time, double dt, cudaStream_t st) {
  SB_LAUNCH(k_time_advance, 1, 32, 0, st, time, dt);
}

void launch_inv_lap(long n, const double* x, const double* y, const double* z, const double* area,
                    const double* pots, double* soln, cudaStream_t st) {
  SB_LAUNCH(k_inv_lap, blocks_for(n, kInvLapThreads), kInvLapThreads, 0, st, n, x, y, z, area, pots, soln);
}

}  // namespace sbslpm
