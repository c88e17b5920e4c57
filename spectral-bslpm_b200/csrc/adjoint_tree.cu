// Adjoint of the decoupled-degree treecode velocity (float64): the reverse
// of k_bltc_sources -> upward pass -> well-separated proxy interactions ->
// downward pass -> leaf interpolation + near field.  Every forward piece is
// linear in the strengths; the source positions enter the near field and the
// anterpolation onto the leaf proxies (the proxies themselves are fixed):
//
//   v_i      = near_i + sum_k B_k(x_i) T_leaf(i),k          B: leaf-box BLI basis (fixed)
//   T        = D (cc(Q))                                    D: downward pass
//   cc(Q)_t  = K x_t x sum_s sum_k g (y_k - x_t) Q_s,k       fixed proxies x_t, y_k
//   Q        = U (A(y) q)                                   U: upward pass, A: anterpolation
//   near_i   = K x_i x sum_j g (y_j - x_i) q_j              near leaf pairs
//
// Reverse: Tbar_leaf = B^T vbar; Tbar = D^T Tbar (an upward accumulation of
// three fields); Qbar_s = cc^T(Tbar) (a source-owned sum over the transposed
// well-separated list); Qbar = U^T Qbar (a downward accumulation); then per
// particle qbar_j = [A^T Qbar]_j + near^T, ybar_j = q_j grad_y(A^T Qbar) +
// near^T, with near^T the source-owned sum over the transposed near list.
//
// The reference's own spectral FMM (proxies = the panels' interp_degree
// points, displaced and re-projected at every stage; bve_vel_impl.hpp:85-122,
// bve_time_step.cpp:69-170) reverses the same way on the panel quadtree, with
// two differences: the interactions' sources move, so their transpose also
// gives position adjoints, and a non-leaf proxy's displacement is the BLI
// interpolation of its containing leaf's (bve_disp_interp), whose transpose
// scatters back onto the leaf velocities.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "adjoint_pair32.cuh"
#include "adjoint_tree.cuh"
#include "device_common.cuh"
#include "leaf_moments.cuh"

namespace sbslpm {
namespace {

using namespace dev;

constexpr int kT = 128;

constexpr int kLeafThreads = 256;

// Blocks of a cluster that share a source panel or leaf: enough that the tree
// gives each SM about eight blocks (the 96 leaves of a 24,576-particle tree
// left a third of the SMs without one), at most the portable eight.
unsigned split_ranks(int units) {
  unsigned r = 1;
  while (r < 8 && units * (int)r < 8 * 148) r *= 2;
  return r;
}

// Tbar_leaf[c][k] = sum_i B_k(x_i) vbar_c,i over the leaf's particles, one
// block per (leaf, component c), a direction at a time.
__global__ void __launch_bounds__(kLeafThreads) k_tree_to_particles_T(TreeGeom tg, StepGeom fg,
                                                                     const double* __restrict__ vbar,
                                                                     double* __restrict__ tbar) {
  extern __shared__ double sh[];  // npl values, side n1 half-contracted
  const int f = blockIdx.x, c = blockIdx.y, npl = tg.npl, qx = (tg.n + 1) * (tg.n + 1);
  double* to = tbar + c * (long)fg.panels * qx + (long)(fg.offset + f) * qx;
  for (int i = threadIdx.x; i < npl; i += blockDim.x) sh[grid_slot(tg, i)] = vbar[c * tg.N + (long)f * npl + i];
  __syncthreads();
  grid_moments(tg, sh, sh + npl, [&](int m, double s) { to[m] = s; });
}

// One level of the transpose of the downward pass: a parent at `level` adds
// the anterpolation of its children's fields (child_to_parent form), one
// direction at a time as in the forward pass, a block per (parent, field).
__global__ void __launch_bounds__(kT) k_tree_up3(StepGeom fg, int level, double* __restrict__ t) {
  extern __shared__ double sh[];  // 4 children, 4 half-contracted
  const int n1 = fg.degree + 1, q = fg.q;
  const long pn = (long)fg.panels * q;
  const int p = blockIdx.x;  // relative to the level
  double* field = t + blockIdx.y * pn;
  const double* ch = field + ((long)level_start(level + 1) + 4 * p) * q;
  double* half = sh + 4 * q;
  for (int k = threadIdx.x; k < 4 * q; k += blockDim.x) sh[k] = ch[k];
  __syncthreads();
  for (int k = threadIdx.x; k < 4 * q; k += blockDim.x) {  // half[c][i][b] = sum_j Ly_c[j][b] S_c[i][j]
    const int c = k / q, i = (k - c * q) / n1, b = k % n1;
    const double* ly = fg.child_1d + (c >= 2 ? n1 * n1 : 0) + b;
    const double* sc = sh + c * q + i * n1;
    double acc = 0;
    for (int j = 0; j < n1; j++) acc = fma(__ldg(ly + j * n1), sc[j], acc);
    half[k] = acc;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < q; k += blockDim.x) {
    const int a = k / n1, b = k - a * n1;
    double acc = 0;
    for (int c = 0; c < 4; c++) {
      const double* lx = fg.child_1d + ((c == 1 || c == 2) ? n1 * n1 : 0) + a;
      const double* hc = half + c * q + b;
      for (int i = 0; i < n1; i++) acc = fma(__ldg(lx + i * n1), hc[i * n1], acc);
    }
    field[((long)level_start(level) + p) * q + k] += acc;
  }
}

// One level of the transpose of the upward pass: the children of `level` add
// the interpolation of their parent's (final) adjoint strengths, a block per
// parent.
__global__ void __launch_bounds__(kT) k_tree_down1(StepGeom fg, int level, double* __restrict__ qb) {
  extern __shared__ double sh[];  // the parent, 2 halves contracted in eta
  const int n1 = fg.degree + 1, q = fg.q, p = blockIdx.x;
  const double* parent = qb + ((long)level_start(level) + p) * q;
  double* ch = qb + ((long)level_start(level + 1) + 4 * p) * q;
  double* half = sh + q;
  for (int k = threadIdx.x; k < q; k += blockDim.x) sh[k] = parent[k];
  __syncthreads();
  for (int k = threadIdx.x; k < 2 * q; k += blockDim.x) {  // half[e][a][j] = sum_b Ly_e[j][b] Q[a][b]
    const int e = k / q, a = (k - e * q) / n1, j = k % n1;
    const double* ly = fg.child_1d + e * n1 * n1 + j * n1;
    double acc = 0;
    for (int b = 0; b < n1; b++) acc = fma(__ldg(ly + b), sh[a * n1 + b], acc);
    half[k] = acc;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 4 * q; k += blockDim.x) {
    const int c = k / q, i = (k - c * q) / n1, j = k % n1;
    const double* lx = fg.child_1d + ((c == 1 || c == 2) ? n1 * n1 : 0) + i * n1;
    const double* h = half + (c >= 2 ? q : 0) + j;
    double acc = 0;
    for (int a = 0; a < n1; a++) acc = fma(__ldg(lx + a), h[a * n1], acc);
    ch[k] += acc;
  }
}

// Adds the cluster's partial sums v (COUNT values of each of `n` items, this
// block's at sum[COUNT][n] in shared memory) rank by rank and calls
// done(item, totals) for this rank's share of the items.
template <int COUNT, class Done>
__device__ __forceinline__ void cluster_totals(double* sum, int n, const Done& done) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  cl.sync();
  const int ranks = (int)cl.num_blocks(), share = (n + ranks - 1) / ranks, i0 = (int)cl.block_rank() * share;
  for (int i = i0 + threadIdx.x; i < min(n, i0 + share); i += blockDim.x) {
    double tot[COUNT];
#pragma unroll
    for (int c = 0; c < COUNT; c++) tot[c] = 0;
    for (int r = 0; r < ranks; r++) {
      const double* b = cl.map_shared_rank(sum, r);
#pragma unroll
      for (int c = 0; c < COUNT; c++) tot[c] += b[c * n + i];
    }
    done(i, tot);
  }
  cl.sync();  // the sums stay until every rank has read them
}

// Transposed well-separated interactions: source panel s (blockIdx.x) sums
// over the target panels t whose list holds s: Qbar_s,k = K sum_t sum_i g c.d,
// c = Tbar_t,i x x_i, d = y_k - x_i.  A thread per source proxy; the cluster's
// blocks (split_ranks) take the list's entries in turn.
template <bool GUARD>
__global__ void __launch_bounds__(kT) k_tree_cc_T(StepGeom fg, const int* __restrict__ tstart,
                                                 const int* __restrict__ ttgt, const double* __restrict__ tbar,
                                                 double* __restrict__ qbar) {
  __shared__ __align__(16) double2 tile[kT][3];  // x, y | z, cx | cy, cz
  __shared__ double sum[kT];
  const int s = blockIdx.x, q = fg.q;
  const long pn = (long)fg.panels * q;
  const int k = threadIdx.x;
  double yx = 0, yy = 0, yz = 0;
  if (k < q) {
    yx = fg.px[(long)s * q + k];
    yy = fg.px[pn + (long)s * q + k];
    yz = fg.px[2 * pn + (long)s * q + k];
  }
  double acc = 0;
  for (int e = tstart[s] + blockIdx.y; e < tstart[s + 1]; e += gridDim.y) {
    const long tb = (long)ttgt[e] * q;
    __syncthreads();
    if (k < q) {
      const double x = fg.px[tb + k], y = fg.px[pn + tb + k], z = fg.px[2 * pn + tb + k];
      const double a = tbar[tb + k], b = tbar[pn + tb + k], c = tbar[2 * pn + tb + k];
      tile[k][0] = make_double2(x, y);
      tile[k][1] = make_double2(z, b * z - c * y);
      tile[k][2] = make_double2(c * x - a * z, a * y - b * x);
    }
    __syncthreads();
    if (k < q) {
#pragma unroll 4
      for (int i = 0; i < q; i++) {
        const double2 A = tile[i][0], B = tile[i][1], C = tile[i][2];
        const double dx = yx - A.x, dy = yy - A.y, dz = yz - B.x;
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        double g = recip_nr(fma(0.5, r2, fg.eps));
        if (GUARD) g = r2 > 0.0 ? g : 0.0;
        acc = fma(g, fma(B.y, dx, fma(C.x, dy, C.y * dz)), acc);
      }
    }
  }
  if (k < q) sum[k] = acc;
  cluster_totals<1>(sum, q, [&](int i, const double* v) { qbar[(long)s * q + i] = kBiotSavart * v[0]; });
}

// Transposed near field: blockIdx.x = (source leaf sl, chunk of 2 NT of its
// particles), two source particles per thread, over the target leaves whose
// near list holds sl, cut into tiles of 64 targets that the cluster's blocks
// (split_ranks) share out.  Writes qbar_j
// and ybar_j (3 components) of the leaf's particles.  One block of 256 threads
// per leaf took 345 us at 24,576 particles (96 blocks), this 215 us: bound by
// the FP64 pipe and its register reads (22 operations a pair, 9 of them with
// three different registers).
template <int NT, bool GUARD>
__global__ void __launch_bounds__(NT) k_tree_near_T(TreeGeom tg, const int* __restrict__ tstart,
                                                   const int* __restrict__ ttgt, const double* __restrict__ x,
                                                   const double* __restrict__ y, const double* __restrict__ z,
                                                   const double* __restrict__ vbar, const double4* __restrict__ psrc,
                                                   double* __restrict__ qbar, double* __restrict__ ybar) {
  constexpr int TPT = 2, TS = 64, NSRC = TPT * NT;
  __shared__ __align__(16) double2 tile[TS][3];  // x, y | z, cx | cy, cz with c = vbar x x
  __shared__ double sum[4 * NSRC];
  const int npl = tg.npl, chunks = (npl + NSRC - 1) / NSRC, sl = blockIdx.x / chunks;
  const int first = (blockIdx.x - sl * chunks) * NSRC, count = min(NSRC, npl - first);
  const long N = tg.N, o0 = (long)sl * npl + first;
  double sx[TPT], sy[TPT], sz[TPT], qb[TPT], bx[TPT], by[TPT], bz[TPT];
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    const int j = threadIdx.x + r * NT;
    const double4 s = psrc[o0 + (j < count ? j : 0)];
    sx[r] = s.x;
    sy[r] = s.y;
    sz[r] = s.z;
    qb[r] = bx[r] = by[r] = bz[r] = 0;
  }
  const int e0 = tstart[sl], tiles = (npl + TS - 1) / TS;
  const long total = (long)(tstart[sl + 1] - e0) * tiles;
  const long t1 = total * (blockIdx.y + 1) / gridDim.y;
  for (long tt = total * blockIdx.y / gridDim.y; tt < t1; tt++) {
    const int i0 = (int)(tt % tiles) * TS, cnt = min(TS, npl - i0);
    const long tb = (long)ttgt[e0 + tt / tiles] * npl + i0;
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += NT) {
      const double a = vbar[tb + i], b = vbar[N + tb + i], c = vbar[2 * N + tb + i];
      const double px = x[tb + i], py = y[tb + i], pz = z[tb + i];
      tile[i][0] = make_double2(px, py);
      tile[i][1] = make_double2(pz, b * pz - c * py);
      tile[i][2] = make_double2(c * px - a * pz, a * py - b * px);
    }
    __syncthreads();
    // not unrolled: 64 registers either way, and 195 us against 216 us with four
#pragma unroll 1
    for (int i = 0; i < cnt; i++) {
      const double2 A = tile[i][0], B = tile[i][1], C = tile[i][2];
      // step by step for both sources: an operand held over from the
      // instruction before saves a register read (pairs64)
      double dx[TPT], dy[TPT], dz[TPT], g[TPT], u[TPT], t[TPT];
#pragma unroll
      for (int r = 0; r < TPT; r++) dx[r] = sx[r] - A.x;
#pragma unroll
      for (int r = 0; r < TPT; r++) dy[r] = sy[r] - A.y;
#pragma unroll
      for (int r = 0; r < TPT; r++) dz[r] = sz[r] - B.x;
#pragma unroll
      for (int r = 0; r < TPT; r++) {
        const double r2 = fma(dx[r], dx[r], fma(dy[r], dy[r], dz[r] * dz[r]));
        g[r] = recip_nr(fma(0.5, r2, tg.eps));
        if (GUARD) g[r] = r2 > 0.0 ? g[r] : 0.0;
      }
#pragma unroll
      for (int r = 0; r < TPT; r++) u[r] = C.y * dz[r];
#pragma unroll
      for (int r = 0; r < TPT; r++) u[r] = fma(C.x, dy[r], u[r]);
#pragma unroll
      for (int r = 0; r < TPT; r++) u[r] = fma(B.y, dx[r], u[r]);
#pragma unroll
      for (int r = 0; r < TPT; r++) {
        u[r] = g[r] * u[r];
        qb[r] += u[r];
        t[r] = -g[r] * u[r];
      }
#pragma unroll
      for (int r = 0; r < TPT; r++) {
        bx[r] = fma(t[r], dx[r], bx[r]);
        by[r] = fma(t[r], dy[r], by[r]);
        bz[r] = fma(t[r], dz[r], bz[r]);
        bx[r] = fma(g[r], B.y, bx[r]);
        by[r] = fma(g[r], C.x, by[r]);
        bz[r] = fma(g[r], C.y, bz[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    const int j = threadIdx.x + r * NT;
    sum[j] = qb[r];
    sum[NSRC + j] = bx[r];
    sum[2 * NSRC + j] = by[r];
    sum[3 * NSRC + j] = bz[r];
  }
  cluster_totals<4>(sum, NSRC, [&](int j, const double* v) {
    if (j >= count) return;
    const long o = o0 + j;
    const double w = kBiotSavart * psrc[o].w;
    qbar[o] = kBiotSavart * v[0];
    ybar[o] = w * v[1];
    ybar[N + o] = w * v[2];
    ybar[2 * N + o] = w * v[3];
  });
}

// Mixed-precision transposed near field: source leaf sl (blockIdx.x), one
// thread per source particle; per target leaf of the transposed list the
// float32 sums are added into float64.
template <bool GUARD>
__global__ void __launch_bounds__(512) k_tree_near_T32(TreeGeom tg, StepGeom fg, const int* __restrict__ tstart,
                                                     const int* __restrict__ ttgt, const double* __restrict__ x,
                                                     const double* __restrict__ y, const double* __restrict__ z,
                                                     const double* __restrict__ vbar,
                                                     const double4* __restrict__ psrc, double* __restrict__ qbar,
                                                     double* __restrict__ ybar) {
  extern __shared__ float4 tile32[];  // [(npl+1)/2][3]
  const int sl = blockIdx.x, npl = tg.npl, np2 = (npl + 1) >> 1;
  const long N = tg.N;
  const int j = threadIdx.x;
  const long oj = (long)sl * npl + (j < npl ? j : 0);
  const double4 s = psrc[oj];
  const double* cs = fg.pd_centre + 4 * (long)(fg.offset + sl);
  const float sx = (float)((s.x - cs[0]) * kPackScale), sy = (float)((s.y - cs[1]) * kPackScale),
              sz = (float)((s.z - cs[2]) * kPackScale);
  const float feps = (float)tg.eps;
  const float2 eps2 = make_float2(feps, feps);
  double qb = 0, bx = 0, by = 0, bz = 0;
  for (int e = tstart[sl]; e < tstart[sl + 1]; e++) {
    const int tl = ttgt[e];
    const long tb = (long)tl * npl;
    const double* ct = fg.pd_centre + 4 * (long)(fg.offset + tl);
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * np2; i += blockDim.x) {
      if (i < npl)
        adj_stage(tile32, i, x[tb + i], y[tb + i], z[tb + i], vbar[tb + i], vbar[N + tb + i], vbar[2 * N + tb + i],
                  ct);
      else
        adj_stage_zero(tile32, i);
    }
    __syncthreads();
    const float a0 = sx + (float)((cs[0] - ct[0]) * kPackScale), a1 = sy + (float)((cs[1] - ct[1]) * kPackScale),
                a2 = sz + (float)((cs[2] - ct[2]) * kPackScale);
    const float2 ax = make_float2(a0, a0), ay = make_float2(a1, a1), az = make_float2(a2, a2);
    float2 q = make_float2(0.f, 0.f), cx = q, cy = q, cz = q, dx = q, dy = q, dz = q;
#pragma unroll 4
    for (int k2 = 0; k2 < np2; k2++)
      adj_pair32x2<GUARD>(ax, ay, az, tile32[3 * k2], tile32[3 * k2 + 1], tile32[3 * k2 + 2], eps2, q, cx, cy, cz,
                          dx, dy, dz);
    qb += (double)q.x + (double)q.y;
    bx += ((double)cx.x + (double)cx.y) - 2.0 * ((double)dx.x + (double)dx.y);
    by += ((double)cy.x + (double)cy.y) - 2.0 * ((double)dy.x + (double)dy.y);
    bz += ((double)cz.x + (double)cz.y) - 2.0 * ((double)dz.x + (double)dz.y);
  }
  if (j < npl) {
    qbar[oj] = kBiotSavart / kPackScale * qb;
    ybar[oj] = kBiotSavart * s.w * bx;
    ybar[N + oj] = kBiotSavart * s.w * by;
    ybar[2 * N + oj] = kBiotSavart * s.w * bz;
  }
}

// Mixed-precision transposed well-separated interactions: source panel s
// (blockIdx.x), one thread per source proxy, target panels' proxies and
// c = Tbar x x staged as pairs.
template <bool GUARD>
__global__ void __launch_bounds__(kT) k_tree_cc_T32(StepGeom fg, const int* __restrict__ tstart,
                                                   const int* __restrict__ ttgt, const double* __restrict__ tbar,
                                                   double* __restrict__ qbar) {
  __shared__ float4 tile[3 * ((kT + 1) / 2)];
  const int s = blockIdx.x, q = fg.q, q2 = (q + 1) >> 1;
  const long pn = (long)fg.panels * q;
  const int k = threadIdx.x;
  const long ok = (long)s * q + (k < q ? k : 0);
  const double* cs = fg.pd_centre + 4 * (long)s;
  const float sx = (float)((fg.px[ok] - cs[0]) * kPackScale), sy = (float)((fg.px[pn + ok] - cs[1]) * kPackScale),
              sz = (float)((fg.px[2 * pn + ok] - cs[2]) * kPackScale);
  const float feps = (float)fg.eps;
  const float2 eps2 = make_float2(feps, feps);
  double acc = 0;
  for (int e = tstart[s]; e < tstart[s + 1]; e++) {
    const int t = ttgt[e];
    const long tb = (long)t * q;
    const double* ct = fg.pd_centre + 4 * (long)t;
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * q2; i += blockDim.x) {
      if (i < q)
        adj_stage(tile, i, fg.px[tb + i], fg.px[pn + tb + i], fg.px[2 * pn + tb + i], tbar[tb + i], tbar[pn + tb + i],
                  tbar[2 * pn + tb + i], ct);
      else
        adj_stage_zero(tile, i);
    }
    __syncthreads();
    const float a0 = sx + (float)((cs[0] - ct[0]) * kPackScale), a1 = sy + (float)((cs[1] - ct[1]) * kPackScale),
                a2 = sz + (float)((cs[2] - ct[2]) * kPackScale);
    const float2 ax = make_float2(a0, a0), ay = make_float2(a1, a1), az = make_float2(a2, a2);
    float2 qq = make_float2(0.f, 0.f), cx = qq, cy = qq, cz = qq, dx = qq, dy = qq, dz = qq;
#pragma unroll 4
    for (int k2 = 0; k2 < q2; k2++)
      adj_pair32x2<GUARD>(ax, ay, az, tile[3 * k2], tile[3 * k2 + 1], tile[3 * k2 + 2], eps2, qq, cx, cy, cz, dx, dy,
                          dz);
    acc += (double)qq.x + (double)qq.y;
  }
  if (k < q) qbar[(long)s * q + k] = kBiotSavart / kPackScale * acc;
}

// 1-D barycentric basis on the leaf's Chebyshev proxies and its derivative,
// without a range check (displaced particles may leave their leaf).
template <int n>
__device__ __forceinline__ void bli_free_deriv(double t, double lo, double hi, const BliTable& tab, double* f,
                                               double* df) {
  const double range = 0.5 * (hi - lo), offset = 0.5 * (hi + lo);
  int hit = -1;
#pragma unroll
  for (int i = 0; i <= n; i++)
    if (hit < 0 && fabs(t - (tab.cosv[i] * range + offset)) < 1e-15) hit = i;
  if (hit >= 0) {
    const double th = tab.cosv[hit] * range + offset;
    double sum = 0;
#pragma unroll
    for (int a = 0; a <= n; a++) {
      f[a] = a == hit ? 1.0 : 0.0;
      df[a] = a == hit ? 0.0 : (tab.w[a] / tab.w[hit]) / (th - (tab.cosv[a] * range + offset));
      sum += df[a];
    }
#pragma unroll
    for (int a = 0; a <= n; a++) df[a] = a == hit ? -sum : df[a];
    return;
  }
  double S = 0, T = 0;
#pragma unroll
  for (int k = 0; k <= n; k++) {
    const double inv = 1.0 / (t - (tab.cosv[k] * range + offset));
    const double r = tab.w[k] * inv;
    f[k] = r;
    df[k] = inv;
    S += r;
    T = fma(r, inv, T);
  }
  const double iS = 1.0 / S, TS = T * iS;
#pragma unroll
  for (int a = 0; a <= n; a++) {
    f[a] *= iS;
    df[a] = f[a] * (TS - df[a]);
  }
}

__device__ __forceinline__ void atan_grad2(double u, int iu, double su, double w, int iw, double sw, double* gr) {
  const double den = 1.0 / (u * u + w * w);
  gr[0] = gr[1] = gr[2] = 0;
  gr[iu] += w * su * den;
  gr[iw] -= u * sw * den;
}

// Anterpolation adjoint: particle j of tree leaf f (blockIdx.x) adds
// sum_k B_k(y_j) Qbar_k to qbar_j and q_j sum_k grad B_k(y_j) Qbar_k to ybar_j,
// B_k = Lx_a(xi(y)) Ly_b(eta(y)) on the leaf's face.
template <int PD>  // proxy degree (the bases stay in registers)
__global__ void __launch_bounds__(kLeafThreads) k_tree_sources_T(TreeGeom tg, StepGeom fg, BliTable tab, const double4* __restrict__ psrc,
                                 const double* __restrict__ qbl, double* __restrict__ qbar,
                                 double* __restrict__ ybar) {
  extern __shared__ double sq[];  // the leaf's adjoint proxy strengths, qx
  const int f = blockIdx.x, npl = tg.npl;
  constexpr int n = PD, n1 = n + 1, qx = n1 * n1;
  const long N = tg.N;
  const int panel = fg.offset + f;
  for (int k = threadIdx.x; k < qx; k += blockDim.x) sq[k] = qbl[(long)panel * qx + k];
  __syncthreads();
  const double* bd = tg.fbounds + 4 * panel;
  const int face = tg.fface[panel];
  for (int jj = threadIdx.x; jj < npl; jj += blockDim.x) {
    const long o = (long)f * npl + jj;
    const double4 s = psrc[o];
    double xi, eta;
    xieta_from_xyz_face(s.x, s.y, s.z, face, xi, eta);
    double fx[n1], dfx[n1], fe[n1], dfe[n1];
    bli_free_deriv<n>(xi, bd[0], bd[1], tab, fx, dfx);
    bli_free_deriv<n>(eta, bd[2], bd[3], tab, fe, dfe);
    double val = 0, dxi = 0, deta = 0;
#pragma unroll
    for (int a = 0; a <= n; a++) {
      double row = 0, drow = 0;
#pragma unroll
      for (int b = 0; b <= n; b++) {
        const double qk = sq[a * n1 + b];
        row = fma(fe[b], qk, row);
        drow = fma(dfe[b], qk, drow);
      }
      val = fma(fx[a], row, val);
      dxi = fma(dfx[a], row, dxi);
      deta = fma(fx[a], drow, deta);
    }
    double gxi[3], geta[3];
    const double X = s.x, Y = s.y, Z = s.z;
    switch (face) {
      case 0: atan_grad2(Y, 1, 1, X, 0, 1, gxi); atan_grad2(Z, 2, 1, X, 0, 1, geta); break;
      case 1: atan_grad2(-X, 0, -1, Y, 1, 1, gxi); atan_grad2(Z, 2, 1, Y, 1, 1, geta); break;
      case 2: atan_grad2(Y, 1, 1, X, 0, 1, gxi); atan_grad2(-Z, 2, -1, X, 0, 1, geta); break;
      case 3: atan_grad2(-X, 0, -1, Y, 1, 1, gxi); atan_grad2(-Z, 2, -1, Y, 1, 1, geta); break;
      case 4: atan_grad2(Y, 1, 1, Z, 2, 1, gxi); atan_grad2(-X, 0, -1, Z, 2, 1, geta); break;
      default: atan_grad2(-Y, 1, -1, Z, 2, 1, gxi); atan_grad2(-X, 0, -1, Z, 2, 1, geta); break;
    }
    qbar[o] += val;
    for (int c = 0; c < 3; c++) ybar[c * N + o] += s.w * (dxi * gxi[c] + deta * geta[c]);
  }
}

// Transposed spectral-FMM interactions: one group of G lanes per source panel
// s (kT / G groups per block; G = q rounded up to a power of two for q <= 32,
// the whole block above), lane k its proxy k, over the target panels whose
// list holds s: Qbar_s,k = K sum g c.d and ybar_s,k = K S_s,k sum [g c -
// g^2 (c.d) d], c = Tbar_t,i x x_t,i, d = y_s,k - x_t,i (y: the stage's
// displaced proxy).  Float64, or mixed: d' = d kPackScale from coordinates
// packed relative to the two panels' centres (their offset rounded once per
// entry), one source against two targets per paired FP32 instruction
// (adj_pair32x2), per-entry float32 sums added into float64.  Writes qbar
// [panels*q]; position adjoints of leaf proxies to ybar_leaf [3][leaves*q],
// of non-leaf proxies to ybar_nl [3][offset*q].
template <int G, bool GUARD, bool MIXED>
__global__ void __launch_bounds__(kT) k_spec_interact_T(StepGeom g, const int* __restrict__ tstart,
                                                       const int* __restrict__ ttgt, const double* __restrict__ tbar,
                                                       const double4* __restrict__ src, double* __restrict__ qbar,
                                                       double* __restrict__ ybar_leaf, double* __restrict__ ybar_nl) {
  constexpr int S = kT / G;
  __shared__ double sd64[6][kT];                  // float64: x, y, z, c of each group's target panel
  __shared__ float4 sd32[S][3 * ((G + 1) / 2)];  // mixed: pairs of packed targets and c
  const int gi = threadIdx.x / G, k = threadIdx.x % G, base = gi * G;
  const int s = blockIdx.x * S + gi, q = g.q, qh = (q + 1) >> 1;
  const long pn = (long)g.panels * q;
  const bool panel = s < g.panels;
  const bool act = panel && k < q;
  const unsigned lanes = G >= 32 ? 0xffffffffu : (((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1)));
  auto sync = [&] {
    if (G > 32) __syncthreads();
    else __syncwarp(lanes);
  };
  const double4 y = src[panel ? (long)s * q + (k < q ? k : 0) : 0];
  const double* cs = g.pd_centre + 4 * (long)(panel ? s : 0);
  const float ysx = (float)((y.x - cs[0]) * kPackScale), ysy = (float)((y.y - cs[1]) * kPackScale),
              ysz = (float)((y.z - cs[2]) * kPackScale);
  const float feps = (float)g.eps;
  const float2 eps2 = make_float2(feps, feps);
  double qb = 0, bx = 0, by = 0, bz = 0;
  const int e0 = panel ? tstart[s] : 0, e1 = panel ? tstart[s + 1] : 0;
  for (int e = e0; e < e1; e++) {
    const long tb = (long)ttgt[e] * q;
    sync();
    if constexpr (MIXED) {
      const double* ct = g.pd_centre + 4 * (long)ttgt[e];
      for (int i = k; i < 2 * qh; i += G) {
        if (i < q)
          adj_stage(sd32[gi], i, g.px[tb + i], g.px[pn + tb + i], g.px[2 * pn + tb + i], tbar[tb + i],
                    tbar[pn + tb + i], tbar[2 * pn + tb + i], ct);
        else
          adj_stage_zero(sd32[gi], i);
      }
      sync();
      if (act) {
        const float a0 = ysx + (float)((cs[0] - ct[0]) * kPackScale), a1 = ysy + (float)((cs[1] - ct[1]) * kPackScale),
                    a2 = ysz + (float)((cs[2] - ct[2]) * kPackScale);
        const float2 ax = make_float2(a0, a0), ay = make_float2(a1, a1), az = make_float2(a2, a2);
        float2 qq = make_float2(0.f, 0.f), cx = qq, cy = qq, cz = qq, dx = qq, dy = qq, dz = qq;
        for (int k2 = 0; k2 < qh; k2++)
          adj_pair32x2<GUARD>(ax, ay, az, sd32[gi][3 * k2], sd32[gi][3 * k2 + 1], sd32[gi][3 * k2 + 2], eps2, qq, cx,
                              cy, cz, dx, dy, dz);
        qb += (double)qq.x + (double)qq.y;
        bx += ((double)cx.x + (double)cx.y) - 2.0 * ((double)dx.x + (double)dx.y);
        by += ((double)cy.x + (double)cy.y) - 2.0 * ((double)dy.x + (double)dy.y);
        bz += ((double)cz.x + (double)cz.y) - 2.0 * ((double)dz.x + (double)dz.y);
      }
    } else {
      for (int i = k; i < q; i += G) {
        const double x = g.px[tb + i], yy = g.px[pn + tb + i], z = g.px[2 * pn + tb + i];
        const double a = tbar[tb + i], b = tbar[pn + tb + i], c = tbar[2 * pn + tb + i];
        sd64[0][base + i] = x;
        sd64[1][base + i] = yy;
        sd64[2][base + i] = z;
        sd64[3][base + i] = b * z - c * yy;
        sd64[4][base + i] = c * x - a * z;
        sd64[5][base + i] = a * yy - b * x;
      }
      sync();
      if (act)
        for (int i = 0; i < q; i++) {
          const double dx = y.x - sd64[0][base + i], dy = y.y - sd64[1][base + i], dz = y.z - sd64[2][base + i];
          const double cx = sd64[3][base + i], cy = sd64[4][base + i], cz = sd64[5][base + i];
          const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
          double gg = recip_nr(fma(0.5, r2, g.eps));
          if (GUARD) gg = r2 > 0.0 ? gg : 0.0;
          const double sdot = fma(cx, dx, fma(cy, dy, cz * dz));
          qb = fma(gg, sdot, qb);
          const double t = gg * gg * sdot;
          bx = fma(gg, cx, fma(-t, dx, bx));
          by = fma(gg, cy, fma(-t, dy, by));
          bz = fma(gg, cz, fma(-t, dz, bz));
        }
    }
  }
  if (!act) return;
  const long o = (long)s * q + k;
  qbar[o] = (MIXED ? kBiotSavart / kPackScale : kBiotSavart) * qb;
  if (s >= g.offset) {
    const long ln = (long)g.leaves * q, l = o - (long)g.offset * q;
    ybar_leaf[l] = kBiotSavart * y.w * bx;
    ybar_leaf[ln + l] = kBiotSavart * y.w * by;
    ybar_leaf[2 * ln + l] = kBiotSavart * y.w * bz;
  } else {
    const long nn = (long)g.offset * q;
    ybar_nl[o] = kBiotSavart * y.w * bx;
    ybar_nl[nn + o] = kBiotSavart * y.w * by;
    ybar_nl[2 * nn + o] = kBiotSavart * y.w * bz;
  }
}

template <int G>
void launch_spec_interact_T_g(const StepGeom& g, bool mixed, const int* tstart, const int* ttgt, const double* tbar,
                              const double4* src, double* qbar, double* ybar_leaf, double* ybar_nl, cudaStream_t st) {
  const unsigned blocks = (unsigned)((g.panels + kT / G - 1) / (kT / G));
  const bool guard = !(g.eps > 0);
  if (mixed) {
    if (guard) SB_LAUNCH((k_spec_interact_T<G, true, true>), blocks, kT, 0, st, g, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl);
    else SB_LAUNCH((k_spec_interact_T<G, false, true>), blocks, kT, 0, st, g, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl);
  } else {
    if (guard) SB_LAUNCH((k_spec_interact_T<G, true, false>), blocks, kT, 0, st, g, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl);
    else SB_LAUNCH((k_spec_interact_T<G, false, false>), blocks, kT, 0, st, g, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl);
  }
}

// Non-leaf proxy positions, reversed: y_i = proj(p_i + h sum_m B_mi v[row_i + m])
// (nonleaf_position); vbar[c][row_i + m] += h B_mi J(p)^T ybar_i with
// J(p)^T ybar = (ybar - yhat (yhat.ybar)) / |p|.  Proxies of one leaf row add
// into the same velocity entries: double atomics.
__global__ void k_nonleaf_positions_T(StepGeom g, double h, const double* __restrict__ vprev,
                                      const double* __restrict__ ybar_nl, double* __restrict__ vbar) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int q = g.q;
  const long np = (long)g.offset * q;
  if (i >= np) return;
  const long pn = (long)g.panels * q, ln = (long)g.leaves * q;
  const long row = (long)g.il_row[i] * q;
  double px = g.px[i], py = g.px[pn + i], pz = g.px[2 * pn + i];
  for (int m = 0; m < q; m++) {
    const double bm = g.il_basis[m * np + i];
    px += (h * vprev[row + m]) * bm;
    py += (h * vprev[ln + row + m]) * bm;
    pz += (h * vprev[2 * ln + row + m]) * bm;
  }
  const double r = sqrt(px * px + py * py + pz * pz), ir = 1.0 / r;
  const double hx = px * ir, hy = py * ir, hz = pz * ir;
  const double gx = ybar_nl[i], gy = ybar_nl[np + i], gz = ybar_nl[2 * np + i];
  const double dd = hx * gx + hy * gy + hz * gz;
  const double ax = h * (gx - hx * dd) * ir, ay = h * (gy - hy * dd) * ir, az = h * (gz - hz * dd) * ir;
  for (int m = 0; m < q; m++) {
    const double bm = g.il_basis[m * np + i];
    atomicAdd(vbar + row + m, ax * bm);
    atomicAdd(vbar + ln + row + m, ay * bm);
    atomicAdd(vbar + 2 * ln + row + m, az * bm);
  }
}

void launch_up3(const StepGeom& g, double* t, cudaStream_t st) {
  for (int lev = g.levels - 2; lev >= 0; lev--)
    SB_LAUNCH(k_tree_up3, dim3(6u << (2 * lev), 3), kT, sizeof(double) * 8 * g.q, st, g, lev, t);
}

void launch_down1(const StepGeom& g, double* qb, cudaStream_t st) {
  for (int lev = 0; lev < g.levels - 1; lev++)
    SB_LAUNCH(k_tree_down1, 6u << (2 * lev), kT, sizeof(double) * 3 * g.q, st, g, lev, qb);
}

template <int NT>
void launch_near_T(const TreeGeom& tg, int leaves, const TreeAdjointLists& tl, const double* x, const double* y,
                   const double* z, const double* vbar, const double4* psrc, double* qbar, double* ybar,
                   cudaStream_t st) {
  const int blocks = leaves * ((tg.npl + 2 * NT - 1) / (2 * NT));
  const unsigned ranks = split_ranks(blocks);
  if (tg.eps > 0)
    launch_cluster(k_tree_near_T<NT, false>, blocks, ranks, NT, 0, st, tg, tl.near_tstart, tl.near_ttgt, x, y, z, vbar,
                   psrc, qbar, ybar);
  else
    launch_cluster(k_tree_near_T<NT, true>, blocks, ranks, NT, 0, st, tg, tl.near_tstart, tl.near_ttgt, x, y, z, vbar,
                   psrc, qbar, ybar);
}

void launch_sources_T(const TreeGeom& tg, const StepGeom& fg, const BliTable& ftab, const double4* psrc,
                      const double* qbl, double* qbar, double* ybar, cudaStream_t st) {
#define SB_ST(N)                                                                                             \
  case N:                                                                                                    \
    SB_LAUNCH(k_tree_sources_T<N>, (unsigned)fg.leaves, kLeafThreads, sizeof(double) * fg.q, st, tg, fg, ftab, \
              psrc, qbl, qbar, ybar);                                                                        \
    break;
  switch (tg.n) {
    SB_ST(1) SB_ST(2) SB_ST(3) SB_ST(4) SB_ST(5) SB_ST(6) SB_ST(7) SB_ST(8) SB_ST(9) SB_ST(10)
  }
#undef SB_ST
}

}  // namespace

void launch_spectral_velocity_adjoint(const StepGeom& g, const int* tstart, const int* ttgt, const double* vbar,
                                      const double4* src, double* tbar, double* qbar, double* ybar_leaf,
                                      double* ybar_nl, bool mixed, cudaStream_t st) {
  const int q = g.q;
  const long pn = (long)g.panels * q, ln = (long)g.leaves * q, off = (long)g.offset * q;
  // the leaf targets' adjoint is vbar itself (leaf proxies = particles); the
  // downward pass transposed accumulates it up the tree
  cudaMemsetAsync(tbar, 0, sizeof(double) * 3 * pn, st);
  for (int c = 0; c < 3; c++)
    cudaMemcpyAsync(tbar + c * pn + off, vbar + c * ln, sizeof(double) * ln, cudaMemcpyDeviceToDevice, st);
  launch_up3(g, tbar, st);
  if (q <= 4) launch_spec_interact_T_g<4>(g, mixed, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl, st);
  else if (q <= 16) launch_spec_interact_T_g<16>(g, mixed, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl, st);
  else if (q <= 32) launch_spec_interact_T_g<32>(g, mixed, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl, st);
  else launch_spec_interact_T_g<kT>(g, mixed, tstart, ttgt, tbar, src, qbar, ybar_leaf, ybar_nl, st);
  // the strengths' upward pass transposed: interpolate their adjoints down
  launch_down1(g, qbar, st);
}

void launch_nonleaf_positions_adjoint(const StepGeom& g, double h, const double* vprev, const double* ybar_nl,
                                      double* vbar, cudaStream_t st) {
  const long np = (long)g.offset * g.q;
  if (np > 0) SB_LAUNCH(k_nonleaf_positions_T, blocks_for(np, 256), 256, 0, st, g, h, vprev, ybar_nl, vbar);
}

void launch_tree_velocity_adjoint(const TreeGeom& tg, const StepGeom& fg, const BliTable& ftab,
                                  const TreeAdjointLists& tl, const double* x, const double* y, const double* z,
                                  const double* vbar, const double4* psrc, double* tbar, double* qbl, double* qbar,
                                  double* ybar, bool mixed, cudaStream_t st, cudaStream_t tree_st, cudaEvent_t fork,
                                  cudaEvent_t join) {
  const int qx = fg.q, Pf = fg.panels;
  const long pn = (long)Pf * qx;
  // the tree's passes need only vbar, the near field only vbar and the
  // particle sources: the tree runs beside it
  if (tree_st != st) {
    cudaEventRecord(fork, st);
    cudaStreamWaitEvent(tree_st, fork, 0);
  }
  // leaf interpolation, transposed; non-leaf rows start at zero
  cudaMemsetAsync(tbar, 0, sizeof(double) * 3 * pn, tree_st);
  SB_LAUNCH(k_tree_to_particles_T, dim3((unsigned)fg.leaves, 3), kLeafThreads,
            sizeof(double) * (tg.npl + tg.side * (tg.n + 1)), tree_st, tg, fg, vbar, tbar);
  launch_up3(fg, tbar, tree_st);
  // well-separated interactions, transposed
  if (mixed) {
    if (fg.eps > 0) SB_LAUNCH(k_tree_cc_T32<false>, (unsigned)Pf, kT, 0, tree_st, fg, tl.cc_tstart, tl.cc_ttgt, tbar, qbl);
    else SB_LAUNCH(k_tree_cc_T32<true>, (unsigned)Pf, kT, 0, tree_st, fg, tl.cc_tstart, tl.cc_ttgt, tbar, qbl);
  } else if (fg.eps > 0) {
    launch_cluster(k_tree_cc_T<false>, Pf, split_ranks(Pf), kT, 0, tree_st, fg, tl.cc_tstart, tl.cc_ttgt, tbar, qbl);
  } else {
    launch_cluster(k_tree_cc_T<true>, Pf, split_ranks(Pf), kT, 0, tree_st, fg, tl.cc_tstart, tl.cc_ttgt, tbar, qbl);
  }
  // upward pass, transposed: interpolate down the tree
  launch_down1(fg, qbl, tree_st);
  if (tree_st != st) cudaEventRecord(join, tree_st);
  // near field, transposed (writes qbar, ybar), then the anterpolation adjoint (adds)
  const int nth = tg.npl <= 256 ? 256 : 512;
  if (mixed) {
    const size_t sm32 = sizeof(float4) * 3 * ((tg.npl + 1) / 2);
    if (tg.eps > 0)
      SB_LAUNCH(k_tree_near_T32<false>, (unsigned)fg.leaves, nth, sm32, st, tg, fg, tl.near_tstart, tl.near_ttgt, x, y,
                z, vbar, psrc, qbar, ybar);
    else
      SB_LAUNCH(k_tree_near_T32<true>, (unsigned)fg.leaves, nth, sm32, st, tg, fg, tl.near_tstart, tl.near_ttgt, x, y,
                z, vbar, psrc, qbar, ybar);
  } else if (tg.npl <= 128) {
    launch_near_T<64>(tg, fg.leaves, tl, x, y, z, vbar, psrc, qbar, ybar, st);
  } else {
    launch_near_T<128>(tg, fg.leaves, tl, x, y, z, vbar, psrc, qbar, ybar, st);
  }
  if (tree_st != st) cudaStreamWaitEvent(st, join, 0);
  launch_sources_T(tg, fg, ftab, psrc, qbl, qbar, ybar, st);
}

}  // namespace sbslpm
