// Treecode leaves: the free barycentric basis of displaced particles, the
// moments (anterpolation) S[a][b] = sum_k lx[k][a] ly[k][b] w_k of a leaf's
// particles on its proxies, and the shared-memory row length both use.
#pragma once

#include "bve_kernels.cuh"
#include "geometry.cuh"

namespace sbslpm::dev {

// Barycentric Lagrange basis of degree n on Chebyshev extrema of [lo, hi]
// without the reference's range check: displaced sources may sit slightly
// outside their leaf, where the interpolant extrapolates smoothly.  The
// second barycentric form multiplied through by prod_j (t - c_j):
// f_i = w_i P_i / sum_k w_k P_k with P_i = prod_{j != i} (t - c_j), one
// division instead of n + 2 (nodes within 1e-15 are hit exactly).  N1 = n + 1,
// or 0 for any n: the unrolled products of the general form run to the
// largest degree.  The roundings are written out so that every form gives
// the same values.
template <int N1>
__device__ __forceinline__ void bli_1d_free(double t, double lo, double hi, int n, const double* cosv,
                                            const double* w, double* f) {
  constexpr int M = N1 ? N1 : kMaxDegree + 1;
  if (n == 0) {
    f[0] = 1;
    return;
  }
  const double range = 0.5 * (hi - lo), offset = 0.5 * (hi + lo);
  double dl[M];
  int hit = -1;
#pragma unroll
  for (int i = 0; i < M; i++) {
    dl[i] = N1 || i <= n ? t - fma(cosv[i], range, offset) : 1.0;
    if ((N1 || i <= n) && hit < 0 && fabs(dl[i]) < 1e-15) hit = i;
  }
  if (hit >= 0) {
    for (int i = 0; i <= n; i++) f[i] = (i == hit) ? 1.0 : 0.0;
    return;
  }
  double pre[M];
  pre[0] = 1.0;
#pragma unroll
  for (int i = 1; i < M; i++) pre[i] = pre[i - 1] * dl[i - 1];
  double suf = 1.0, den = 0.0, v[M];
#pragma unroll
  for (int i = M - 1; i >= 0; i--) {
    v[i] = N1 || i <= n ? __dmul_rn(w[i], __dmul_rn(pre[i], suf)) : 0.0;
    den = __dadd_rn(den, v[i]);
    suf *= dl[i];
  }
  const double inv = 1.0 / den;
#pragma unroll
  for (int i = 0; i < M; i++)
    if (N1 || i <= n) f[i] = v[i] * inv;
}

constexpr int kMomentWarps = 8;

// Doubles per particle of a basis in shared memory: odd, so that the threads
// that write a row each meet different banks.
__host__ __device__ constexpr int leaf_stride(int n1) { return n1 | 1; }

// Shared memory of a leaf's sources: two bases, `rows` more doubles per
// particle (at most 512 particles), the warps' partial moments.
constexpr long kLeafSmem = 128 * 1024;
inline size_t leaf_smem(int npl, int n1, int rows) {
  return sizeof(double) * ((size_t)npl * (2 * leaf_stride(n1) + rows) + kMomentWarps * n1 * n1);
}

// part[warp][a][b] = sum over the warp's particles of lx[k][a] ly[k][b] w_k,
// for a block of kMomentWarps warps and rows of ls doubles.  Bound by the
// shared-memory reads: a thread that owned one (a, b) paid three reads and
// two operations per particle and moment.  Here nine threads share a
// particle, each with a T x T tile of the moments in registers (T =
// ceil(n1 / 3)), so that 2 T + 1 reads feed T^2 FMAs; three particles run
// side by side in a warp and are added by shuffles.  393,216 particles in
// leaves of 256 with 81 proxies: the whole source kernel 34.5 us before, 23.1
// now (the positions, bases and stores are the rest); the two fields of 98,304
// particles 23.0 -> 11.9.
template <int T>
__device__ __forceinline__ void leaf_moments_t(const double* lx, const double* ly, int ls, const double* w, int npl,
                                               int n1, double* part) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / 9, tile = lane - 9 * g, a0 = tile / 3 * T, b0 = tile % 3 * T;
  double acc[T][T];
  int ia[T], ib[T];
#pragma unroll
  for (int i = 0; i < T; i++) {
    ia[i] = min(a0 + i, n1 - 1);
    ib[i] = min(b0 + i, n1 - 1);
#pragma unroll
    for (int j = 0; j < T; j++) acc[i][j] = 0;
  }
  if (g < 3) {
    for (int k = 3 * warp + g; k < npl; k += 3 * kMomentWarps) {
      const double wk = w[k];
      double av[T], bv[T];
#pragma unroll
      for (int i = 0; i < T; i++) {
        av[i] = lx[k * ls + ia[i]];
        bv[i] = ly[k * ls + ib[i]] * wk;
      }
#pragma unroll
      for (int i = 0; i < T; i++)
#pragma unroll
        for (int j = 0; j < T; j++) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < T; i++)
#pragma unroll
    for (int j = 0; j < T; j++) {
      const double s1 = __shfl_down_sync(0xffffffffu, acc[i][j], 9), s2 = __shfl_down_sync(0xffffffffu, acc[i][j], 18);
      if (g == 0 && a0 + i < n1 && b0 + j < n1) part[(warp * n1 + a0 + i) * n1 + b0 + j] = (acc[i][j] + s1) + s2;
    }
}

template <int N1>
__device__ __forceinline__ void leaf_moments(const double* lx, const double* ly, int ls, const double* w, int npl,
                                             int n1, double* part) {
  if constexpr (N1 > 0) {
    leaf_moments_t<(N1 + 2) / 3>(lx, ly, ls, w, npl, N1, part);
  } else {  // n1 <= 5 (SB_LEAF_N1)
    if (n1 <= 3) leaf_moments_t<1>(lx, ly, ls, w, npl, n1, part);
    else leaf_moments_t<2>(lx, ly, ls, w, npl, n1, part);
  }
}

// Moment m of the leaf: the warps' parts added in order (after a barrier).
__device__ __forceinline__ double leaf_moment(const double* part, int qx, int m) {
  double acc = part[m];
#pragma unroll
  for (int p = 1; p < kMomentWarps; p++) acc += part[p * qx + m];
  return acc;
}

// Moments of values at the grid's own particles, T[a][b] = sum_k lx[k][a]
// ly[k][b] v_k, one direction at a time over the leaf's tensor grid (side^2 n1
// + side n1^2 operations instead of side^2 n1^2).  v[row][column] and the
// half-contracted half[row][a] in shared memory, after a barrier; emit(m,
// T[m]) for every moment.
template <typename E>
__device__ __forceinline__ void grid_moments(const TreeGeom& tg, const double* v, double* half, E emit) {
  const int n1 = tg.n + 1, side = tg.side;
  for (int o = threadIdx.x; o < side * n1; o += blockDim.x) {
    const int row = o / n1, a = o - row * n1;
    double acc = 0;
    for (int i = 0; i < side; i++) acc = fma(__ldg(tg.lx + i * n1 + a), v[row * side + i], acc);
    half[o] = acc;
  }
  __syncthreads();
  for (int m = threadIdx.x; m < n1 * n1; m += blockDim.x) {
    const int a = m / n1, b = m - a * n1;
    double acc = 0;
    for (int i = 0; i < side; i++) acc = fma(__ldg(tg.ly + i * n1 + b), half[i * n1 + a], acc);
    emit(m, acc);
  }
}

__device__ __forceinline__ int grid_slot(const TreeGeom& tg, int k) {
  const int p = __ldg(tg.place + k);
  return (p >> 16) * tg.side + (p & 0xffff);
}

}  // namespace sbslpm::dev

// Proxy degrees 5..10 (the well-separated kernels' range) run with the degree
// as a constant, which bounds the basis' products; below, one general form.
// Every form is held to 64 registers, four blocks per SM (98,304 particles in
// 384 blocks: one wave, 21.6 -> 13.9 us).  Source kernels at two and at four
// blocks, us: degree 10, 393,216 particles in leaves of 256 35.4 / 27.4, 13,824
// in leaves of 9 24.2 / 15.5; degree 4, 393,216 particles 31 / 22.  In a batch
// each block finds its member's.
#define SB_LEAF_N1(n1, CALL)     \
  switch (n1) {                  \
    case 6: CALL(6); break;      \
    case 7: CALL(7); break;      \
    case 8: CALL(8); break;      \
    case 9: CALL(9); break;      \
    case 10: CALL(10); break;    \
    case 11: CALL(11); break;    \
    default: CALL(0); break;     \
  }
