// Device helpers shared by the kernel files: the reciprocal used by every
// pair kernel, the Biot-Savart pair in float64 / float32 / paired float32,
// the device error word, and the launch macro that counts launches.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "bve_kernels.cuh"

namespace sbslpm {
namespace dev {

// The device error word (alloc_error_word): the bits, and at err + 2 the
// address of a page-locked host word that any error sets, so that the host
// reads the bits back only after one.
__device__ __forceinline__ void flag(unsigned* err, unsigned bits) {
  if (bits) {
    atomicOr(err, bits);
    *static_cast<volatile unsigned*>(*reinterpret_cast<unsigned**>(err + 2)) = 1u;
  }
}

// 1/d from the hardware approximation r and one third-order step
// (Householder's iteration for 1/d): with e = 1 - d r, r (1 + e + e^2) leaves
// an error of e^3 -- at most 2^-60 from the approximation's 2^-20 or better --
// before the last rounding, in three FP64 operations instead of the four of two
// Newton steps.  d of either sign, 1/d normal.
__device__ __forceinline__ double recip_nr(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// 1/d with a residual step on recip_nr: what is left of the error before the
// last rounding is its square (below 2^-105), so the result is off by that
// rounding alone, 2^-53 (1 + 2^-50) relative.  d of either sign, 1/d normal.
__device__ __forceinline__ double recip_full(double d) {
  const double r = recip_nr(d);
  return fma(r, fma(-d, r, 1.0), r);
}

__device__ __forceinline__ float recip_f32(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}

// One Biot-Savart pair in float64.  With d = y - x and |x| = |y| = 1,
// 1 - x.y = |d|^2 / 2, and x cross y = x cross d, so the accumulated
// a = sum (g / 2) d gives u = -2/(4 pi) x cross a (kBiotSavartTwice): the
// denominator is taken as |d|^2 + 2 eps, one chain of fused multiply-adds
// with eps2 = twice_eps(eps), 13 FP64 operations in all.  Coincident points
// add nothing: because d = 0 where g is finite, which an eps > 0 of ordinary
// size and a finite strength give; otherwise (GUARD: eps = 0, eps so small
// that g overflows, any other eps) because g is zeroed where |d|^2 is not
// positive, the eps added to it afterwards.
__host__ __device__ __forceinline__ double twice_eps(double eps) { return eps < 8e307 ? 2.0 * eps : eps; }

template <bool GUARD>
__device__ __forceinline__ double pair_weight64(double dx, double dy, double dz, double sw, double eps2) {
  if (!GUARD) return sw * recip_nr(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
  const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
  const double g = sw * recip_nr(r2 + eps2);
  return r2 > 0.0 ? g : 0.0;
}

template <bool GUARD>
__device__ __forceinline__ void pair64(double tx, double ty, double tz, double sx, double sy, double sz, double sw,
                                       double eps2, double& ax, double& ay, double& az) {
  const double dx = sx - tx, dy = sy - ty, dz = sz - tz;
  const double g = pair_weight64<GUARD>(dx, dy, dz, sw, eps2);
  ax = fma(g, dx, ax);
  ay = fma(g, dy, ay);
  az = fma(g, dz, az);
}

template <bool GUARD>
__device__ __forceinline__ void pair64(double tx, double ty, double tz, const double4 s, double eps2, double& ax,
                                       double& ay, double& az) {
  pair64<GUARD>(tx, ty, tz, s.x, s.y, s.z, s.w, eps2, ax, ay, az);
}

// One source against T targets, step by step for all of them: an FP64
// instruction with three different registers is issued in three cycles, one
// with two (or with an operand held over from the instruction before) in
// two, so the order that keeps s.x or g in place for the next instruction
// measured 1.22e12 pairs/s against 1.18e12 target by target (two targets).
template <bool GUARD, int T>
__device__ __forceinline__ void pairs64(const double (&tx)[T], const double (&ty)[T], const double (&tz)[T],
                                        double sx, double sy, double sz, double sw, double eps2, double (&ax)[T],
                                        double (&ay)[T], double (&az)[T]) {
  double dx[T], dy[T], dz[T], g[T];
#pragma unroll
  for (int r = 0; r < T; r++) dz[r] = sz - tz[r];
#pragma unroll
  for (int r = 0; r < T; r++) dy[r] = sy - ty[r];
#pragma unroll
  for (int r = 0; r < T; r++) dx[r] = sx - tx[r];
#pragma unroll
  for (int r = 0; r < T; r++) g[r] = pair_weight64<GUARD>(dx[r], dy[r], dz[r], sw, eps2);
#pragma unroll
  for (int r = 0; r < T; r++) {
    ax[r] = fma(g[r], dx[r], ax[r]);
    ay[r] = fma(g[r], dy[r], ay[r]);
    az[r] = fma(g[r], dz[r], az[r]);
  }
}

// The same pair in float32 on panel-relative coordinates scaled by 1/sqrt(2)
// (kPackScale): d' = base + s.xyz with base = (c_S - c_T)/sqrt(2) - delta_t,
// and |d'|^2 + eps = |d|^2/2 + eps in one FMA chain.
template <bool GUARD>
__device__ __forceinline__ void pair32(float bx, float by, float bz, const float4 s, float eps, float& ax, float& ay,
                                       float& az) {
  float dx = bx + s.x, dy = by + s.y, dz = bz + s.z;
  float den = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps)));
  float g = s.w * recip_f32(den);
  if (GUARD) g = den > 0.0f ? g : 0.0f;
  ax = fmaf(g, dx, ax);
  ay = fmaf(g, dy, ay);
  az = fmaf(g, dz, az);
}

// Two pairs at once with the paired FP32 instructions of sm_100 (FADD2 /
// FFMA2 / FMUL2): one target (b broadcast in both halves) against two
// sources given as register pairs (x0,x1), (y0,y1), (z0,z1), (w0,w1).
template <bool GUARD>
__device__ __forceinline__ void pair32x2(const float2 bx, const float2 by, const float2 bz, const float2 sx,
                                         const float2 sy, const float2 sz, const float2 sw, const float2 eps2,
                                         float2& ax, float2& ay, float2& az) {
  const float2 dx = __fadd2_rn(bx, sx), dy = __fadd2_rn(by, sy), dz = __fadd2_rn(bz, sz);
  const float2 den = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, eps2)));
  float2 g = __fmul2_rn(sw, make_float2(recip_f32(den.x), recip_f32(den.y)));
  if (GUARD) {
    g.x = den.x > 0.0f ? g.x : 0.0f;
    g.y = den.y > 0.0f ? g.y : 0.0f;
  }
  ax = __ffma2_rn(g, dx, ax);
  ay = __ffma2_rn(g, dy, ay);
  az = __ffma2_rn(g, dz, az);
}

// Two pairs in the expanded form: with b = base (target side, as above) and
// s the source's packed offset, |b + s|^2 + eps = (|s|^2 + eps) + |b|^2 +
// 2 b.s, and sum g (b + s) = sum r (w s) + b sum r w with r = 1/den.  The
// source side is staged as (x0,x1,y0,y1) (z0,z1,q0,q1) (w0x0,w1x1,w0y0,w1y1)
// (w0z0,w1z1,w0,w1) with q = |s|^2 + eps, the target side as m = 2b and
// bb = |b|^2: 4 paired operations for the denominator and 4 for the sums, 8
// per two pairs against 10 in pair32x2.  The expansion rounds the
// denominator to u (|b| + |s|)^2 instead of u |b + s| (|b| + |s|), so it is
// used only where eps dominates that (a coincident pair still adds nothing:
// its s = -b cancels in the final b sum r w + sum r w s up to rounding of
// w s / eps).  fx, fy, fz accumulate sum r w s; fw accumulates sum r w.
__device__ __forceinline__ void pair32x2_expanded(const float2 mx, const float2 my, const float2 mz, const float2 bb,
                                                  const float4 A, const float4 B, const float4 C, const float4 D,
                                                  float2& fx, float2& fy, float2& fz, float2& fw) {
  float2 den = __fadd2_rn(make_float2(B.z, B.w), bb);
  den = __ffma2_rn(mz, make_float2(B.x, B.y), den);
  den = __ffma2_rn(my, make_float2(A.z, A.w), den);
  den = __ffma2_rn(mx, make_float2(A.x, A.y), den);
  const float2 r = make_float2(recip_f32(den.x), recip_f32(den.y));
  fx = __ffma2_rn(r, make_float2(C.x, C.y), fx);
  fy = __ffma2_rn(r, make_float2(C.z, C.w), fy);
  fz = __ffma2_rn(r, make_float2(D.x, D.y), fz);
  fw = __ffma2_rn(r, make_float2(D.z, D.w), fw);
}

// Stages the sources 2k, 2k+1 of a packed float4 array (x, y, z, w) in the
// expanded form's four float4 (a missing partner past n has zero strength).
__device__ __forceinline__ void stage_expanded(const float4* __restrict__ src, int k2, int n, float eps,
                                               float4* __restrict__ out) {
  const float4 s0 = src[2 * k2];
  const float4 s1 = (2 * k2 + 1 < n) ? src[2 * k2 + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float q0 = fmaf(s0.x, s0.x, fmaf(s0.y, s0.y, fmaf(s0.z, s0.z, eps)));
  const float q1 = fmaf(s1.x, s1.x, fmaf(s1.y, s1.y, fmaf(s1.z, s1.z, eps)));
  out[0] = make_float4(s0.x, s1.x, s0.y, s1.y);
  out[1] = make_float4(s0.z, s1.z, q0, q1);
  out[2] = make_float4(s0.w * s0.x, s1.w * s1.x, s0.w * s0.y, s1.w * s1.y);
  out[3] = make_float4(s0.w * s0.z, s1.w * s1.z, s0.w, s1.w);
}

// Where the packed float32 source j (of q) of a panel lies.  Panels of up to
// kPairedQ sources (list32.cuh) hold them two by two, transposed, as the
// paired FP32 instructions take them: (x0,x1,y0,y1) (z0,z1,w0,w1), an odd
// count closing on a source that stays zero; larger panels hold one float4
// per source.
__device__ __forceinline__ void store_packed_xyz(float4* srcf, int q, long panel, int j, float x, float y, float z) {
  if (q <= kPairedQ) {
    float* p = reinterpret_cast<float*>(srcf + panel * packed_stride(q)) + 8 * (j >> 1) + (j & 1);
    p[0] = x;
    p[2] = y;
    p[4] = z;
  } else {
    float4& f = srcf[panel * q + j];
    f.x = x;
    f.y = y;
    f.z = z;
  }
}

__device__ __forceinline__ void store_packed_w(float4* srcf, int q, long panel, int j, float w) {
  if (q <= kPairedQ) (reinterpret_cast<float*>(srcf + panel * packed_stride(q)) + 8 * (j >> 1) + (j & 1))[6] = w;
  else srcf[panel * q + j].w = w;
}

__device__ __forceinline__ void store_packed(float4* srcf, int q, long panel, int j, const double* c, double x,
                                             double y, double z, double w) {
  store_packed_xyz(srcf, q, panel, j, (float)((x - c[0]) * kPackScale), (float)((y - c[1]) * kPackScale),
                   (float)((z - c[2]) * kPackScale));
  store_packed_w(srcf, q, panel, j, (float)w);
}

// Nodes per direction of a panel of q = n^2 nodes: the length to which float64
// loops over a panel of more than 25 sources are unrolled (whole rounds at any
// q).  Three or four sources, with remainders, hid too little latency where a
// tree has few panels: lists of a step at levels 3, us, 49 points 190 / 147, 64
// 239 / 184, 100 461 / 382; two fields of 36 points at levels 4 1,006 / 706.
constexpr int row_of(int q) {
  int n = 1;
  while (n * n < q) n++;
  return n;
}

// First panel id of the k-th level below the subtree root (level, root_rel).
__device__ __forceinline__ int subtree_first(int level, int root_rel, int k) {
  return level_start(level + k) + (root_rel << (2 * k));
}

// Displaced, re-projected position of non-leaf proxy i: its containing leaf's
// BLI interpolation of dt_s * vprev, unrolled where Q (= q) is given.
template <int Q>
__device__ __forceinline__ void nonleaf_position(const StepGeom& g, long i, int stage, double dt_s,
                                                 const double* __restrict__ vprev, double& px, double& py,
                                                 double& pz) {
  const int q = Q > 0 ? Q : g.q;
  const long pn = (long)g.panels * q, ln = (long)g.leaves * q;
  px = g.px[i];
  py = g.px[pn + i];
  pz = g.px[2 * pn + i];
  if (stage > 0) {
    const long np = (long)g.offset * q;
    const long row = (long)g.il_row[i] * q;
    double ax = 0, ay = 0, az = 0;
#pragma unroll
    for (int m = 0; m < (Q > 0 ? Q : q); m++) {
      const double bm = g.il_basis[m * np + i];
      ax += (dt_s * vprev[row + m]) * bm;
      ay += (dt_s * vprev[ln + row + m]) * bm;
      az += (dt_s * vprev[2 * ln + row + m]) * bm;
    }
    px += ax;
    py += ay;
    pz += az;
  }
  project_to_sphere(px, py, pz);
}

// Point location + tensor-product BLI basis at a point (point_locate_panel
// and interp_vals_bli, src/interp_funcs_impl.hpp:11-142), and gathers of a
// [leaf][q] field with it.
template <int D>
struct Basis {
  double fx[D + 1], fe[D + 1];
  long row;  // (leaf - offset) * q
};

template <int D>
__device__ __forceinline__ void locate_basis(const StepGeom& g, const BliTable& tab, double x, double y, double z,
                                             Basis<D>& b, unsigned& err) {
  double xi, eta;
  Bounds bd;
  int leaf = locate_leaf(x, y, z, g.levels, xi, eta, bd, err);
  bli_1d(xi, kPi / 4.0 * bd.min_xi, kPi / 4.0 * bd.max_xi, D, tab.cosv, tab.w, b.fx, err);
  bli_1d(eta, kPi / 4.0 * bd.min_eta, kPi / 4.0 * bd.max_eta, D, tab.cosv, tab.w, b.fe, err);
  b.row = (long)(leaf - g.offset) * g.q;
}

// The same basis with fewer float64 divisions, for the departure / remap
// kernel (one thread per particle, four locations each): the projection and
// the face coordinates multiply by one reciprocal, and the barycentric basis
// uses the common-denominator form f_i = w_i P_i / sum_k w_k P_k with
// P_i = prod_{j != i} (t - c_j) -- the second barycentric form multiplied
// through by prod_j (t - c_j): one division per direction instead of 2(D+1).
// Nodes within 1e-15 are hit exactly as in bli_1d; results differ from
// locate_basis by rounding only.
template <int D>
__device__ __forceinline__ void bli_1d_common(double t, double lo, double hi, const BliTable& tab, double* f,
                                              unsigned& err) {
  const double range = 0.5 * (hi - lo), offset = 0.5 * (hi + lo);
  if (t < lo - 1e-15 || t > hi + 1e-15) err |= kErrOutOfPanel;
  if (D == 0) {
    f[0] = 1;
    return;
  }
  double dl[D + 1];
  int hit = -1;
#pragma unroll
  for (int i = 0; i <= D; i++) {
    dl[i] = t - (tab.cosv[i] * range + offset);
    if (hit < 0 && fabs(dl[i]) < 1e-15) hit = i;
  }
  if (hit >= 0) {
#pragma unroll
    for (int i = 0; i <= D; i++) f[i] = (i == hit) ? 1.0 : 0.0;
    return;
  }
  double pre[D + 1], suf = 1.0, den = 0.0;
  pre[0] = 1.0;
#pragma unroll
  for (int i = 1; i <= D; i++) pre[i] = pre[i - 1] * dl[i - 1];
#pragma unroll
  for (int i = D; i >= 0; i--) {
    f[i] = tab.w[i] * (pre[i] * suf);
    den += f[i];
    suf *= dl[i];
  }
  const double inv = recip_full(den);
#pragma unroll
  for (int i = 0; i <= D; i++) f[i] *= inv;
}

__device__ __forceinline__ void project_to_sphere_rcp(double& x, double& y, double& z) {
  // written out: the single and the batched step's kernels must contract alike
  const double inv = rsqrt(fma(z, z, fma(y, y, x * x)));
  x *= inv;
  y *= inv;
  z *= inv;
}

// locate_basis for the departure / remap kernel: one reciprocal for the face's
// axis, the leaf from the cells of xi and eta (leaf_by_cells) instead of a
// descent through the levels, the barycentric basis with one reciprocal per
// direction.
template <int D>
__device__ __forceinline__ void locate_basis_rcp(const StepGeom& g, const BliTable& tab, double x, double y, double z,
                                                 Basis<D>& b, unsigned& err) {
  const int face = face_from_xyz(x, y, z);
  // xieta_from_xyz_face: face 0 (y, z)/x, 1 (-x, z)/y, 2 (y, -z)/x, 3 (-x, -z)/y, 4 (y, -x)/z, 5 (-y, -x)/z
  const double den = face == 0 || face == 2 ? x : face == 1 || face == 3 ? y : z;
  const double num_xi = face == 1 || face == 3 ? -x : face == 5 ? -y : y;
  const double num_eta = face >= 4 ? -x : face >= 2 ? -z : z;
  const double r = recip_full(den);
  const double xi = atan(num_xi * r), eta = atan(num_eta * r);
  if (!(xi == xi) || !(eta == eta)) err |= kErrNonFinite;  // NaN coordinates
  Bounds bd;
  const unsigned leaf = leaf_by_cells(xi, eta, g.levels, bd);
  bli_1d_common<D>(xi, kPi / 4.0 * bd.min_xi, kPi / 4.0 * bd.max_xi, tab, b.fx, err);
  bli_1d_common<D>(eta, kPi / 4.0 * bd.min_eta, kPi / 4.0 * bd.max_eta, tab, b.fe, err);
  b.row = (((long)face << (2 * (g.levels - 1))) + leaf) * g.q;
}

// sum_m field[row + m] * fx[i] fe[j] with m = i (D+1) + j, in m order.
template <int D>
__device__ __forceinline__ double gather(const Basis<D>& b, const double* __restrict__ f, long stride = 1,
                                         long base = 0) {
  double acc = 0;
  int m = 0;
#pragma unroll
  for (int i = 0; i <= D; i++)
#pragma unroll
    for (int j = 0; j <= D; j++, m++) acc += f[(b.row + m) * stride + base] * (b.fx[i] * b.fe[j]);
  return acc;
}

// The same for q even and rows on 16-byte boundaries, two values per load: a
// particle's 160 loads (degree 3) otherwise fill the load/store unit.
template <int D>
__device__ __forceinline__ double gather_vec(const Basis<D>& b, const double* __restrict__ f) {
  constexpr int n1 = D + 1, q = n1 * n1;
  const double2* p = reinterpret_cast<const double2*>(f + b.row);
  double acc = 0;
#pragma unroll
  for (int m = 0; m < q; m += 2) {
    const double2 v = p[m / 2];
    acc += v.x * (b.fx[m / n1] * b.fe[m % n1]);
    acc += v.y * (b.fx[(m + 1) / n1] * b.fe[(m + 1) % n1]);
  }
  return acc;
}

template <int D>
__device__ __forceinline__ void gather3(const Basis<D>& b, const double* __restrict__ v, long n, double& a,
                                        double& c, double& e) {
  a = 0;
  c = 0;
  e = 0;
  int m = 0;
#pragma unroll
  for (int i = 0; i <= D; i++)
#pragma unroll
    for (int j = 0; j <= D; j++, m++) {
      double bm = b.fx[i] * b.fe[j];
      a += v[b.row + m] * bm;
      c += v[n + b.row + m] * bm;
      e += v[2 * n + b.row + m] * bm;
    }
}

// Non-leaf points per block of an upward pass's first launch: few enough that
// the points reach every SM (all threads of the block where there are many).
inline int nonleaf_chunk(long points, unsigned threads) {
  const long per = (points / 148 + 31) / 32 * 32;
  return (int)(per < 128 ? (threads < 128 ? threads : 128) : per < threads ? per : threads);
}

inline unsigned blocks_for(long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace dev

// Kernel launches made by the library (a process-wide diagnostic count).
std::atomic<long>& launch_counter();

// Raises kernels' dynamic shared-memory limit on the current device, once per
// device (the attribute is per device: a process that drives several GPUs
// must set it on each).  done: the caller's static record of the devices set
// (device ordinals >= 64 are set on every call).
template <typename... K>
inline void raise_smem_once(std::atomic<unsigned long long>& done, int bytes, K... kernels) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return;
  (cudaFuncSetAttribute(kernels, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), ...);
  if (bit) done.fetch_or(bit, std::memory_order_acq_rel);
}

// A launch whose blocks (x, 0 .. ranks-1) form one cluster for every x.
template <typename... P, typename... A>
inline void launch_cluster(void (*kernel)(P...), unsigned blocks, unsigned ranks, unsigned threads, size_t smem,
                           cudaStream_t st, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1;
  at.val.clusterDim.y = ranks;
  at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks, ranks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  launch_counter()++;
}

}  // namespace sbslpm

#define SB_LAUNCH(kernel, grid, block, shmem, st, ...)      \
  do {                                                     \
    kernel<<<grid, block, shmem, st>>>(__VA_ARGS__);       \
    ::sbslpm::launch_counter()++;                          \
  } while (0)
