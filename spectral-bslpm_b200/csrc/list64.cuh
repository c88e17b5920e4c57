// Float64 proxy interactions over a target panel's list of source panels
// (CSR list, or, for the shallow-water direct velocity, every leaf of a group),
// for one source field (BVE) or two (shallow water), q <= 25.
//
// The FP64 pipe bounds the pairs (13 operations each; about 1.2e12 pairs/s
// with the operands that a pair reads from registers).  What kept the kernels
// from it were one target per lane (every pair paid for two 16-byte
// shared-memory reads), a load -> store -> barrier chain per source panel, and
// on small trees too few warps.  Hence:
//  * a warp holds one target panel as S source splits of LPT lanes with TPT
//    targets each, so a shared-memory read feeds TPT pairs; TPT is chosen per
//    q so that few target slots stay empty (q = 9: 3 x 3 lanes x 10 splits,
//    16: 2 x 8 x 4, 25: 5 x 5 x 6);
//  * each split's source panel arrives by cp.async in a double-buffered tile
//    (the next panel in flight while the current one is evaluated, its index
//    loaded one panel earlier still), no block-wide barrier in the loop; a
//    split's tile is padded by 16 bytes so that the splits' broadcast reads
//    fall on different banks;
//  * WPT warps of a block share a target panel (list_warps).
// The S * WPT partial sums are added in a fixed order.
//
// Above 25 points the shape serves the Poisson kernel alone (poisson.cu): TPT by
// the same rule, few empty target slots with at most a whole warp per panel.  Its
// lists of one solve at levels 4, theta 0.7, a thread per node / by these
// shapes, us: 36 points 430 / 87, 49 580 / 146, 64 749 / 228, 81 1,005 / 413, 100
// 1,397 / 740, 121 1,690 / 806.
#pragma once

#include "device_common.cuh"

namespace sbslpm {
namespace dev {

template <int Q, int FIELDS>
struct ListShape {
  static constexpr int TPT = Q <= 1    ? 1
                             : Q <= 4   ? 2
                             : Q <= 9   ? 3
                             : Q <= 16  ? 2
                             : Q <= 49  ? 5
                             : Q <= 64  ? 4
                             : Q <= 81  ? 3
                             : Q <= 100 ? 7
                                        : 4;
  static constexpr int LPT = (Q + TPT - 1) / TPT;
  static constexpr int S = 32 / LPT;
  static constexpr int STRIDE = 2 * Q + 1;              // double2 per split, buffer and field
  static constexpr int WARP = FIELDS * 2 * S * STRIDE;  // double2 per warp
  static constexpr int NW = WARP * 4 * 16 <= 48 * 1024 ? 4 : 2;  // warps per block
  static_assert(S * 3 * FIELDS * Q * sizeof(double) <= WARP * sizeof(double2), "a warp's partial sums fit its tile");
  static_assert(NW * WARP * sizeof(double2) <= 48 * 1024, "static shared memory");
};

// Warps per target panel: a whole block while the tree has fewer panels than
// 16 warps per SM would take, else two (lists are then short enough for the
// splits of two warps).  BVE step, degree 3, theta 0.7, us per step at 1 / 2 / 4
// warps: levels 3 198 / 180 / 172, levels 5 269 / 251 / 247, levels 7 1625 /
// 1605 / 1649.  Where one warp alone splits the list ten ways or more, a list
// of some 40 entries leaves the splits of more warps without any: list kernels
// of a step, us at 1 / 2 / 4 warps, theta 0.7, q = 9 at levels 4 41 / 30 / 27
// (float64), 21 / 19 / 19 (mixed), levels 5 61 / 59 / 62, 35 / 40 / 50, levels 6
// 168 / 168 / 197, 100 / 119 / 166; q = 4 levels 3 16 / 14 / 12, levels 5 26 /
// 24 / 34, 20 / 24 / 37; q = 1 levels 3 10 / 10 / 12, levels 5 15 / 18 / 28.
template <int Q, int FIELDS, bool MIXED>
inline int list_warps(int target_panels) {
  using W = ListShape<Q, FIELDS>;
  constexpr int NW = MIXED ? 4 : W::NW;
  const bool few = target_panels <= 148 * 4, some = target_panels <= 148 * 16;
  if (W::S >= 32) return 1;
  if (W::S >= 16) return few ? 2 : 1;
  if (W::S >= 10) return few ? NW : some && !MIXED ? 2 : 1;
  return some ? NW : 2;
}

__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
               :
               : "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

__device__ __forceinline__ void copy_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
               :
               : "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Evaluates target panel blockIdx.x * (NW / WPT) + (this warp's group) and
// calls done(target panel, its index, node, sums) for each of its nodes, sums
// being sum (g / 2) d of each field.  Every thread of the block calls it.
template <int Q, int FIELDS, int WPT, bool ALL_LEAVES, bool GUARD, class Done>
__device__ __forceinline__ void list64_sweep(const StepGeom& g, const double4* __restrict__ src,
                                             const double4* __restrict__ src2, double2* __restrict__ tiles,
                                             const Done& done) {
  using W = ListShape<Q, FIELDS>;
  constexpr int TPT = W::TPT, LPT = W::LPT, S = W::S, STEP = S * WPT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wi = warp % WPT;
  const int tp_first = ALL_LEAVES ? g.offset : 0;
  const int tp_count = ALL_LEAVES ? g.leaves : g.panels;
  const int tix = blockIdx.x * (W::NW / WPT) + warp / WPT;
  const bool live = tix < tp_count;
  const int t = tp_first + (live ? tix : 0);
  const long pn = (long)g.panels * Q;
  int e0 = 0, e1 = 0;
  if (live) {
    if (ALL_LEAVES) {
      const int per = (g.leaves + gridDim.y - 1) / gridDim.y;
      e0 = blockIdx.y * per;
      e1 = min(g.leaves, e0 + per);
    } else {
      e0 = g.tgt_start[t];
      e1 = g.tgt_start[t + 1];
    }
  }
  const int h = lane / LPT, jl = lane - h * LPT;
  const bool act = h < S;
  double tx[TPT], ty[TPT], tz[TPT], ax[TPT], ay[TPT], az[TPT], bx[TPT], by[TPT], bz[TPT];
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    const int j = jl + r * LPT;
    const long o = (long)t * Q + (j < Q ? j : 0);
    tx[r] = g.px[o];
    ty[r] = g.px[pn + o];
    tz[r] = g.px[2 * pn + o];
    ax[r] = ay[r] = az[r] = bx[r] = by[r] = bz[r] = 0;
  }
  const double eps2 = twice_eps(g.eps);
  auto source_of = [&](int e) { return ALL_LEAVES ? g.offset + e : __ldg(g.src_panel + e); };
  double2* mine = tiles + warp * W::WARP + (act ? h : 0) * FIELDS * 2 * W::STRIDE;
  auto fetch = [&](int buf, int sp) {
    double2* to = mine + buf * FIELDS * W::STRIDE;
    const double2* from = reinterpret_cast<const double2*>(src + (long)sp * Q);
    for (int c = jl; c < 2 * Q; c += LPT) copy_async16(to + c, from + c);
    if constexpr (FIELDS == 2) {
      const double2* from2 = reinterpret_cast<const double2*>(src2 + (long)sp * Q);
      for (int c = jl; c < 2 * Q; c += LPT) copy_async16(to + W::STRIDE + c, from2 + c);
    }
  };
  const int first = e0 + wi * S;
  const int iters = first < e1 ? (e1 - first + STEP - 1) / STEP : 0;
  int e = first + h;
  bool on = act && e < e1;
  if (on) fetch(0, source_of(e));
  asm volatile("cp.async.commit_group;" ::: "memory");
  e += STEP;
  bool on_n = act && e < e1;
  int sp_n = on_n ? source_of(e) : 0;
  for (int it = 0; it < iters; it++) {
    if (on_n) fetch((it + 1) & 1, sp_n);
    asm volatile("cp.async.commit_group;" ::: "memory");
    e += STEP;
    const bool on_2 = act && e < e1;
    sp_n = on_2 ? source_of(e) : 0;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    if (on) {
      const double2* st = mine + (it & 1) * FIELDS * W::STRIDE;
      constexpr int kUnroll = Q > 16 ? 5 : Q;  // fully unrolled, 25 x 5 pairs leave the instruction cache: 1.36x slower
#pragma unroll kUnroll
      for (int k = 0; k < Q; k++) {
        const double2 a = st[2 * k], b = st[2 * k + 1];
        pairs64<GUARD>(tx, ty, tz, a.x, a.y, b.x, b.y, eps2, ax, ay, az);
        if constexpr (FIELDS == 2) {
          const double2 c = st[W::STRIDE + 2 * k], d = st[W::STRIDE + 2 * k + 1];
          pairs64<GUARD>(tx, ty, tz, c.x, c.y, d.x, d.y, eps2, bx, by, bz);
        }
      }
    }
    __syncwarp();
    on = on_n;
    on_n = on_2;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // partial sums [warp][split][component][node] of the target panel, from its first warp's tile on
  constexpr int PART = 3 * FIELDS * Q;
  double* red = reinterpret_cast<double*>(tiles + (warp - wi) * W::WARP);
  if (WPT > 1) __syncthreads();
  else __syncwarp();
  if (act) {
#pragma unroll
    for (int r = 0; r < TPT; r++) {
      const int j = jl + r * LPT;
      if (j < Q) {
        double* p = red + (wi * S + h) * PART + j;
        p[0] = ax[r];
        p[Q] = ay[r];
        p[2 * Q] = az[r];
        if constexpr (FIELDS == 2) {
          p[3 * Q] = bx[r];
          p[4 * Q] = by[r];
          p[5 * Q] = bz[r];
        }
      }
    }
  }
  if (WPT > 1) __syncthreads();
  else __syncwarp();
  if (!live || wi > 0) return;
  for (int j = lane; j < Q; j += 32) {
    double sums[3 * FIELDS];
#pragma unroll
    for (int c = 0; c < 3 * FIELDS; c++) sums[c] = red[c * Q + j];
    for (int k = 1; k < S * WPT; k++)
#pragma unroll
      for (int c = 0; c < 3 * FIELDS; c++) sums[c] += red[k * PART + c * Q + j];
    done(t, tix, j, sums);
  }
}

}  // namespace dev
}  // namespace sbslpm
