// Mixed-precision proxy interactions over a target panel's list of source
// panels, q <= 25, one source field or two: list64.cuh's organisation with
// float32 pairs on coordinates packed relative to the panels' centres.
//
// A target's float32 sums run over one source panel at a time, two
// interleaved halves (the paired FP32 instructions of sm_100 take two
// sources, an odd last source goes to the first half alone), and are added in
// float32 before the float64 conversion: with few sources per panel the
// conversions would otherwise load the MUFU pipe more than the reciprocals
// do.  One target per lane read two 16-byte shared-memory words per two pairs
// and staged every panel by load, shuffle, store and barrier; several targets
// per lane feed on one read, and panels arrive by cp.async one ahead, their
// entries (panel, centre offset) loaded one panel earlier still.  An FP32
// pair instruction with three different register pairs issues in three
// cycles, with two in two: 3.2e12 pairs/s is what the arithmetic allows.  The
// sources lie in memory as those instructions take them (store_packed_xyz).
// 25 points, levels 6, theta 0.5: 264 us per launch before, 180 us now (2.0e12
// pairs/s).
#pragma once

#include "list64.cuh"

namespace sbslpm {
namespace dev {

template <int Q, int FIELDS>
struct ListShape32 {
  static constexpr int TPT = Q <= 1 ? 1 : Q <= 4 ? 2 : Q <= 9 ? 3 : Q <= 16 ? 2 : FIELDS == 1 ? 5 : 3;
  static constexpr int LPT = (Q + TPT - 1) / TPT;
  static constexpr int S = 32 / LPT;
  static constexpr int STRIDE = packed_stride(Q) | 1;   // float4 per split, buffer and field: odd, for the banks
  static constexpr int PARTS = 3 * FIELDS * Q;          // partial sums per split
  static constexpr int TILE = FIELDS * 2 * S * STRIDE;  // float4 per warp
  static constexpr int WARP = TILE * 2 > S * PARTS ? TILE * 2 : S * PARTS;  // doubles per warp (tile or partial sums)
  static constexpr int NW = 4;
  static_assert(Q <= kPairedQ && NW * (WARP + 1) * sizeof(double) <= 48 * 1024, "pairs in static shared memory");
};

// Calls done(target panel, its index, node, sums) for each node of the target
// panels, sums being sum g d' of each field (d' = d kPackScale).  src, src2:
// packed sources; every thread of the block calls it.
template <int Q, int FIELDS, int WPT, bool ALL_LEAVES, bool GUARD, class Done>
__device__ __forceinline__ void list32_sweep(const StepGeom& g, const float4* __restrict__ src,
                                             const float4* __restrict__ src2, double* __restrict__ shared,
                                             const Done& done) {
  using W = ListShape32<Q, FIELDS>;
  constexpr int TPT = W::TPT, LPT = W::LPT, S = W::S, STEP = S * WPT, STRIDE = W::STRIDE;
  constexpr int PACKED = packed_stride(Q);
  constexpr int WARP = (W::WARP + 1) & ~1;  // 16-byte aligned
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
  const double* ct = g.pd_centre + 4 * (long)t;
  float dtx[TPT], dty[TPT], dtz[TPT];
  double a[FIELDS][3][TPT];
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    const int j = jl + r * LPT;
    const long o = (long)t * Q + (j < Q ? j : 0);
    dtx[r] = (float)((g.px[o] - ct[0]) * kPackScale);
    dty[r] = (float)((g.px[pn + o] - ct[1]) * kPackScale);
    dtz[r] = (float)((g.px[2 * pn + o] - ct[2]) * kPackScale);
#pragma unroll
    for (int f = 0; f < FIELDS; f++) a[f][0][r] = a[f][1][r] = a[f][2][r] = 0;
  }
  const float eps = (float)g.eps;
  const float2 eps2 = make_float2(eps, eps);
  // list entry e: the source panel and its centre's offset from the target's
  auto entry_of = [&](int e) -> int4 {
    if constexpr (ALL_LEAVES) {
      const int sp = g.offset + e;
      const double* cs = g.pd_centre + 4 * (long)sp;
      return make_int4(sp, __float_as_int((float)((cs[0] - ct[0]) * kPackScale)),
                       __float_as_int((float)((cs[1] - ct[1]) * kPackScale)),
                       __float_as_int((float)((cs[2] - ct[2]) * kPackScale)));
    } else {
      return __ldg(g.entry + e);
    }
  };
  float4* mine = reinterpret_cast<float4*>(shared + warp * WARP) + (act ? h : 0) * FIELDS * 2 * STRIDE;
  auto fetch = [&](int buf, int sp) {
    float4* to = mine + buf * FIELDS * STRIDE;
    for (int k = jl; k < PACKED; k += LPT) {
      copy_async16(to + k, src + (long)sp * PACKED + k);
      if constexpr (FIELDS == 2) copy_async16(to + STRIDE + k, src2 + (long)sp * PACKED + k);
    }
  };
  const int4 none = make_int4(0, 0, 0, 0);
  const int first = e0 + wi * S;
  const int iters = first < e1 ? (e1 - first + STEP - 1) / STEP : 0;
  int e = first + h;
  bool on = act && e < e1;
  int4 en = on ? entry_of(e) : none;
  if (on) fetch(0, en.x);
  asm volatile("cp.async.commit_group;" ::: "memory");
  e += STEP;
  bool on_n = act && e < e1;
  int4 en_n = on_n ? entry_of(e) : none;
  for (int it = 0; it < iters; it++) {
    if (on_n) fetch((it + 1) & 1, en_n.x);
    asm volatile("cp.async.commit_group;" ::: "memory");
    e += STEP;
    const bool on_2 = act && e < e1;
    const int4 en_2 = on_2 ? entry_of(e) : none;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    if (on) {
      const float cx = __int_as_float(en.y), cy = __int_as_float(en.z), cz = __int_as_float(en.w);
      float2 b[3][TPT];
#pragma unroll
      for (int r = 0; r < TPT; r++) {
        const float b0 = cx - dtx[r], b1 = cy - dty[r], b2 = cz - dtz[r];
        b[0][r] = make_float2(b0, b0);
        b[1][r] = make_float2(b1, b1);
        b[2][r] = make_float2(b2, b2);
      }
#pragma unroll
      for (int f = 0; f < FIELDS; f++) {
        const float4* st = mine + ((it & 1) * FIELDS + f) * STRIDE;
        float2 fx[TPT], fy[TPT], fz[TPT];
#pragma unroll
        for (int r = 0; r < TPT; r++) fx[r] = fy[r] = fz[r] = make_float2(0.f, 0.f);
        constexpr int kPairs = Q / 2, kUnroll = Q > 16 ? 4 : kPairs > 0 ? kPairs : 1;
#pragma unroll kUnroll
        for (int k = 0; k < kPairs; k++) {
          const float4 u = st[2 * k], v = st[2 * k + 1];
#pragma unroll
          for (int r = 0; r < TPT; r++)
            pair32x2<GUARD>(b[0][r], b[1][r], b[2][r], make_float2(u.x, u.y), make_float2(u.z, u.w),
                            make_float2(v.x, v.y), make_float2(v.z, v.w), eps2, fx[r], fy[r], fz[r]);
        }
        if constexpr (Q & 1) {
          const float4 u = st[Q - 1], v = st[Q];
#pragma unroll
          for (int r = 0; r < TPT; r++)
            pair32<GUARD>(b[0][r].x, b[1][r].x, b[2][r].x, make_float4(u.x, u.z, v.x, v.z), eps, fx[r].x, fy[r].x,
                          fz[r].x);
        }
#pragma unroll
        for (int r = 0; r < TPT; r++) {
          a[f][0][r] += (double)(fx[r].x + fx[r].y);
          a[f][1][r] += (double)(fy[r].x + fy[r].y);
          a[f][2][r] += (double)(fz[r].x + fz[r].y);
        }
      }
    }
    __syncwarp();
    on = on_n;
    en = en_n;
    on_n = on_2;
    en_n = en_2;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // partial sums [warp][split][component][node] of the target panel
  if (WPT > 1) __syncthreads();
  else __syncwarp();
  double* red = shared + warp * WARP;
  if (act) {
#pragma unroll
    for (int r = 0; r < TPT; r++) {
      const int j = jl + r * LPT;
      if (j < Q) {
#pragma unroll
        for (int f = 0; f < FIELDS; f++)
#pragma unroll
          for (int c = 0; c < 3; c++) red[h * W::PARTS + (3 * f + c) * Q + j] = a[f][c][r];
      }
    }
  }
  if (WPT > 1) __syncthreads();
  else __syncwarp();
  if (!live || wi > 0) return;
  for (int j = lane; j < Q; j += 32) {
    double sums[3 * FIELDS];
#pragma unroll
    for (int c = 0; c < 3 * FIELDS; c++) sums[c] = 0;
    for (int w = 0; w < WPT; w++)
      for (int k = 0; k < S; k++)
#pragma unroll
        for (int c = 0; c < 3 * FIELDS; c++) sums[c] += shared[(warp + w) * WARP + k * W::PARTS + c * Q + j];
    done(t, tix, j, sums);
  }
}

}  // namespace dev
}  // namespace sbslpm
