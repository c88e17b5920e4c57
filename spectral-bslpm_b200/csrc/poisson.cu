// Poisson (inverse Laplacian) FMM of executables/poisson_eq_fmm.cpp on the
// device: the reference's upward pass, poisson_fmm_interactions
// (src/fmm_interactions/inverse_poisson.cpp:9-34) and downward_pass
// (src/fmm_funcs.cpp:357-372), on a spectral-FMM context (proxy degree = the
// particle degree).  The kernel -1/(4 pi) log(1 - x.y) is the reference's,
// evaluated as it writes it (1 - x.y, pairs with x.y >= 1 - 1e-15 skipped), so
// the solve is u with -Laplacian(u) = f for mean-zero f.
#include <cuda_runtime.h>

#include "context_internal.hpp"
#include "device_common.cuh"
#include "list64.cuh"
#include "log_table.cuh"

using namespace sbslpm;

namespace {

constexpr double kInvLapConst = -0.07957747154594767;  // -1/(4 pi), as the reference writes it

// poisson_panel_interaction (src/fmm_interactions/inverse_poisson_impl.hpp:22-52)
// owner-computes, on the list organisation of list64.cuh: S source splits of
// LPT lanes with TPT targets each per warp, WPT warps per target panel, the
// splits' source panels brought in by cp.async one ahead, partial sums added
// in a fixed order.  One block of 128 threads per panel, a thread per node,
// left 112 of them idle at 16 nodes: 98,304 points, theta 0.7, 922 us; this
// organisation 310 us with CUDA's log, 207 us with table_log (about 25 FP64
// operations a pair): the FP64 pipe is 54% busy, and what holds the warps is
// the table's reads from shared memory (45% of their stalled cycles).
template <int Q, int WPT>
__global__ void __launch_bounds__(32 * dev::ListShape<Q, 1>::NW)
    k_poisson_interact(StepGeom g, const double* __restrict__ table, const double* __restrict__ src,
                       double* __restrict__ tgt) {
  using W = dev::ListShape<Q, 1>;
  constexpr int TPT = W::TPT, LPT = W::LPT, S = W::S, STEP = S * WPT;
  __shared__ __align__(16) double2 tiles[W::NW * W::WARP];
  __shared__ __align__(16) double log_cv[2 * kLogN];
  __shared__ double log_lo[kLogN];
  for (int k = threadIdx.x; k < 2 * kLogN; k += blockDim.x) log_cv[k] = table[k];
  for (int k = threadIdx.x; k < kLogN; k += blockDim.x) log_lo[k] = table[2 * kLogN + k];
  const double2* cv = reinterpret_cast<const double2*>(log_cv);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wi = warp % WPT;
  const int tix = blockIdx.x * (W::NW / WPT) + warp / WPT;
  const bool live = tix < g.panels;
  const int t = live ? tix : 0;
  const long pn = (long)g.panels * Q;
  const int e0 = live ? g.tgt_start[t] : 0, e1 = live ? g.tgt_start[t + 1] : 0;
  const int h = lane / LPT, jl = lane - h * LPT;
  const bool act = h < S;
  double tx[TPT], ty[TPT], tz[TPT], acc[TPT];
#pragma unroll
  for (int r = 0; r < TPT; r++) {
    const int j = jl + r * LPT;
    const long o = (long)t * Q + (j < Q ? j : 0);
    tx[r] = g.px[o];
    ty[r] = g.px[pn + o];
    tz[r] = g.px[2 * pn + o];
    acc[r] = 0;
  }
  double2* mine = tiles + warp * W::WARP + (act ? h : 0) * 2 * W::STRIDE;
  auto fetch = [&](int buf, int sp) {
    double* to = reinterpret_cast<double*>(mine + buf * W::STRIDE);
    const long sb = (long)sp * Q;
    for (int k = jl; k < Q; k += LPT) {
#pragma unroll
      for (int c = 0; c < 4; c++) dev::copy_async8(to + 4 * k + c, c < 3 ? g.px + c * pn + sb + k : src + sb + k);
    }
  };
  const int first = e0 + wi * S;
  const int iters = first < e1 ? (e1 - first + STEP - 1) / STEP : 0;
  int e = first + h;
  bool on = act && e < e1;
  if (on) fetch(0, __ldg(g.src_panel + e));
  asm volatile("cp.async.commit_group;" ::: "memory");
  e += STEP;
  bool on_n = act && e < e1;
  int sp_n = on_n ? __ldg(g.src_panel + e) : 0;
  for (int it = 0; it < iters; it++) {
    if (on_n) fetch((it + 1) & 1, sp_n);
    asm volatile("cp.async.commit_group;" ::: "memory");
    e += STEP;
    const bool on_2 = act && e < e1;
    sp_n = on_2 ? __ldg(g.src_panel + e) : 0;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    if (on) {
      const double2* st = mine + (it & 1) * W::STRIDE;
#pragma unroll 2
      for (int k = 0; k < Q; k++) {
        const double2 a = st[2 * k], b = st[2 * k + 1];
#pragma unroll
        for (int r = 0; r < TPT; r++) {
          const double dp = tx[r] * a.x + ty[r] * a.y + tz[r] * b.x;
          const double v = fma(table_log(1 - dp, cv, log_lo), b.y, acc[r]);
          acc[r] = dp < 1.0 - 1e-15 ? v : acc[r];
        }
      }
    }
    __syncwarp();
    on = on_n;
    on_n = on_2;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  double* red = reinterpret_cast<double*>(tiles + (warp - wi) * W::WARP);  // [warp][split][node]
  if (WPT > 1) __syncthreads();
  else __syncwarp();
  if (act) {
#pragma unroll
    for (int r = 0; r < TPT; r++)
      if (jl + r * LPT < Q) red[(wi * S + h) * Q + jl + r * LPT] = acc[r];
  }
  if (WPT > 1) __syncthreads();
  else __syncwarp();
  if (!live || wi > 0) return;
  for (int j = lane; j < Q; j += 32) {
    double a = red[j];
    for (int k = 1; k < S * WPT; k++) a += red[k * Q + j];
    tgt[(long)t * Q + j] += kInvLapConst * a;
  }
}

template <int Q>
void launch_poisson_q(const StepGeom& g, const double* table, const double* src, double* tgt, cudaStream_t st) {
  constexpr int NW = dev::ListShape<Q, 1>::NW, threads = 32 * NW;
  const int wpt = dev::list_warps<Q, 1, false>(g.panels);
  if (wpt == NW) SB_LAUNCH((k_poisson_interact<Q, NW>), g.panels, threads, 0, st, g, table, src, tgt);
  else if (wpt == 2) SB_LAUNCH((k_poisson_interact<Q, 2>), dev::blocks_for(g.panels, NW / 2), threads, 0, st, g, table, src, tgt);
  else SB_LAUNCH((k_poisson_interact<Q, 1>), dev::blocks_for(g.panels, NW), threads, 0, st, g, table, src, tgt);
}

void launch_poisson(const StepGeom& g, const double* table, const double* src, double* tgt, cudaStream_t st) {
  switch (g.q) {
    case 1: launch_poisson_q<1>(g, table, src, tgt, st); break;
    case 4: launch_poisson_q<4>(g, table, src, tgt, st); break;
    case 9: launch_poisson_q<9>(g, table, src, tgt, st); break;
    case 16: launch_poisson_q<16>(g, table, src, tgt, st); break;
    case 25: launch_poisson_q<25>(g, table, src, tgt, st); break;
    case 36: launch_poisson_q<36>(g, table, src, tgt, st); break;
    case 49: launch_poisson_q<49>(g, table, src, tgt, st); break;
    case 64: launch_poisson_q<64>(g, table, src, tgt, st); break;
    case 81: launch_poisson_q<81>(g, table, src, tgt, st); break;
    case 100: launch_poisson_q<100>(g, table, src, tgt, st); break;
    default: launch_poisson_q<121>(g, table, src, tgt, st); break;
  }
}

sbslpm_status need_spectral_fmm(const sbslpm_ctx* c) {
  if (c->tree || c->cfg.velocity != SBSLPM_VEL_FMM)
    return set_last_error("the reference's spectral FMM passes need proxy_degree 0 and FMM velocity"), SBSLPM_ERR_CONFIG;
  if (c->q > 128) return set_last_error("interp_degree above 10"), SBSLPM_ERR_CONFIG;
  return SBSLPM_OK;
}

bool bad(const void* p) { return p == nullptr; }

// downward_pass of one field through the three-field device pass: the
// field in component 0 of the context's proxy-target buffer, the other two
// components zero (their results are not used).
void downward_one(sbslpm_ctx* c, cudaStream_t st) {
  const size_t pn = (size_t)c->P * c->q;
  cudaMemsetAsync(c->tgt + pn, 0, sizeof(double) * 2 * pn, st);
  launch_downward_fused(c->geom, c->tgt, nullptr, st);
}

}  // namespace

sbslpm_status sbslpm::poisson_setup(sbslpm_ctx* c) { return upload(&c->log_table, log_table()); }

extern "C" {

sbslpm_status sbslpm_poisson_fmm_interactions(sbslpm_ctx* c, const double* source, double* target) {
  if (!c || bad(source) || bad(target)) return SBSLPM_ERR_ARG;
  SB_TRY(need_spectral_fmm(c));
  cudaStream_t st = c->stream();
  launch_poisson(c->geom, c->log_table, source, target, st);
  return finish(c);
}

sbslpm_status sbslpm_downward_pass(sbslpm_ctx* c, double* proxy_target, double* soln) {
  if (!c || bad(proxy_target) || bad(soln)) return SBSLPM_ERR_ARG;
  SB_TRY(need_spectral_fmm(c));
  cudaStream_t st = c->stream();
  const size_t pn = (size_t)c->P * c->q, ln = (size_t)c->A * c->q, off = (size_t)c->off * c->q;
  SB_CUDA(cudaMemcpyAsync(c->tgt, proxy_target, sizeof(double) * pn, cudaMemcpyDeviceToDevice, st));
  downward_one(c, st);
  SB_CUDA(cudaMemcpyAsync(proxy_target, c->tgt, sizeof(double) * pn, cudaMemcpyDeviceToDevice, st));
  SB_CUDA(cudaMemcpyAsync(soln, c->tgt + off, sizeof(double) * ln, cudaMemcpyDeviceToDevice, st));
  return finish(c);
}

sbslpm_status sbslpm_poisson_fmm(sbslpm_ctx* c, const double* area, const double* pots, double* soln) {
  if (!c || bad(area) || bad(pots) || bad(soln)) return SBSLPM_ERR_ARG;
  SB_TRY(need_spectral_fmm(c));
  cudaStream_t st = c->stream();
  const size_t pn = (size_t)c->P * c->q, ln = (size_t)c->A * c->q, off = (size_t)c->off * c->q;
  // upward pass: proxy source weights into component 1 of the proxy-target buffer
  SB_CUDA(cudaMemsetAsync(c->src, 0, sizeof(double4) * pn, st));
  launch_upward_fused(c->geom, 1, 0, 0.0, nullptr, nullptr, nullptr, nullptr, pots, area, c->src, false, st);
  launch_copy_strength(c->geom, c->src, c->tgt + pn, st);
  SB_CUDA(cudaMemsetAsync(c->tgt, 0, sizeof(double) * pn, st));
  launch_poisson(c->geom, c->log_table, c->tgt + pn, c->tgt, st);
  downward_one(c, st);
  SB_CUDA(cudaMemcpyAsync(soln, c->tgt + off, sizeof(double) * ln, cudaMemcpyDeviceToDevice, st));
  return finish(c);
}

}  // extern "C"
