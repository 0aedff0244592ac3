// hg_launch.cuh -- definitions of the per-order launch templates declared in hg_ctx.h.
// Included only by the instantiation units hg_inst_*.cu.
#pragma once
#include "hg_ctx.h"

#include <algorithm>
#include <atomic>

// Resident CTAs per SM of a persistent kernel with `smem` bytes of dynamic shared memory, after allowing it
// that much; looked up once per kernel and device.
template <typename K>
static int resident_ctas(const hg_ctx* c, std::atomic<int>* known, K kernel, int threads, size_t smem) {
  std::atomic<int>* slot = c->device < HG_KNOWN_DEVICES ? &known[c->device] : nullptr;
  int n = slot ? slot->load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  HG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  max_carveout(kernel);
  HG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem));
  if (n < 1) throw std::runtime_error("stage kernel does not fit on this device");
  if (slot) slot->store(n, std::memory_order_relaxed);
  return n;
}

template <int P, typename real>
static StageOps<P, real> stage_ops(const hg_ctx* c) {
  StageOps<P, real> o;
  const double* m = c->h_mats.data();
  for (int k = 0; k < P * P; ++k) o.hatD[k] = real(m[k]);
  m += P * P;
  for (int k = 0; k < P; ++k) {
    o.lb0[k] = real(m[k]);
    o.lb1[k] = real(m[P + k]);
    o.lbw0[k] = real(m[2 * P + k]);
    o.lbw1[k] = real(m[3 * P + k]);
  }
  return o;
}

template <int P, typename real, int V, bool AFFINE, bool LGL>
static void launch_stage_PAL(hg_ctx* c, const StageArgs<real>& a) {
  using Tl = StageTiles<P, V, real, AFFINE, LGL>;
  static std::atomic<int> known[HG_KNOWN_DEVICES];
  const int groups = (a.n_el + Tl::EPB - 1) / Tl::EPB;
  const int most = c->n_sm * std::min(32, resident_ctas(c, known, stage_kernel<P, V, real, AFFINE, LGL>, Tl::T, sizeof(Tl)));
  // every CTA takes the same number of groups but the last ones: no more CTAs than that needs
  const int rounds = (groups + most - 1) / most, grid = (groups + rounds - 1) / rounds;
  if (a.resid) c->n_resid = grid;
  const StageOps<P, real> op = stage_ops<P, real>(c);
  timed(c, HG_KERNEL_STAGE, [&] { stage_kernel<P, V, real, AFFINE, LGL><<<grid, Tl::T, sizeof(Tl), c->stream>>>(a, op); });
  ++c->launches;
}

template <int P, typename real, int V>
void launch_stage_PV(hg_ctx* c, const StageArgs<real>& a) {
  const bool lgl = c->node_type == HG_NODES_LGL;
  if (c->affine) {
    if (lgl) launch_stage_PAL<P, real, V, true, true>(c, a); else launch_stage_PAL<P, real, V, true, false>(c, a);
  } else {
    if (lgl) launch_stage_PAL<P, real, V, false, true>(c, a); else launch_stage_PAL<P, real, V, false, false>(c, a);
  }
}

template <int P, typename real>
void launch_trace_P(hg_ctx* c) {
  constexpr int EPB = epb_for(P);
  const int grid = (c->n_el + EPB - 1) / EPB;
  timed(c, HG_KERNEL_TRACE, [&] {
    trace_kernel<P, EPB, real><<<grid, block_for(P), 0, c->stream>>>(c->n_el, c->d_Q, c->d_mats,
                                                                     static_cast<real*>(c->d_T[c->cur]), c->ns);
  });
  ++c->launches;
}

template <int P, typename real, int V, bool AFFINE, bool IP, bool AV>
static void launch_ns_PAI(hg_ctx* c, const NSArgs<real>& a) {
  constexpr int EPB = epb_ns_of(P, V);
  constexpr int BLK = block_of(P, EPB);
  const int grid = (a.n_el + EPB - 1) / EPB;
  static bool attr = false;
  if (!attr) {
    max_carveout(ns_gradient_kernel<P, EPB, real, AFFINE, IP, AV>);
    max_carveout(ns_stage_kernel<P, EPB, real, AFFINE, IP, AV>);
    attr = true;
  }
  if (a.run_gradient) {
    timed(c, HG_KERNEL_GRADIENT,
          [&] { ns_gradient_kernel<P, EPB, real, AFFINE, IP, AV><<<grid, BLK, 0, c->stream>>>(a); });
    ++c->launches;
  }
  if (a.run_stage) {
    if (a.resid) c->n_resid = grid;
    timed(c, HG_KERNEL_STAGE,
          [&] { ns_stage_kernel<P, EPB, real, AFFINE, IP, AV><<<grid, BLK, 0, c->stream>>>(a); });
    ++c->launches;
  }
}

template <int P, typename real, int V>
void launch_ns_PV(hg_ctx* c, const NSArgs<real>& a) {
  // artificial dissipation is a template switch so that the plain kernels keep their register budget
  if (c->av) {
    if (c->affine) {
      if (c->ip) launch_ns_PAI<P, real, V, true, true, true>(c, a); else launch_ns_PAI<P, real, V, true, false, true>(c, a);
    } else {
      if (c->ip) launch_ns_PAI<P, real, V, false, true, true>(c, a); else launch_ns_PAI<P, real, V, false, false, true>(c, a);
    }
  } else {
    if (c->affine) {
      if (c->ip) launch_ns_PAI<P, real, V, true, true, false>(c, a); else launch_ns_PAI<P, real, V, true, false, false>(c, a);
    } else {
      if (c->ip) launch_ns_PAI<P, real, V, false, true, false>(c, a); else launch_ns_PAI<P, real, V, false, false, false>(c, a);
    }
  }
}

// Sensor indicators of the resident state, per element: features [n_el][16] (optional) and
// {modal G, learned G, out-of-distribution flag, G used} [n_el][4] (optional).  The learned G is
// evaluated whenever weights are set.
template <int P, int EPB, typename real>
__global__ void __launch_bounds__(block_ns(P)) sensor_eval_kernel(int n_el, const double* Q, const double* mats,
                                                                  SensorArgs sa, PhysConst pc, float* feat,
                                                                  double* out) {
  constexpr int NP = P * P;
  __shared__ real sQ[4][EPB][NP];
  __shared__ real sV[NP];
  const int flat = threadIdx.x, le = flat / NP, tid = flat - le * NP;
  const int e = blockIdx.x * EPB + le;
  const bool active = le < EPB && e < n_el;
  for (int k = flat; k < NP; k += blockDim.x) sV[k] = real(mats[2 * NP + 7 * P + k]);
  if (active) {
    const double* q = Q + (size_t(e) * NP + tid) * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) sQ[k][le][tid] = real(q[k]);
  }
  __syncthreads();
  Phys<real> ph;
  ph.load(pc);
  SensorArgs s2 = sa;
  if (sa.mlp) s2.kind = SENSOR_LEARNED;
  const int n_active = n_el - int(blockIdx.x) * EPB < EPB ? n_el - int(blockIdx.x) * EPB : EPB;
  SensorOut so = element_sensor<P, EPB, real>(s2, ph, sQ, n_active, sV, le, tid, active,
                                             (active && feat) ? feat + size_t(e) * MLP_IN : nullptr);
  if (active && tid == 0 && out) {
    const double g = sa.kind == SENSOR_LEARNED ? so.g : (sa.kind == SENSOR_MODAL ? so.g_modal : -1.0);
    out[size_t(e) * 4 + 0] = so.g_modal;
    out[size_t(e) * 4 + 1] = sa.mlp ? so.g_learned : -1.0;
    out[size_t(e) * 4 + 2] = so.ood;
    out[size_t(e) * 4 + 3] = g;
  }
}

template <int P, typename real>
void launch_sensor_eval_P(hg_ctx* c, float* feat, double* out) {
  constexpr int EPB = epb_ns(P);
  const int grid = (c->n_el + EPB - 1) / EPB;
  sensor_eval_kernel<P, EPB, real><<<grid, block_ns(P), 0, c->stream>>>(c->n_el, c->d_Q, c->d_mats, sensor_args(c),
                                                                         c->pc, feat, out);
  ++c->launches;
}
