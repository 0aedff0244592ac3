// hg_launch.cuh -- definitions of the per-order launch templates declared in hg_ctx.h.
// Included only by the instantiation units hg_inst_*.cu.
#pragma once
#include "hg_ctx.h"

#include <algorithm>
#include <atomic>

// Resident CTAs per SM of a persistent kernel with `smem` bytes of dynamic shared memory; looked up once per kernel,
// size and device.  `most` is the largest size that any launch of the kernel uses: the attribute holds for all of
// them, so that it must not be lowered by a launch that needs less.
template <typename K>
static int resident_ctas(const hg_ctx* c, std::atomic<int>* known, K kernel, int threads, size_t smem, size_t most) {
  std::atomic<int>* slot = c->device < HG_KNOWN_DEVICES ? &known[c->device] : nullptr;
  int n = slot ? slot->load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  HG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most)));
  max_carveout(kernel);
  HG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem));
  if (n < 1) throw std::runtime_error("stage kernel does not fit on this device");
  if (slot) slot->store(n, std::memory_order_relaxed);
  return n;
}

// CTAs of a persistent launch over `groups` groups of elements, at most `most` resident.  Every CTA takes the same number
// of groups but the last ones, and there are no more CTAs than that needs.  With few groups to a CTA (`few` or less) that
// leaves up to half of the residency empty, and an SM a CTA more or less than its neighbour: there all resident CTAs run,
// some of them for a group more (an RK3 step of 3,750 elements, order 3, interior penalty in double: 41 -> 36 us, 2,400
// elements of order 4 with BR1 56 -> 51 us).  With many the even split is the faster one (cylinder 64 x 128 N = 5 in
// double 780 us against 876, shock 512 x 64 1455 against 1555), for Euler from four on: the members of an ensemble run
// beside one another and fill what each leaves (128 boxes 2.63 against 2.71 ms).
static inline int persistent_grid(int groups, int most, int few) {
  const int rounds = (groups + most - 1) / most;
  return rounds <= few ? std::min(groups, most) : (groups + rounds - 1) / rounds;
}

// Launch that may overlap the end of the kernel before it on the stream (grid_wait, hg_stage.cuh).  Not under
// per-kernel timing, whose events stand between the kernels.
template <typename... KA, typename... A>
static void launch_dependent(hg_ctx* c, void (*kernel)(KA...), int grid, int threads, size_t smem, const A&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  // (the default streams keep plain launches: their ordering against other streams is their own)
  cfg.numAttrs = c->prof || reinterpret_cast<uintptr_t>(c->stream) <= uintptr_t(2) ? 0 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) {
    cudaGetLastError();   // reported here: not left behind for the next call
    throw std::runtime_error(std::string("stage kernel launch: ") + cudaGetErrorString(e));
  }
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
  const int most = c->n_sm * std::min(32, resident_ctas(c, known, stage_kernel<P, V, real, AFFINE, LGL>, Tl::T, sizeof(Tl), sizeof(Tl)));
  const int grid = persistent_grid(groups, most, 3);
  const StageOps<P, real> op = stage_ops<P, real>(c);
  timed(c, HG_KERNEL_STAGE, [&] { launch_dependent(c, stage_kernel<P, V, real, AFFINE, LGL>, grid, Tl::T, sizeof(Tl), a, op); });
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
                                                                     static_cast<real*>(c->d_T[c->cur]),
                                                                     !c->ns && c->node_type == HG_NODES_LGL);
  });
  ++c->launches;
}

template <int P, typename real>
static NSOps<P, real> ns_ops(const hg_ctx* c) {
  NSOps<P, real> o;
  const double* m = c->h_mats.data();   // hatD lb0 lb1 lbw0 lbw1 D dlbw0 dlbw1 w Vinv
  const auto put = [&](real* d, int n) {
    for (int k = 0; k < n; ++k) d[k] = real(m[k]);
    m += n;
  };
  const double *lb = m + P * P, *D = m + P * P + 4 * P;
  for (int l = 0; l < P; ++l) {
    double d0 = 0.0, d1 = 0.0;
    for (int i = 0; i < P; ++i) {
      d0 += lb[i] * D[i * P + l];
      d1 += lb[P + i] * D[i * P + l];
    }
    o.dl0[l] = real(d0);
    o.dl1[l] = real(d1);
  }
  put(o.hatD, P * P);
  put(o.lb0, P); put(o.lb1, P); put(o.lbw0, P); put(o.lbw1, P);
  put(o.D, P * P);
  put(o.dlbw0, P); put(o.dlbw1, P);
  m += P;
  put(o.Vinv, P * P);
  return o;
}

// Persistent launch of a Navier-Stokes kernel with tiles Tl.
template <typename Tl, typename K, typename A, typename O>
static void launch_groups(hg_ctx* c, std::atomic<int>* known, K kernel, int kind, bool weights, const A& a, const O& op) {
  static_assert(sizeof(Tl) + MLP_BYTES <= 227 * 1024, "shared memory of a CTA");
  const size_t smem = sizeof(Tl) + (weights ? MLP_BYTES : 0);
  const int groups = (a.n_el + Tl::EPB - 1) / Tl::EPB;
  const int most = c->n_sm * std::min(32, resident_ctas(c, known, kernel, Tl::T, smem, sizeof(Tl) + MLP_BYTES));
  const int grid = persistent_grid(groups, most, 4);
  timed(c, kind, [&] { launch_dependent(c, kernel, grid, Tl::T, smem, a, op); });
  ++c->launches;
}

template <int P, typename real, int V, bool AFFINE, bool IP, bool AV>
static void launch_ns_PAI(hg_ctx* c, const NSArgs<real>& a) {
  const NSOps<P, real> op = ns_ops<P, real>(c);
  const bool learned = AV && a.sensor.kind == SENSOR_LEARNED;
  if (a.run_gradient) {
    using Tl = NSTiles<P, V, real, AFFINE, IP, AV, true, true>;
    static std::atomic<int> known[2][HG_KNOWN_DEVICES];
    launch_groups<Tl>(c, known[learned], ns_gradient_kernel<P, V, real, AFFINE, IP, AV>, HG_KERNEL_GRADIENT, learned, a, op);
  }
  if (AV && a.run_jumps) {
    EdgeWeights<P, real> ew;
    const double* w = c->h_mats.data() + 2 * P * P + 6 * P;
    for (int k = 0; k < P; ++k) ew.w[k] = real(w[k]);
    const int grid = (a.n_el + jumps_epb(P) - 1) / jumps_epb(P);
    timed(c, HG_KERNEL_GRADIENT, [&] { launch_dependent(c, jumps_kernel<P, real, AFFINE>, grid, 128, 0, a, ew); });
    ++c->launches;
  }
  if (a.run_stage) {
    const bool w = learned && a.fuse && a.update && a.last;
    if (!AV || a.viscous) {
      using Tl = NSTiles<P, V, real, AFFINE, IP, AV, true, false>;
      static std::atomic<int> known[2][HG_KNOWN_DEVICES];
      launch_groups<Tl>(c, known[w], ns_stage_kernel<P, V, real, AFFINE, IP, AV, true>, HG_KERNEL_STAGE, w, a, op);
    } else {
      using Tl = NSTiles<P, V, real, AFFINE, IP, AV, !AV, false>;
      static std::atomic<int> known[2][HG_KNOWN_DEVICES];
      launch_groups<Tl>(c, known[w], ns_stage_kernel<P, V, real, AFFINE, IP, AV, !AV>, HG_KERNEL_STAGE, w, a, op);
    }
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
template <int P, typename real>
struct SensorTiles {
  static constexpr int EPB = epb_ns(P, sizeof(real) == 8), T = ns_threads(P, 0, sizeof(real) == 8), V0 = EPB * P * (P | 1);
  static constexpr int VM = sizeof(real) == 8 ? 16 : 32, VS = V0 + (VM + VM / 4 - V0 % VM) % VM;
  alignas(16) real Q[4 * VS];
  real U[2 * VS];
  alignas(16) real scr[T / 32 * sensor_scratch(P)];
  alignas(16) float w[MLP_PARAMS];
};
template <int P, typename real>
struct SensorOps { real Vinv[P * P]; };
template <int P, typename real>
__global__ void __launch_bounds__(ns_threads(P, 0, sizeof(real) == 8)) sensor_eval_kernel(int n_el, const double* Q, const __grid_constant__ SensorOps<P, real> op,
                                                                       SensorArgs sa, PhysConst pc, float* feat,
                                                                       double* out) {
  using Tl = SensorTiles<P, real>;
  constexpr int NP = P * P, PO = P | 1;
  extern __shared__ __align__(16) unsigned char sensor_smem[];
  Tl& s = *reinterpret_cast<Tl*>(sensor_smem);
  const int tid = threadIdx.x, e0 = blockIdx.x * Tl::EPB, n_act = min(Tl::EPB, n_el - e0);
  SensorArgs s2 = sa;
  if (sa.mlp) {
    s2.kind = SENSOR_LEARNED;
    sensor_weights_async(s.w, sa.mlp, tid, Tl::T);
  }
  for (int m = tid; m < n_act * NP; m += Tl::T)
#pragma unroll
    for (int k = 0; k < 4; ++k) s.Q[k * Tl::VS + (m / P) * PO + m % P] = real(Q[(size_t(e0) * NP + m) * 4 + k]);
  cp_async_wait_all();
  __syncthreads();
  Phys<real> ph;
  ph.load(pc);
  FlatG flat_g;
  group_sensor<P, Tl::EPB, Tl::T, real>(s2, ph, op.Vinv, s.Q, s.U, Tl::VS, s.scr, s.w, n_act, tid,
                                        feat ? feat + size_t(e0) * MLP_IN : nullptr, flat_g,
                                        [&](int le, double gm, double gl, bool ood, double) {
                                          if (!out) return;
                                          double* o = out + size_t(e0 + le) * 4;
                                          o[0] = gm;
                                          o[1] = sa.mlp ? gl : -1.0;
                                          o[2] = ood ? 1.0 : 0.0;
                                          o[3] = sa.kind == SENSOR_JUMPS ? -1.0 : sa.kind == SENSOR_LEARNED && !ood ? gl : gm;
                                        });
}

template <int P, typename real>
void launch_sensor_eval_P(hg_ctx* c, float* feat, double* out) {
  using Tl = SensorTiles<P, real>;
  static std::atomic<int> known[HG_KNOWN_DEVICES];
  resident_ctas(c, known, sensor_eval_kernel<P, real>, Tl::T, sizeof(Tl), sizeof(Tl));   // allows the shared memory
  SensorOps<P, real> op;
  const double* vinv = c->h_mats.data() + 2 * P * P + 7 * P;
  for (int k = 0; k < P * P; ++k) op.Vinv[k] = real(vinv[k]);
  const int grid = (c->n_el + Tl::EPB - 1) / Tl::EPB;
  sensor_eval_kernel<P, real><<<grid, Tl::T, sizeof(Tl), c->stream>>>(c->n_el, c->d_Q, op, sensor_args(c), c->pc, feat, out);
  ++c->launches;
}
