// hg_ns.cuh -- Navier-Stokes stage kernels (BR1 and interior penalty) for sm_100a.
//
// Launches per Runge-Kutta stage:
//   ns_gradient_kernel  BR1: the lifted gradient
//        dQ = [ -VolGreen(Q Ja) + sum_faces lift(u* dS n) ] / J,  u* = (QL + QR)/2 or the
//        boundary's viscous state (BR1_ComputeGradient, Approximation/DGViscous_BR1.f90:48-111;
//        ComputeSolutionRiemann_*, DGViscousMethods.f90:538-917), stored ([n_el][2][4][NP]) with its traces on
//        the four sides (interpolateGradientsToBoundaries, DGSpatialDiscretizationMethods.f90:1577-1631);
//        interior penalty: the traces of the local gradient (ComputeInteriorGradient,
//        Mesh/QuadElement_QuadProcedures.incf:42-88) and the element-local indicator -- only as the prologue
//        after the state is replaced (hg_set_state), or per stage on a mixed-order mesh;
//   jumps_kernel        the reference's interface-jumps indicator, from the traces alone;
//   ns_stage_kernel     F = Fi - Fv at the nodes (QDotVolumeLoop :243-268), face fluxes F* = (Fi* - Fv*) dS
//        with the neighbours' Q and dQ traces (BR1: (FvL+FvR)/2 . n; IP adds sigma0 mu N^2 invh (uL - uR),
//        DGViscous_IP.f90:45-130), boundary viscous fluxes by condition (Dirichlet / adiabatic / Neumann,
//        :1142-1511), the interior-penalty gradient-face terms lifted by Scalar_StdGradientFace
//        (DGWeakIntegrals.f90:268-495), 1/J, the RK update and the new Q traces.  Interior penalty with an
//        element-local indicator (none, modal, learned): it ends with the gradient traces of the state it
//        wrote (GT_out, the other half of a ping-pong pair, as for the Q traces) and, on the last stage of
//        a time step, the indicator of that state (mu_next): everything the next stage reads from its
//        neighbours, so a stage is this one launch.
//
// Both kernels are built like the Euler stage kernel (hg_stage.cuh): persistent CTAs over groups of EPB
// elements with the next group's inputs in flight, and inside a group phases over items (face nodes, volume
// nodes, lines) between barriers.  A product with a nodal operator is a line: one thread holds the P
// nodes of a (variable, line) in registers and takes the operator from the constant bank (BR1 in float:
// row_sums and node_volume_gradient, a node's sums in one order).  The kernels before held one node per
// thread and read the operators and the tiles from shared memory, 1.25 loads per multiply-add: their
// shared-memory pipe ran at 78-81 % of its peak at N = 7 with a quarter of the FP64 rate used, and a third
// of the warps' time went into global loads at the phase that needed them.  Measured per stage (then ->
// now): shear layer 384 x 384 N = 7 SIPG FP64 1.57 -> 1.04 ms, FP32 0.81 -> 0.62 ms; cylinder 64 x 128 N = 5
// BR1 (both kernels and the residuals) FP64 89 -> 65 us, FP32 53 -> 42 us; shock 512 x 64 N = 3 FP64
// 62 -> 48 us, FP32 35 -> 32 us.  What bounds them now: the chain of a face task (700 instructions in
// double) at 12 to 24 warps per SM, and barriers.
#pragma once
#include "hg_stage.cuh"
#include "hg_sensor.cuh"

namespace hg {

template <typename real>
struct NSArgs {
  int n_el;
  const int4* side;         // [n_el*4] {neighbour trace slot, flags, zone, per-node state row or -1}
  const real* side_geo;     // normals / dS (per node, or per side when AFFINE)
  const double* side_invh;  // [n_el*4] invh of the side's edge
  const real* vol_geo;      // element records of vol_geo_stride reals (hg_stage.cuh)
  const real* jac;          // [n_el][P*P] J (curved BR1 in float)
  const real* face_metric;  // [n_el*4][P][4] Ja00/J Ja01/J Ja10/J Ja11/J at the side nodes (curved, gradient faces)
  const Zone* zones;
  const double* bq;         // per-node Dirichlet states [rows][P][4] (sides whose side.w >= 0)
  const real* FX;           // exact-solver face fluxes [n_el*4][P][4] of this stage (RIEMANN_EXACT faces)
  const real* NF;           // mortar face fluxes [slots][P][4] of the SIDE_FLUX sides (stage kernel)
  const real* NFG;          // mortar BR1 gradient face terms [slots][P][2][4] of the SIDE_FLUX sides
  const real* NJ;           // mortar jump sums [slots][2] of the SIDE_FLUX sides (dissipation indicator)
  double* Q;
  real* G;
  const real* T_in;         // Q traces of the current state  [n_el*4][P][4]
  real* T_out;
  real* GT;                 // dQ traces of the current state [n_el*4][P][2][4]
  real* GT_out;             // dQ traces of the updated state (fused interior-penalty stages)
  real* dQ;                 // element gradients              [n_el][2][4][NP]
  int viscous;              // viscous fluxes present (ns_viscous)
  int run_gradient;         // host side: whether this stage needs the gradient kernel
  int run_jumps;            // host side: whether it needs the jumps kernel
  int run_stage;            // host side: whether to launch the stage kernel (a composite runs the
                            // mortar fluxes between the parts' gradient and stage kernels)
  double* QDot;
  double* resid;
  double a, b, c;
  int first, update, riemann;
  int ip, grad_faces;       // interior penalty (else BR1); gradient-face terms (SIPG/NIPG)
  double sigma0, epsilon;
  PhysConst pc;
  // artificial dissipation (jumps-based indicator)
  int av;                   // 0 none, 1 Laplacian, 2 Physical
  const double* av_el;      // [n_el][2] Ceps sqrt(Volume)/(N+1), sum of the 4 edge areas
  const double* side_area;  // [n_el*4] Area of each side's edge
  double* mu_av;            // [n_el] element viscosity of the current state (written by the gradient or jumps kernel)
  SensorArgs sensor;        // which indicator sets it (jumps, modal, learned)
  int fuse;                 // interior penalty, element-local indicator: the stage kernel writes GT_out and,
  int last;                 //   on the last stage of a step (last), the indicator of its new state into
  double* mu_next;          //   mu_next
  int* health;              // device health word {bits, first element} (check_state)
  int* health_host;         // mapped host flag set beside it
  int polls;                // limit of a wait for copies (mbar_wait)
};

// Elements per group and threads per CTA: variant 0, and variant 1 for small meshes.  At orders 3 and 5 a double group
// is half a float one: a CTA's shared memory then lets twice as many and more reside on an SM (order 5, where both
// variants then have groups of two: stage and gradient on the cylinder mesh 58.5 -> 56.4 us, with the jumps indicator
// 36.3 -> 32.9, in float 33.5 against 34.6; order 3, 25,000 elements, an RK3 step: interior penalty 189 -> 172 us, with
// the modal indicator 234 -> 209 us, which groups of eight ran slower than one node per thread did (220 us); in float the
// learned indicator's weights weigh more on a smaller CTA: shock 512 x 64 955 against 1050 us).
__host__ __device__ constexpr int epb_ns(int P, bool dbl) {
  return P == 2 ? 16 : P == 3 ? 8 : P == 4 ? (dbl ? 4 : 8) : P == 5 ? 4 : P == 6 ? (dbl ? 2 : 4) : P <= 8 ? 2 : 1;
}
__host__ __device__ constexpr int epb_ns_small(int P) { return P <= 3 ? 4 : P <= 6 ? 2 : 1; }
__host__ __device__ constexpr int epb_ns_of(int P, int variant, bool dbl) { return variant ? epb_ns_small(P) : epb_ns(P, dbl); }
__host__ __device__ constexpr int ns_threads(int P, int variant, bool dbl) {
  return (cmax(P * P, 4 * P) * epb_ns_of(P, variant, dbl) + 31) / 32 * 32;
}

// Nodal operators, passed by value (constant bank); dl = lb^T D, the normal derivatives at the sides.
template <int P, typename real>
struct NSOps {
  real hatD[P * P], D[P * P], lb0[P], lb1[P], lbw0[P], lbw1[P], dlbw0[P], dlbw1[P], dl0[P], dl1[P], Vinv[P * P];
};

// out = M in, row by row
template <int P, typename real>
__device__ __forceinline__ void apply(const real* M, const real (&in)[P], real (&out)[P]) {
#pragma unroll
  for (int i = 0; i < P; ++i) {
    real r = real(0);
#pragma unroll
    for (int l = 0; l < P; ++l) r += M[i * P + l] * in[l];
    out[i] = r;
  }
}
template <int P, typename real>
__device__ __forceinline__ real dot(const real* c, const real (&in)[P]) {
  real r = real(0);
#pragma unroll
  for (int l = 0; l < P; ++l) r += c[l] * in[l];
  return r;
}
template <int P, typename real>
__device__ __forceinline__ void load_line(const real* u, const int st, real (&in)[P]) {
#pragma unroll
  for (int l = 0; l < P; ++l) in[l] = u[l * st];
}
template <int P, typename real>
__device__ __forceinline__ void store_line(real* u, const int st, const real (&v)[P]) {
#pragma unroll
  for (int l = 0; l < P; ++l) u[l * st] = v[l];
}

// Shared memory of a CTA.  GRAD: the gradient kernel's (no RK register, no stored gradient to read).
template <int P, int V, typename real, bool AFFINE, bool IP, bool AV, bool VISC, bool GRAD>
struct NSTiles {
  static constexpr int EPB = epb_ns_of(P, V, sizeof(real) == 8), T = ns_threads(P, V, sizeof(real) == 8);
  static constexpr int NP = P * P, FT = 4 * P, PO = P | 1, NN = EPB * NP, NF = EPB * FT, GS = vol_geo_stride(P, AFFINE);
  static constexpr int VM = sizeof(real) == 8 ? 16 : 32, V0 = EPB * P * PO;
  static constexpr int VS = V0 + (VM + VM / 4 - V0 % VM) % VM;   // = VM / 4 modulo VM
  static constexpr bool FACES = !(GRAD && IP);            // reads traces
  static constexpr bool GT = (VISC && !GRAD) || (GRAD && !IP);   // 8-value records of the neighbours
  // Side-node records as they are copied in (one thread each): strides of an odd number of 16-byte units, so that
  // eight lanes' 128-bit reads fall into different banks.
  static constexpr int RT = sizeof(real) == 8 ? 6 : 4, RG = sizeof(real) == 8 ? 10 : 12;
  // Side tile of the fluxes (4 values) and gradient terms (8): variable-major, rows of PO per side, variable stride
  // FS = VM / 4 modulo VM.
  static constexpr int F0 = EPB * 4 * PO, FS = F0 + (VM + VM / 4 - F0 % VM) % VM;
  static constexpr int FV = GRAD ? (IP ? (AFFINE ? 12 : 0) : 8) : (IP && VISC ? 12 : 4);
  // The state record is needed again for the update; in double the Q tile holds the same values.
  static constexpr bool KEEP_Q = sizeof(real) == 4 && !GRAD;
  struct Once {                        // inputs of a group that are dead before its contraction (phase D): single,
    double Q[KEEP_Q ? 2 : NN * 4];     // the next group's are fetched as soon as they are
    real To[FACES ? NF * RT : 4];      // own traces
    real Tn[FACES ? NF * RT : 4];      // neighbours' traces (or mortar fluxes)
    real GTo[VISC && !GRAD ? NF * RG : 4];  // own gradient traces
    real GTn[GT ? NF * RG : 4];        // neighbours' gradient traces (or mortar terms)
    real dQ[!GRAD && !IP ? NN * 8 : 4];     // BR1 gradient
    real sg[!AFFINE && FACES ? NF * 3 : 4];
    double invh[EPB * 4], area[EPB * 4], mun[EPB * 4];
  };
  struct In {                          // inputs of a group that live longer: double
    double Q[KEEP_Q ? NN * 4 : 2];
    real vg[EPB * GS];
    double mu[(EPB + 1) / 2 * 2];
  };
  alignas(16) Once one;
  alignas(16) In in[2];
  alignas(16) int4 side[3][EPB * 4];
  real G[GRAD ? 4 : NN * 4];
  // Q tile (interior penalty, indicator); Fc, Gc: derivatives along the lines, then contravariant fluxes, then
  // their contractions
  alignas(16) real Q[4 * VS];
  real Fc[4 * VS], Gc[4 * VS];
  static constexpr bool SUMS = !IP && SumOps<P, real>::ON;   // BR1 in float: a node's sums in one order (hg_stage.cuh)
  // BR1 volume terms of the second direction
  real X[GRAD && !IP && !SUMS ? 4 * VS : 4], Y[GRAD && !IP && !SUMS ? 4 * VS : 4];
  SumOps<P, real, SUMS> sum;
  real F[FV ? FV * FS : 4];
  alignas(16) real sens[AV ? T / 32 * sensor_scratch(P) : 4];
  unsigned long long mx[GRAD ? 1 : 4][GRAD ? 1 : T / 32];   // per-warp max |QDot| as bits (NaN above all)
  // Registers a thread that the launch bounds leave.  Order 4 with the Laplacian dissipation alone spills 250 bytes a
  // thread at 128 (jumps indicator on 800 curved elements 55.1 -> 45.0 us an RK3 step, 16,000 elements 208 -> 181).
  static constexpr int REGS = sizeof(real) == 8 ? (P == 5 && IP && AV && !VISC ? 168 : 128) : 80;
  uint64_t bar[2];                     // inputs, RK register
  __device__ __forceinline__ const double* state(int b) const { return KEEP_Q ? in[b].Q : one.Q; }
};
// CTAs per SM the launch bounds ask for: what shared memory holds, down to Tl::REGS registers a thread.  Left
// to itself the compiler takes up to twice as many for the phase with the longest expressions.  (A learned launch holds
// the network's weights too and may have a CTA less.)
template <typename Tl>
constexpr int ns_min_ctas() {
  return cmax(1, cmin(cmin(int(227 * 1024 / (sizeof(Tl) + 1024)), 65536 / (Tl::T * Tl::REGS)), 32));
}
constexpr size_t MLP_BYTES = (size_t(MLP_PARAMS) * sizeof(float) + 15) / 16 * 16;   // after the tiles, when learned

// The part of the persistent loop that both kernels share: barriers and prefetch.
template <typename Tl, int P, typename real, bool AFFINE, bool IP, bool AV, bool VISC, bool GRAD>
struct NSPipe {
  static constexpr int EPB = Tl::EPB, T = Tl::T, NP = Tl::NP, FT = Tl::FT, GS = Tl::GS;
  const NSArgs<real>& a;
  Tl& s;
  const int tid, n_groups;
  unsigned phase = 0u;   // parities of the barriers

  __device__ __forceinline__ int count(int g) const { return min(EPB, a.n_el - g * EPB); }
  // inputs of group g (those of struct In into half b), and the side table of the group after it (thread 0)
  // first: of the CTA's first group, where the constant ones (tables, metrics) go ahead of the wait for the kernel before
  __device__ __forceinline__ void bulk(int g, int b, bool first, int slot) const {
    constexpr unsigned R = sizeof(real);
    const int e0 = g * EPB, n = count(g), gn = g + gridDim.x;
    typename Tl::In& in = s.in[b];
    uint64_t* bar = &s.bar[0];
    const unsigned bq = n * NP * 32u;
    const unsigned bd = !GRAD && !IP ? n * NP * 8u * R : 0u, bv = n * GS * R, bs = !AFFINE && Tl::FACES ? n * FT * 3u * R : 0u;
    const unsigned bh = IP && VISC && !GRAD ? n * 32u : 0u, ba = AV && !GRAD ? n * 32u : 0u;
    const unsigned b0 = first ? n * 64u : 0u, bn = gn < n_groups ? count(gn) * 64u : 0u;
    mbar_expect(bar, bq + bd + bv + bs + bh + ba + b0 + bn);
    if (b0) bulk_copy(s.side[slot], a.side + size_t(e0) * 4, b0, bar);
    bulk_copy(in.vg, a.vol_geo + size_t(e0) * GS, bv, bar);
    if (bs) bulk_copy(s.one.sg, a.side_geo + size_t(e0) * FT * 3, bs, bar);
    if (bh) bulk_copy(s.one.invh, a.side_invh + size_t(e0) * 4, bh, bar);
    if (ba) bulk_copy(s.one.area, a.side_area + size_t(e0) * 4, ba, bar);
    if (bn) bulk_copy(s.side[slot == 2 ? 0 : slot + 1], a.side + size_t(gn) * EPB * 4, bn, bar);
    if (first) grid_wait();
    bulk_copy(const_cast<double*>(s.state(b)), a.Q + size_t(e0) * NP * 4, bq, bar);
    if (bd) bulk_copy(s.one.dQ, a.dQ + size_t(e0) * NP * 8, bd, bar);
  }
  __device__ __forceinline__ int4 side_of(const int4* side, int x) const { return side[(x / FT) * 4 + (x % FT) / P]; }
  // the side-node records of group g, each copied and read by one thread; the viscosities of the group's elements
  // (into half b) and of their neighbours
  // (at0: the side-table entry of the thread's first task)
  __device__ __forceinline__ void rows(int g, int b, const int4* side, int4 at0) const {
    constexpr int RT = Tl::RT, RG = Tl::RG;
    typename Tl::Once& one = s.one;
    const int n = count(g);
    if (Tl::FACES)
      for (int x = tid; x < n * FT; x += T) {
        const int kk = x % P;
        const int4 sd = x == tid ? at0 : side_of(side, x);
        const int kind = sd.y & 15;
        const size_t own = size_t(g) * EPB * FT + x;
        if (kind != SIDE_FLUX) {
          cp_async_4(&one.To[x * RT], a.T_in + own * 4);
          if (VISC && !GRAD) {
            cp_async_4(&one.GTo[x * RG], a.GT + own * 8);
            cp_async_4(&one.GTo[x * RG + 4], a.GT + own * 8 + 4);
          }
        }
        if (kind == SIDE_LEFT || kind == SIDE_RIGHT) {
          const size_t row = size_t(sd.x) * P + ((sd.y & SIDE_REVERSED) ? P - 1 - kk : kk);
          cp_async_4(&one.Tn[x * RT], a.T_in + row * 4);
          if (VISC && !GRAD) {
            cp_async_4(&one.GTn[x * RG], a.GT + row * 8);
            cp_async_4(&one.GTn[x * RG + 4], a.GT + row * 8 + 4);
          }
        } else if (kind == SIDE_FLUX) {
          const size_t row = size_t(sd.x) * P + kk;
          if (!GRAD) cp_async_4(&one.Tn[x * RT], a.NF + row * 4);
          if (GRAD ? !IP : (VISC && IP && a.grad_faces)) {
            cp_async_4(&one.GTn[x * RG], a.NFG + row * 8);
            cp_async_4(&one.GTn[x * RG + 4], a.NFG + row * 8 + 4);
          }
        }
      }
    if (AV && !GRAD) {
      for (int x = tid; x < n * 4; x += T) {
        const int4 sd = side[x];
        const int kind = sd.y & 15;
        const bool inner = (kind == SIDE_LEFT || kind == SIDE_RIGHT) && sd.z < 0;
        cp_async_real(&one.mun[x], a.mu_av + (inner ? sd.x >> 2 : g * EPB + x / 4));
      }
      for (int x = tid; x < n; x += T) cp_async_real(&s.in[b].mu[x], a.mu_av + g * EPB + x);
    }
    cp_async_commit();
  }
  __device__ __forceinline__ void start() const {
    if (tid == 0) {
      for (int k = 0; k < 2; ++k) mbar_init(&s.bar[k]);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    const int4* side0 = a.side + size_t(blockIdx.x) * EPB * 4;
    const int4 at0 = tid < count(blockIdx.x) * FT ? side_of(side0, tid) : make_int4(0, 0, 0, 0);
    if (tid == 0) bulk(blockIdx.x, 0, true, 0);
    else grid_wait();
    rows(blockIdx.x, 0, side0, at0);
    __syncthreads();   // the barriers are initialised
  }
  // Waits for the copies of barrier k, then for the CTA: false (in every thread) where a thread gave up.
  __device__ __forceinline__ bool wait(int k) {
    const bool late = !mbar_wait(&s.bar[k], (phase >> k) & 1u, a.polls);
    if (k == 0) cp_async_wait_all();
    if (__syncthreads_or(late)) return false;
    phase ^= 1u << k;
    return true;
  }
  // ... and then: copies of barrier 0 (the inputs of group g or, while g is worked on, of the group after it) and of
  // barrier 1 may be in flight
  __device__ __forceinline__ void failed(int g, bool working) const {
    if (tid != 0) return;
    if (!working || g + int(gridDim.x) < n_groups) copies_failed(a.health, a.health_host, &s.bar[0], phase & 1u);
    if (working) copies_failed(a.health, a.health_host, &s.bar[1], (phase >> 1) & 1u);
  }
  // top of the loop for group g: its inputs are there, every thread is done with the group before, and its RK
  // register is on its way
  __device__ __forceinline__ bool next(int g, bool rk) {
    if (!wait(0)) { failed(g, false); return false; }
    if (g + int(gridDim.x) >= n_groups) grid_launch_next();   // the CTA's last group
    if (rk && tid == 0) {
      const unsigned bytes = count(g) * NP * 4u * unsigned(sizeof(real));
      mbar_expect(&s.bar[1], bytes);
      bulk_copy(s.G, a.G + size_t(g) * EPB * NP * 4, bytes, &s.bar[1]);
    }
    return true;
  }
  // after the barrier behind the face tasks: the next group's records
  __device__ __forceinline__ void prefetch_rows(int g, int b, int next_slot) const {
    const int gn = g + int(gridDim.x);
    if (gn < n_groups)
      rows(gn, b ^ 1, s.side[next_slot], tid < count(gn) * FT ? side_of(s.side[next_slot], tid) : make_int4(0, 0, 0, 0));
  }
  // after the barrier behind the last use of struct Once: the rest of the next group's inputs
  __device__ __forceinline__ void prefetch(int g, int b, int next_slot) const {
    if (tid == 0 && g + int(gridDim.x) < n_groups) bulk(g + gridDim.x, b ^ 1, false, next_slot);
  }
};

// Derivatives D u along the lines of the Q tile into Fc (xi) and Gc (eta), n_act elements.
template <int P, typename Tl, typename real>
__device__ __forceinline__ void tile_derivatives(Tl& s, const real* D, int n_act, int tid) {
  constexpr int EPB = Tl::EPB, VS = Tl::VS, PO = Tl::PO, NF = Tl::NF;
  for (int x = tid; x < 2 * NF; x += Tl::T) {   // x = (direction, variable, element, line)
    const int y = x % NF, v = y / (P * EPB), le = (y / P) % EPB, m = y % P;
    if (le >= n_act) continue;
    real in[P], out[P];
    if (x < NF) {
      const int o = v * VS + (le * P + m) * PO;
      load_line<P>(&s.Q[o], 1, in);
      apply<P>(D, in, out);
      store_line<P>(&s.Fc[o], 1, out);
    } else {
      const int o = v * VS + le * P * PO + m;
      load_line<P>(&s.Q[o], PO, in);
      apply<P>(D, in, out);
      store_line<P>(&s.Gc[o], PO, out);
    }
  }
}

// Cartesian gradient of node m (element le) from the derivative tiles.
template <int P, typename Tl, bool AFFINE, typename real>
__device__ __forceinline__ void node_gradient(const Tl& s, const real* gp, int o, real* gx, real* gy) {
  const real Ja00 = gp[0], Ja01 = gp[1], Ja10 = gp[2], Ja11 = gp[3], iJ = gp[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const real dxi = s.Fc[k * Tl::VS + o], deta = s.Gc[k * Tl::VS + o];
    gx[k] = (dxi * Ja00 + deta * Ja01) * iJ;
    gy[k] = (dxi * Ja10 + deta * Ja11) * iJ;
  }
}

// The traces at both ends of every line of tile U (4 variables) into rec[x * R + v] in global memory (x the
// element's side node), the variable fastest over the lanes.
template <int P, int R, typename Tl, typename real>
__device__ __forceinline__ void tile_traces(const real* U, const real* c0, const real* c1, real* rec, int n_act, int tid) {
  constexpr int VS = Tl::VS, PO = Tl::PO, FT = Tl::FT;
  for (int x = tid; x < n_act * FT; x += Tl::T) {   // x = (element, line, variable)
    const int v = x & 3, le = x / FT, m = (x >> 2) % P;
    real* r = rec + size_t(le) * FT * R + v;
    real in[P];
    load_line<P>(U + v * VS + (le * P + m) * PO, 1, in);
    r[(3 * P + m) * R] = dot<P>(c0, in);
    r[(P + m) * R] = dot<P>(c1, in);
    load_line<P>(U + v * VS + le * P * PO + m, PO, in);
    r[m * R] = dot<P>(c0, in);
    r[(2 * P + m) * R] = dot<P>(c1, in);
  }
}

// Gradient traces of the state in the Q tile (element-local gradient) into GT.  Affine elements: straight from
// the state -- along a side, D applied to the side's Q traces; across it, each normal line of nodes contracted
// with lb^T D -- the same as the nodal gradient interpolated to the side, without forming it at every node.
// The Q traces go to T_out when given.  Starts after a barrier on the Q tile; uses the side tile (affine) or Fc and
// Gc (curved).
template <int P, bool AFFINE, typename Tl, typename real>
__device__ __forceinline__ void gradient_traces(Tl& s, const NSOps<P, real>& op, const real* vg, real* T_out, real* GT,
                                                int n_act, int tid) {
  constexpr int VS = Tl::VS, PO = Tl::PO, FT = Tl::FT, NP = Tl::NP, GS = Tl::GS, FS = Tl::FS;
  if constexpr (AFFINE) {
    for (int x = tid; x < n_act * FT; x += Tl::T) {   // x = (element, line, variable)
      const int v = x & 3, le = x / FT, m = (x >> 2) % P;
      const auto end = [&](int side, real t, real d) {   // trace and normal derivative
        const int y = v * FS + (le * 4 + side) * PO + m;
        s.F[y] = t;
        s.F[4 * FS + y] = d;
        if (T_out) T_out[size_t(le * FT + side * P + m) * 4 + v] = t;
      };
      real in[P];
      load_line<P>(&s.Q[v * VS + (le * P + m) * PO], 1, in);
      end(3, dot<P>(op.lb0, in), dot<P>(op.dl0, in));
      end(1, dot<P>(op.lb1, in), dot<P>(op.dl1, in));
      load_line<P>(&s.Q[v * VS + le * P * PO + m], PO, in);
      end(0, dot<P>(op.lb0, in), dot<P>(op.dl0, in));
      end(2, dot<P>(op.lb1, in), dot<P>(op.dl1, in));
    }
    __syncthreads();
    for (int x = tid; x < n_act * 16; x += Tl::T) {   // x = (element, side, variable)
      const int v = x & 3, sd = (x >> 2) & 3, le = x >> 4, y = v * FS + (le * 4 + sd) * PO;
      const real* gp = vg + le * GS;
      const real Ja00 = gp[0], Ja01 = gp[1], Ja10 = gp[2], Ja11 = gp[3], iJ = gp[4];
      real in[P], dt[P];
      load_line<P>(&s.F[y], 1, in);
      apply<P>(op.D, in, dt);
      const bool alongXi = (sd & 1) == 0;   // bottom / top: along the side is xi; right / left: eta
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const real d = s.F[4 * FS + y + k];
        const real dxi = alongXi ? dt[k] : d, deta = alongXi ? d : dt[k];
        real* g = GT + size_t(le * FT + sd * P + k) * 8 + v;
        g[0] = (dxi * Ja00 + deta * Ja01) * iJ;
        g[4] = (dxi * Ja10 + deta * Ja11) * iJ;
      }
    }
  } else {
    if (T_out) tile_traces<P, 4, Tl>(s.Q, op.lb0, op.lb1, T_out, n_act, tid);
    tile_derivatives<P>(s, op.D, n_act, tid);
    __syncthreads();
    for (int m = tid; m < n_act * NP; m += Tl::T) {
      const int le = m / NP, node = m % NP, o = (m / P) * PO + node % P;
      real gx[4], gy[4];
      node_gradient<P, Tl, AFFINE>(s, vg + le * GS + node * 5, o, gx, gy);
#pragma unroll
      for (int k = 0; k < 4; ++k) { s.Fc[k * VS + o] = gx[k]; s.Gc[k * VS + o] = gy[k]; }
    }
    __syncthreads();
    tile_traces<P, 8, Tl>(s.Fc, op.lb0, op.lb1, GT, n_act, tid);
    tile_traces<P, 8, Tl>(s.Gc, op.lb0, op.lb1, GT + 4, n_act, tid);
  }
}

// JumpsBasedElementViscosity (Approximation/DGArtificialDissipation.f90:277-338) of each element into a.mu_av,
// one thread per side node.  Edge jumps (Edge_ComputeJumps and the boundary/curved variants,
// Mesh/QuadElement_EdgeProcedures.incf:1348-1619): sum over the edge nodes, in the edge's order, of
// w (2 (QL-QR)/(QL+QR))^2 dS for rho and rhoE; boundary and periodic edges use the viscous boundary
// state (uSB) and dS at their first node.  Reads traces only (the elements' own are in T_in too): bound by
// their loads.
template <int P, typename real>
struct EdgeWeights { real w[P]; };
__host__ __device__ constexpr int jumps_epb(int P) { return 128 / (4 * P); }
template <int P, typename real, bool AFFINE>
__global__ void __launch_bounds__(128) jumps_kernel(const __grid_constant__ NSArgs<real> a,
                                                    const __grid_constant__ EdgeWeights<P, real> ew) {
  constexpr int FT = 4 * P, EPB = jumps_epb(P);
  __shared__ real jr_[EPB * FT], je_[EPB * FT], sr_[EPB * 4], se_[EPB * 4];
  __shared__ bool rev_[EPB * 4];
  __shared__ real s_w[P];
  const int tid = threadIdx.x, e0 = blockIdx.x * EPB, n_act = min(EPB, a.n_el - e0);
  if (tid < P) {
    real w = ew.w[0];
#pragma unroll
    for (int k = 1; k < P; ++k) w = tid == k ? ew.w[k] : w;
    s_w[tid] = w;
  }
  Phys<real> ph;
  ph.load(a.pc);
  // constant tables, ahead of the wait for the kernel before
  const int kk = tid % P;
  const size_t sbase = size_t(e0) * 4 + tid / P, slot = size_t(e0) * FT + tid;
  const int4 sd = tid < n_act * FT ? a.side[sbase] : make_int4(0, 0, 0, 0);
  const int kind = sd.y & 15;
  double visc = 0.0, area = 1.0;
  if (tid < n_act) {
    visc = a.av_el[2 * size_t(e0 + tid)];
    area = a.av_el[2 * size_t(e0 + tid) + 1];
  }
  __syncthreads();
  grid_wait();
  grid_launch_next();
  if (tid < n_act * FT) {
    if (kk == 0) rev_[tid / P] = kind == SIDE_RIGHT && (sd.y & SIDE_REVERSED);
    if (kind == SIDE_FLUX) {   // edge between orders or subdivided edge: the mortar kernel's jump sums
      jr_[tid] = kk == 0 ? a.NJ[size_t(sd.x) * 2] : real(0);
      je_[tid] = kk == 0 ? a.NJ[size_t(sd.x) * 2 + 1] : real(0);
    } else {
      real qo[4], qn0, qn3;
      ld4(a.T_in + slot * 4, qo);
      bool node0 = true;
      if (kind == SIDE_LEFT || kind == SIDE_RIGHT) {
        const int kn = (sd.y & SIDE_REVERSED) ? (P - 1 - kk) : kk;
        real qn[4];
        ld4(a.T_in + (size_t(sd.x) * P + kn) * 4, qn);
        qn0 = qn[0];
        qn3 = qn[3];
        node0 = sd.z >= 0;   // periodic edges are boundary edges of the reference
      } else {
        const real* g3 = AFFINE ? a.side_geo + sbase * 3 : a.side_geo + slot * 3;
        real uB[4], uS[4];
        bc_states(ph, a.zones[sd.z], qo, g3[0], g3[1], uB, uS, sd.w >= 0 ? a.bq + (size_t(sd.w) * P + kk) * 4 : nullptr);
        qn0 = uS[0];
        qn3 = uS[3];
      }
      const real dSn = AFFINE ? a.side_geo[sbase * 3 + 2] : a.side_geo[(sbase * P + (node0 ? 0 : kk)) * 3 + 2];
      const real jr = real(2) * (qo[0] - qn0) / (qo[0] + qn0);
      const real je = real(2) * (qo[3] - qn3) / (qo[3] + qn3);
      jr_[tid] = s_w[kk] * jr * jr * dSn;
      je_[tid] = s_w[kk] * je * je * dSn;
    }
  }
  __syncthreads();
  if (tid < n_act * 4) {   // a side's sum, in its edge's order
    const bool rev = rev_[tid];
    real sr = real(0), se = real(0);
    for (int n = 0; n < P; ++n) {
      const int x = tid * P + (rev ? (P - 1 - n) : n);
      sr = sr + jr_[x];
      se = se + je_[x];
    }
    sr_[tid] = sr;
    se_[tid] = se;
  }
  __syncthreads();
  if (tid < n_act) {
    real gr = real(0), ge = real(0);
#pragma unroll
    for (int sd_ = 0; sd_ < 4; ++sd_) {
      gr = gr + sr_[tid * 4 + sd_];
      ge = ge + se_[tid * 4 + sd_];
    }
    double gk = double(gr > ge ? gr : ge) / area;
    gk = gk > 1.0e-8 ? log10(gk) : -1.7976931348623157e308;
    const double k = 5.0;
    const double s0 = log10(1.0 / ((P * P) * double(P * P))) + 1.0;
    double G;
    if (gk < s0 - k) G = 0.0;
    else if (gk < s0 + k) G = 0.5 * sin(0.5 * 3.141592653589793238462643 * (gk - s0) / k) + 0.5;
    else G = 1.0;
    a.mu_av[e0 + tid] = visc * G;
  }
}

// BR1 in float: the volume terms of a node's gradient (hatD along both lines, times the metrics), x and y components.
template <int P, typename Tl, bool AFFINE, typename real>
__device__ __forceinline__ void node_volume_gradient(const Tl& s, const real* vg, int le, int node, real* vx, real* vy) {
  constexpr int VS = Tl::VS, PO = Tl::PO;
  const int i = node % P, j = node / P;
  const real *row = &s.Q[(le * P + j) * PO], *col = &s.Q[le * P * PO + i];
  real ax[4] = {real(0), real(0), real(0), real(0)}, ay[4] = {real(0), real(0), real(0), real(0)};
#pragma unroll
  for (int l = 0; l < P; ++l) {
    const real hi = s.sum.hatT[l * P + i], hj = s.sum.hatT[l * P + j];
    if constexpr (AFFINE) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        ax[k] += hi * row[k * VS + l];
        ay[k] += hj * col[k * VS + l * PO];
      }
    } else {
      const real *gx = vg + (j * P + l) * 5, *gy = vg + (l * P + i) * 5;
      const real j0 = gx[0], j1 = gy[1], j2 = gx[2], j3 = gy[3];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const real qx = row[k * VS + l] * hi, qy = col[k * VS + l * PO] * hj;
        ax[k] += qx * j0 + qy * j1;
        ay[k] += qx * j2 + qy * j3;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    vx[k] = AFFINE ? ax[k] * vg[0] + ay[k] * vg[1] : ax[k];
    vy[k] = AFFINE ? ax[k] * vg[2] + ay[k] * vg[3] : ay[k];
  }
}

// Gradient kernel.  BR1: lifted gradient (stored) and its traces; interior penalty: gradient traces of the
// resident state.  Then the modal or learned indicator, on the first stage of a time step (and for a bare
// time derivative); the later stages of the step keep that viscosity.
template <int P, int V, typename real, bool AFFINE, bool IP, bool AV>
__global__ void __launch_bounds__(ns_threads(P, V, sizeof(real) == 8))
    ns_gradient_kernel(const __grid_constant__ NSArgs<real> a, const __grid_constant__ NSOps<P, real> op) {
  using Tl = NSTiles<P, V, real, AFFINE, IP, AV, true, true>;
  constexpr int EPB = Tl::EPB, T = Tl::T, NP = Tl::NP, FT = Tl::FT, PO = Tl::PO, VS = Tl::VS, GS = Tl::GS, NF = Tl::NF,
                FS = Tl::FS, RT = Tl::RT, RG = Tl::RG;
  extern __shared__ __align__(16) unsigned char stage_smem[];
  Tl& s = *reinterpret_cast<Tl*>(stage_smem);
  float* s_w = reinterpret_cast<float*>(stage_smem + sizeof(Tl));
  const int tid = threadIdx.x, n_groups = (a.n_el + EPB - 1) / EPB;
  NSPipe<Tl, P, real, AFFINE, IP, AV, true, true> pipe{a, s, tid, n_groups};
  Phys<real> ph;
  ph.load(a.pc);
  const bool sense = AV && a.sensor.kind != SENSOR_JUMPS && a.first;
  if (sense && a.sensor.kind == SENSOR_LEARNED) sensor_weights_async(s_w, a.sensor.mlp, tid, T);
  s.sum.fill(op, tid, T);
  pipe.start();
  FlatG flat_g;
  int b = 0, slot = 0;
  for (int g = blockIdx.x; g < n_groups; g += gridDim.x) {
    const int e0 = g * EPB, n_act = pipe.count(g), next_slot = slot == 2 ? 0 : slot + 1;
    if (!pipe.next(g, false)) return;
    typename Tl::In& in = s.in[b];
    const int4* side = s.side[slot];
    const double* Qg = s.state(b);
    for (int m = tid; m < n_act * NP; m += T) {
      const int o = (m / P) * PO + m % P;
      double q[4];
      ld4(Qg + m * 4, q);
#pragma unroll
      for (int k = 0; k < 4; ++k) s.Q[k * VS + o] = real(q[k]);
    }
    if constexpr (IP) {
      __syncthreads();
      pipe.prefetch(g, b, next_slot);
      if (a.viscous) {
        gradient_traces<P, AFFINE>(s, op, in.vg, static_cast<real*>(nullptr), a.GT + size_t(e0) * FT * 8, n_act, tid);
      }
    } else {
      // face terms u* dS n (outward normal of this element)
      for (int x = tid; x < n_act * FT; x += T) {
        const int t = x % FT, sd_ = t / P, kk = t % P, le = x / FT;
        const int4 sd = side[le * 4 + sd_];
        const int kind = sd.y & 15;
        const int y = (le * 4 + sd_) * PO + kk;
        if (kind == SIDE_FLUX) {   // the mortar kernel's terms
#pragma unroll
          for (int k = 0; k < 8; ++k) s.F[k * FS + y] = s.one.GTn[x * RG + k];
          continue;
        }
        real qo[4], us[4];
        ld4(&s.one.To[x * RT], qo);
        const real* g3 = AFFINE ? &in.vg[le * GS + 8 + sd_ * 3] : &s.one.sg[x * 3];
        const real nx = g3[0], ny = g3[1], dS = g3[2];
        if (kind == SIDE_LEFT || kind == SIDE_RIGHT) {
          real tp[4];
          ld4(&s.one.Tn[x * RT], tp);
#pragma unroll
          for (int k = 0; k < 4; ++k) us[k] = real(0.5) * (tp[k] + qo[k]);
        } else {
          real uB[4];
          bc_states(ph, a.zones[sd.z], qo, nx, ny, uB, us, sd.w >= 0 ? a.bq + (size_t(sd.w) * P + kk) * 4 : nullptr);
        }
        const real sg = kind == SIDE_RIGHT ? -dS : dS;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          s.F[k * FS + y] = us[k] * sg * nx;
          s.F[(4 + k) * FS + y] = us[k] * sg * ny;
        }
      }
      __syncthreads();
      pipe.prefetch(g, b, next_slot);
      pipe.prefetch_rows(g, b, next_slot);
      // per line: minus the volume term plus the lift at its ends, for the x and y components; rows into Fc, Gc,
      // columns into X, Y.  (Float: the sums of a node in one order, below.)
      if constexpr (!Tl::SUMS) for (int x = tid; x < 2 * NF; x += T) {   // x = (direction, variable, element, line)
        const int y = x % NF, v = y / (P * EPB), le = (y / P) % EPB, m = y % P;
        if (le >= n_act) continue;
        const bool xi = x < NF;
        const int o = xi ? v * VS + (le * P + m) * PO : v * VS + le * P * PO + m, st = xi ? 1 : PO;
        const real* f0 = &s.F[v * FS + (le * 4 + (xi ? 3 : 0)) * PO + m];
        const real* f1 = &s.F[v * FS + (le * 4 + (xi ? 1 : 2)) * PO + m];
        real q[P], ox[P], oy[P];
#pragma unroll
        for (int l = 0; l < P; ++l) q[l] = s.Q[o + l * st];
        if constexpr (AFFINE) {
          const real* gp = &in.vg[le * GS];
          const real jx = xi ? gp[0] : gp[1], jy = xi ? gp[2] : gp[3];
          real r[P];
          apply<P>(op.hatD, q, r);
#pragma unroll
          for (int i = 0; i < P; ++i) { ox[i] = r[i] * jx; oy[i] = r[i] * jy; }
        } else {
          const real* gp = &in.vg[le * GS + (xi ? m * P * 5 : m * 5 + 1)];
          const int gst = xi ? 5 : 5 * P;
          real qx[P], qy[P];
#pragma unroll
          for (int l = 0; l < P; ++l) { qx[l] = q[l] * gp[l * gst]; qy[l] = q[l] * gp[l * gst + 2]; }
          apply<P>(op.hatD, qx, ox);
          apply<P>(op.hatD, qy, oy);
        }
        real* dx = xi ? s.Fc : s.X;
        real* dy = xi ? s.Gc : s.Y;
#pragma unroll
        for (int i = 0; i < P; ++i) {
          dx[o + i * st] = f0[0] * op.lbw0[i] + f1[0] * op.lbw1[i] - ox[i];
          dy[o + i * st] = f0[4 * FS] * op.lbw0[i] + f1[4 * FS] * op.lbw1[i] - oy[i];
        }
      }
      if constexpr (!Tl::SUMS) __syncthreads();
      for (int m = tid; m < n_act * NP; m += T) {
        const int le = m / NP, node = m % NP, o = (m / P) * PO + node % P;
        real* gq = a.dQ + size_t(e0 + le) * 8 * NP + node;
        real iJ, vx[4], vy[4];
        if constexpr (Tl::SUMS) {
          iJ = AFFINE ? in.vg[le * GS + 4] : real(1) / a.jac[size_t(e0) * NP + m];
          node_volume_gradient<P, Tl, AFFINE>(s, &in.vg[le * GS], le, node, vx, vy);
        } else {
          iJ = AFFINE ? in.vg[le * GS + 4] : in.vg[le * GS + node * 5 + 4];
        }
        const int i = node % P, j = node / P;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          real gx, gy;
          if constexpr (Tl::SUMS) {
            const real* f = &s.F[k * FS + le * 4 * PO];   // (side, node): f[side * PO + node], the y components 4 FS on
            const real lx = f[i] * s.sum.lbw0[j] + f[PO + j] * s.sum.lbw1[i] + f[2 * PO + i] * s.sum.lbw1[j] +
                            f[3 * PO + j] * s.sum.lbw0[i];
            const real* h = f + 4 * FS;
            const real ly = h[i] * s.sum.lbw0[j] + h[PO + j] * s.sum.lbw1[i] + h[2 * PO + i] * s.sum.lbw1[j] +
                            h[3 * PO + j] * s.sum.lbw0[i];
            gx = (-vx[k] + lx) * iJ;
            gy = (-vy[k] + ly) * iJ;
          } else {
            gx = (s.Fc[k * VS + o] + s.X[k * VS + o]) * iJ;
            gy = (s.Gc[k * VS + o] + s.Y[k * VS + o]) * iJ;
          }
          gq[k * NP] = gx;   // the lifted gradient is not local: stored for the stage kernel
          gq[(4 + k) * NP] = gy;
          s.Fc[k * VS + o] = gx;
          s.Gc[k * VS + o] = gy;
        }
      }
      if (a.viscous) {   // gradient traces only feed viscous face fluxes
        __syncthreads();
        tile_traces<P, 8, Tl>(s.Fc, op.lb0, op.lb1, a.GT + size_t(e0) * FT * 8, n_act, tid);
        tile_traces<P, 8, Tl>(s.Gc, op.lb0, op.lb1, a.GT + size_t(e0) * FT * 8 + 4, n_act, tid);
      }
    }
    if (sense) {
      __syncthreads();
      group_sensor<P, EPB, T, real>(a.sensor, ph, op.Vinv, s.Q, s.Fc, VS, s.sens, s_w, n_act, tid, nullptr, flat_g,
                                    [&](int le, double, double, bool, double g) {
                                      a.mu_av[e0 + le] = a.av_el[2 * size_t(e0 + le)] * g;
                                    });
    }
    b ^= 1;
    slot = next_slot;
  }
}

// Volume flux of a node: F = Fi - (mu + mu_a) Fv (- mu_a grad Q for the Laplacian dissipation, with the
// element-local gradient), contravariant, into Fc and Gc at o.  gx, gy: gradient of the viscous flux;
// ax, ay: that of the dissipation.
template <int VS, bool AV, bool VISC, typename real>
__device__ __forceinline__ void ns_volume_flux(const Phys<real>& ph, const real* q, const real* gx, const real* gy,
                                               const real* ax, const real* ay, real mu_v, real mu_l, const real* gp,
                                               real* Fc, real* Gc) {
  real fi[4], gi[4], fv[4], gv[4];
  volume_flux(ph, q, fi, gi);
  if (VISC) viscous_flux(ph, q, gx, gy, fv, gv);
  const real Ja00 = gp[0], Ja01 = gp[1], Ja10 = gp[2], Ja11 = gp[3];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    real f = fi[k], g = gi[k];
    if (VISC) { f -= mu_v * fv[k]; g -= mu_v * gv[k]; }
    if (AV) { f -= mu_l * ax[k]; g -= mu_l * ay[k]; }
    Fc[k * VS] = f * Ja00 + g * Ja10;
    Gc[k * VS] = f * Ja01 + g * Ja11;
  }
}

// Face task x (element le, side node t): the side's flux F* dS (signed for a RIGHT side) into the side
// tile and, with SIPG / NIPG, the contravariant gradient-face terms behind it (xi components first)
// (ComputeRiemannSolver_* and the viscous face loops, DGSpatialDiscretizationMethods.f90:545-1511;
// DGViscous_BR1.f90:311-371, DGViscous_IP.f90:120-134, 240-247; DGArtificialDissipation.f90:208-249).
template <int P, typename Tl, typename real, bool AFFINE, bool IP, bool AV, bool VISC>
__device__ __forceinline__ void ns_face_task(const NSArgs<real>& a, const Phys<real>& ph, Tl& s, const typename Tl::In& in,
                                             const int4* side, int x, int e0) {
  constexpr int FT = Tl::FT, GS = Tl::GS, FS = Tl::FS, RT = Tl::RT, RG = Tl::RG;
  const typename Tl::Once& one = s.one;
  const int le = x / FT, t = x % FT, sd_ = t / P, kk = t % P;
  real* Fo = &s.F[(le * 4 + sd_) * Tl::PO + kk];
  const int4 sd = side[le * 4 + sd_];
  const int kind = sd.y & 15;
  const bool gf = IP && VISC && a.grad_faces;
  const size_t slot = size_t(e0) * FT + x;
  real fm[4];   // Ja / J at the side node: contravariant components of the gradient-face terms
  if (gf) {
    if (AFFINE) {
      const real* gp = &in.vg[le * GS];
#pragma unroll
      for (int k = 0; k < 4; ++k) fm[k] = gp[k] * gp[4];
    } else {
      ld4(a.face_metric + slot * 4, fm);
    }
  }
  const auto grad_terms = [&](const real* Gx, const real* Gy) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const real gx = Gx[k], gy = Gy[k];
      Fo[(4 + k) * FS] = gx * fm[0] + gy * fm[2];
      Fo[(8 + k) * FS] = gx * fm[1] + gy * fm[3];
    }
  };
  if (kind == SIDE_FLUX) {   // inviscid and viscous flux of the mortar kernel, and its gradient-face terms
    real f[4];
    ld4(&one.Tn[x * RT], f);
#pragma unroll
    for (int k = 0; k < 4; ++k) Fo[k * FS] = f[k];
    if (gf) {
      real gx[4], gy[4];
      ld4(&one.GTn[x * RG], gx);
      ld4(&one.GTn[x * RG + 4], gy);
      grad_terms(gx, gy);
    }
    return;
  }
  real qo[4], gox[4], goy[4];
  ld4(&one.To[x * RT], qo);
  if (VISC) {
    ld4(&one.GTo[x * RG], gox);
    ld4(&one.GTo[x * RG + 4], goy);
  }
  const real* g3 = AFFINE ? &in.vg[le * GS + 8 + sd_ * 3] : &one.sg[x * 3];
  const real nx = g3[0], ny = g3[1], dS = g3[2], mu = ph.mu;
  // edge viscosity (JumpsBasedEdgeViscosity): mean over the edge's elements; boundary and
  // periodic edges have one element (the neighbour's slot then holds this element's)
  real mu_ed = real(0);
  if (AV) mu_ed = (real(one.mun[le * 4 + sd_]) + real(in.mu[le])) / real(2);
  const real mu_f = (AV && a.av == 2) ? mu + mu_ed : mu;
  const real lap = (AV && a.av == 1) ? mu_ed * real(one.area[le * 4 + sd_]) : real(0);
  real penalty = real(0);
  if (IP && VISC) penalty = real(a.sigma0) * mu_f * real(P - 1) * real(P - 1) * real(one.invh[le * 4 + sd_]);
  real F[4], fv[4] = {real(0), real(0), real(0), real(0)};   // fv: viscous flux (times dS on a boundary)
  if (kind == SIDE_LEFT || kind == SIDE_RIGHT) {
    const bool right = kind == SIDE_RIGHT;
    real qn[4], QL[4], QR[4];
    ld4(&one.Tn[x * RT], qn);
#pragma unroll
    for (int k = 0; k < 4; ++k) { QL[k] = right ? qn[k] : qo[k]; QR[k] = right ? qo[k] : qn[k]; }
    int solver = a.riemann;
    if (sd.z >= 0) { const int zr = a.zones[sd.z].riemann; if (zr >= 0) solver = zr; }
    face_riemann(solver, ph, QL, QR, nx, ny, a.FX, slot, F);
    const real sg = right ? -dS : dS;
    if (VISC) {
      real gnx[4], gny[4], ox[4], oy[4], bx[4], by[4];
      ld4(&one.GTn[x * RG], gnx);
      ld4(&one.GTn[x * RG + 4], gny);
      viscous_flux(ph, qo, gox, goy, ox, oy);
      viscous_flux(ph, qn, gnx, gny, bx, by);
      if constexpr (IP) {
        const real hm = real(0.5) * mu_f;
#pragma unroll
        for (int k = 0; k < 4; ++k) F[k] -= hm * (ox[k] + bx[k]) * nx + hm * (oy[k] + by[k]) * ny;
      } else {   // LEFT's term first
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const real lx = right ? bx[k] : ox[k], rx = right ? ox[k] : bx[k], ly = right ? by[k] : oy[k], ry = right ? oy[k] : by[k];
          fv[k] = real(0.5) * (mu_f * lx + mu_f * rx) * nx + real(0.5) * (mu_f * ly + mu_f * ry) * ny;
        }
      }
      if (gf) {
        real fgx[4], fgy[4], Ax[4], Ay[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) { const real d = QL[k] - QR[k]; fgx[k] = d * nx; fgy[k] = d * ny; }
        viscous_flux(ph, qo, fgx, fgy, Ax, Ay);
        const real cf = real(0.5) * real(a.epsilon) * mu_f * sg;
#pragma unroll
        for (int k = 0; k < 4; ++k) { Ax[k] *= cf; Ay[k] *= cf; }
        grad_terms(Ax, Ay);
      }
    }
    if constexpr (IP) {
      const real jump = AV ? penalty + lap : penalty;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (VISC || AV) F[k] += jump * (QL[k] - QR[k]);
        F[k] *= sg;
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (AV) {
          const real fa = -(lap * (QL[k] - QR[k]));
          F[k] = (F[k] - fv[k] - fa) * dS;
        } else {
          F[k] = (F[k] - fv[k]) * dS;
        }
        if (right) F[k] = -F[k];
      }
    }
  } else {
    const Zone& z = a.zones[sd.z];
    real uB[4], uSB[4];
    const int vbc = bc_states(ph, z, qo, nx, ny, uB, uSB, sd.w >= 0 ? a.bq + (size_t(sd.w) * P + kk) * 4 : nullptr);
    if (kind == SIDE_WALL) {
      euler_wall_flux(ph, qo, nx, ny, dS, F);
    } else {
      const int solver = z.riemann >= 0 ? z.riemann : a.riemann;
      face_riemann(solver, ph, qo, uB, nx, ny, a.FX, slot, F);
#pragma unroll
      for (int k = 0; k < 4; ++k) F[k] = F[k] * dS;
    }
    if (VISC) {
      real Gx[4] = {real(0), real(0), real(0), real(0)}, Gy[4] = {real(0), real(0), real(0), real(0)};
      if (vbc != VBC_NEUMANN) {
        real Fx[4], Fy[4];
        if (vbc == VBC_ADIABATIC) viscous_flux_adiabatic(ph, qo, qo, gox, goy, Fx, Fy);
        else viscous_flux(ph, qo, gox, goy, Fx, Fy);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          fv[k] = (mu_f * Fx[k]) * nx + (mu_f * Fy[k]) * ny;
          if (IP) fv[k] = fv[k] - penalty * (qo[k] - uSB[k]);
          fv[k] = fv[k] * dS;
        }
        if (gf) {
          real fgx[4], fgy[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) { fgx[k] = (qo[k] - uSB[k]) * nx; fgy[k] = (qo[k] - uSB[k]) * ny; }
          if (vbc == VBC_ADIABATIC) viscous_flux_adiabatic(ph, qo, qo, fgx, fgy, Gx, Gy);
          else viscous_flux(ph, qo, fgx, fgy, Gx, Gy);
          const real cf = real(a.epsilon) * mu_f;
#pragma unroll
          for (int k = 0; k < 4; ++k) { Gx[k] = (cf * Gx[k]) * dS; Gy[k] = (cf * Gy[k]) * dS; }
        }
      }
      if (gf) grad_terms(Gx, Gy);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = AV ? F[k] - fv[k] - (-(lap * (qo[k] - uSB[k]))) * dS : F[k] - fv[k];
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) Fo[k * FS] = F[k];
}

// Stage kernel, per group (a barrier between the phases):
//   A  face nodes and volume nodes as one list of items, faces first in whole warps.  Where the volume flux needs
//      the element-local gradient (interior penalty with viscous terms; the Laplacian dissipation of a group that
//      holds an element with viscosity) the nodes only fill the Q tile, else they form their fluxes;
//   B  (with that gradient) lines: D along both directions; and the gradient-face terms, contracted with hatD along
//      their side (they enter the lift at every node of a normal line with the same value);
//   C  (with that gradient) nodes: fluxes;
//   D  lines: contraction with hatD, lift of the face fluxes (lbw) and the gradient-face terms (lbw, dlbw); BR1 in float:
//      rows of nodes, both directions in one sum (row_sums, hg_stage.cuh);
//   E  nodes: 1/J, RK update, health check;
//   F  lines: traces of the new state and, on the fused path, of its gradient; then its indicator.
template <int P, int V, typename real, bool AFFINE, bool IP, bool AV, bool VISC>
__global__ void __launch_bounds__(ns_threads(P, V, sizeof(real) == 8), ns_min_ctas<NSTiles<P, V, real, AFFINE, IP, AV, VISC, false>>())
    ns_stage_kernel(const __grid_constant__ NSArgs<real> a, const __grid_constant__ NSOps<P, real> op) {
  using Tl = NSTiles<P, V, real, AFFINE, IP, AV, VISC, false>;
  constexpr int EPB = Tl::EPB, T = Tl::T, NP = Tl::NP, FT = Tl::FT, PO = Tl::PO, VS = Tl::VS, GS = Tl::GS, NF = Tl::NF,
                FS = Tl::FS;
  extern __shared__ __align__(16) unsigned char stage_smem[];
  Tl& s = *reinterpret_cast<Tl*>(stage_smem);
  float* s_w = reinterpret_cast<float*>(stage_smem + sizeof(Tl));
  const int tid = threadIdx.x, n_groups = (a.n_el + EPB - 1) / EPB;
  NSPipe<Tl, P, real, AFFINE, IP, AV, VISC, false> pipe{a, s, tid, n_groups};
  Phys<real> ph;
  ph.load(a.pc);
  const bool sense = IP && AV && a.fuse && a.update && a.last && a.sensor.kind != SENSOR_JUMPS;
  const bool gf = IP && VISC && a.grad_faces, rk = a.update && !a.first;
  if (sense && a.sensor.kind == SENSOR_LEARNED) sensor_weights_async(s_w, a.sensor.mlp, tid, T);
  if ((tid & 31) < 4) s.mx[tid & 31][tid >> 5] = 0ull;
  s.sum.fill(op, tid, T);
  pipe.start();
  FlatG flat_g;
  int b = 0, slot = 0;
  for (int g = blockIdx.x; g < n_groups; g += gridDim.x) {
    const int e0 = g * EPB, n_act = pipe.count(g), next_slot = slot == 2 ? 0 : slot + 1;
    if (!pipe.next(g, rk)) return;
    typename Tl::In& in = s.in[b];
    const int4* side = s.side[slot];
    bool local = IP && VISC;   // the volume fluxes need the element-local gradient (uniform over the CTA)
    if (AV && !local && a.av == 1)
      for (int le = 0; le < n_act; ++le) local = local || in.mu[le] != 0.0;

    // A.  Where the face nodes leave whole warps over, those take all volume nodes (a face task is three times as
    // long as a node's); else every warp does its faces, then its nodes.
    constexpr int NFR = (NF + 31) / 32 * 32, NT = T > NFR ? T - NFR : T;
    static_assert(NFR <= T, "one round of face tasks");
    if (tid < n_act * FT) ns_face_task<P, Tl, real, AFFINE, IP, AV, VISC>(a, ph, s, in, side, tid, e0);
    if (T == NFR || tid >= NFR) {
      for (int m = T == NFR ? tid : tid - NFR; m < n_act * NP; m += NT) {
        const int le = m / NP, node = m % NP, o = (m / P) * PO + node % P;
        double qd[4];
        ld4(&s.state(b)[m * 4], qd);
        const real q[4] = {real(qd[0]), real(qd[1]), real(qd[2]), real(qd[3])};
        if (local || !Tl::KEEP_Q)
#pragma unroll
          for (int k = 0; k < 4; ++k) s.Q[k * VS + o] = q[k];
        if (!local) {
          const real* gp = AFFINE ? &in.vg[le * GS] : &in.vg[le * GS + node * 5];
          real gx[4], gy[4];
          if constexpr (VISC && !IP) {
            const real* gq = &s.one.dQ[le * 8 * NP + node];
#pragma unroll
            for (int k = 0; k < 4; ++k) { gx[k] = gq[k * NP]; gy[k] = gq[(4 + k) * NP]; }
          }
          const real mu_v = (AV && a.av == 2) ? ph.mu + real(in.mu[le]) : ph.mu;
          if constexpr (!(IP && VISC))
            ns_volume_flux<VS, false, VISC>(ph, q, gx, gy, gx, gy, mu_v, real(0), gp, &s.Fc[o], &s.Gc[o]);
        }
      }
    }
    __syncthreads();
    pipe.prefetch_rows(g, b, next_slot);

    if (local) {
      // B
      tile_derivatives<P>(s, op.D, n_act, tid);
      if (gf)
        for (int x = tid; x < n_act * 16; x += T) {   // x = (element, side, variable)
          const int v = x & 3, sd = (x >> 2) & 3, le = x >> 4;
          // bottom / top: the xi component along the side; right / left: the eta one
          real* u = &s.F[(4 + (sd & 1) * 4 + v) * FS + (le * 4 + sd) * PO];
          real c[P], d[P];
          load_line<P>(u, 1, c);
          apply<P>(op.hatD, c, d);
          store_line<P>(u, 1, d);
        }
      __syncthreads();
      // C
      for (int m = tid; m < n_act * NP; m += T) {
        const int le = m / NP, node = m % NP, o = (m / P) * PO + node % P;
        const real* gp = AFFINE ? &in.vg[le * GS] : &in.vg[le * GS + node * 5];
        real q[4], ax[4], ay[4], gx[4], gy[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = s.Q[k * VS + o];
        node_gradient<P, Tl, AFFINE>(s, gp, o, ax, ay);
        if constexpr (VISC && !IP) {
          const real* gq = &s.one.dQ[le * 8 * NP + node];
#pragma unroll
          for (int k = 0; k < 4; ++k) { gx[k] = gq[k * NP]; gy[k] = gq[(4 + k) * NP]; }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) { gx[k] = ax[k]; gy[k] = ay[k]; }
        }
        const real mu_e = AV ? real(in.mu[le]) : real(0);
        ns_volume_flux<VS, AV, VISC>(ph, q, gx, gy, ax, ay, (AV && a.av == 2) ? ph.mu + mu_e : ph.mu,
                                     a.av == 1 ? mu_e : real(0), gp, &s.Fc[o], &s.Gc[o]);
      }
      __syncthreads();
    }

    pipe.prefetch(g, b, next_slot);

    // D
    if constexpr (Tl::SUMS) {
      for (int x = tid; x < NF; x += T) {   // x = (variable, element, row)
        const int v = x / (P * EPB), le = (x / P) % EPB, m = x % P;
        if (le >= n_act) continue;
        const real* Fv = &s.F[v * FS + le * 4 * PO];
        real r[P], *Fc = &s.Fc[v * VS + (le * P + m) * PO];
        row_sums<P, PO, false>(op, s.sum, Fc, &s.Gc[v * VS + le * P * PO], m, [&](int sd, int k) { return Fv[sd * PO + k]; }, r);
        store_line<P>(Fc, 1, r);
      }
    } else for (int x = tid; x < 2 * NF; x += T) {   // x = (direction, variable, element, line)
      const int y = x % NF, v = y / (P * EPB), le = (y / P) % EPB, m = y % P;
      if (le >= n_act) continue;
      const bool xi = x < NF;
      // the line's end nodes
      const real* f0 = &s.F[v * FS + (le * 4 + (xi ? 3 : 0)) * PO + m];
      const real* f1 = &s.F[v * FS + (le * 4 + (xi ? 1 : 2)) * PO + m];
      real c0 = *f0, c1 = *f1, d0 = real(0), d1 = real(0);
      if (gf) {   // contracted terms add to the lbw part, the normal components to the dlbw part
        const int ct = (xi ? 8 : 4) * FS, nt = (xi ? 4 : 8) * FS;
        c0 += f0[ct];
        c1 += f1[ct];
        d0 = f0[nt];
        d1 = f1[nt];
      }
      const auto line = [&](real* u, const int st) {
        real f[P], r[P];
        load_line<P>(u, st, f);
        apply<P>(op.hatD, f, r);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          r[i] -= c0 * op.lbw0[i];
          r[i] -= c1 * op.lbw1[i];
          if (IP && VISC) {
            r[i] -= d0 * op.dlbw0[i];
            r[i] -= d1 * op.dlbw1[i];
          }
        }
        store_line<P>(u, st, r);
      };
      if (xi) line(&s.Fc[v * VS + (le * P + m) * PO], 1);
      else line(&s.Gc[v * VS + le * P * PO + m], PO);
    }
    if (!rk) {
      __syncthreads();
    } else if (!pipe.wait(1)) {
      pipe.failed(g, true);
      return;
    }

    // E
    for (int m = tid; m < (Tl::NN + 31) / 32 * 32; m += T) {
      const bool on = m < n_act * NP;
      const int le = m / NP, node = m % NP, o = (m / P) * PO + node % P;
      const size_t off = (size_t(e0) * NP + m) * 4;
      real qd[4] = {real(0), real(0), real(0), real(0)};
      if (on) {
        const real iJ = AFFINE ? in.vg[le * GS + 4] : in.vg[le * GS + node * 5 + 4];
#pragma unroll
        for (int k = 0; k < 4; ++k) qd[k] = (Tl::SUMS ? s.Fc[k * VS + o] : s.Fc[k * VS + o] + s.Gc[k * VS + o]) * iJ;
      }
      if (a.resid)   // the whole warp takes part
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned long long w = warp_max_bits(fabs(double(qd[k])));
          if ((tid & 31) == 0 && w > s.mx[k][tid >> 5]) s.mx[k][tid >> 5] = w;
        }
      if (!on) continue;
      if (a.QDot) {
        const double dq[4] = {double(qd[0]), double(qd[1]), double(qd[2]), double(qd[3])};
        st4(a.QDot + off, dq);
      }
      if (a.update) {
        real gn[4];
        if (a.first) {
#pragma unroll
          for (int k = 0; k < 4; ++k) gn[k] = real(a.b) * qd[k];
        } else {
          ld4(&s.G[m * 4], gn);
#pragma unroll
          for (int k = 0; k < 4; ++k) gn[k] = real(a.a) * gn[k] + real(a.b) * qd[k];
        }
        st4(a.G + off, gn);
        double q[4];
        if constexpr (Tl::KEEP_Q) {
          ld4(&in.Q[m * 4], q);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) q[k] = double(s.Q[k * VS + o]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = q[k] + a.c * double(gn[k]);
        st4(a.Q + off, q);
        check_state(a.health, a.health_host, q[0], q[1], q[2], q[3], e0 + le);
#pragma unroll
        for (int k = 0; k < 4; ++k) s.Q[k * VS + o] = real(q[k]);
      }
    }

    // F
    if (a.update) {
      __syncthreads();
      real* T_out = a.T_out + size_t(e0) * FT * 4;
      if (IP && VISC && a.fuse)   // the side tile is free since the lift
        gradient_traces<P, AFFINE>(s, op, in.vg, T_out, a.GT_out + size_t(e0) * FT * 8, n_act, tid);
      else
        tile_traces<P, 4, Tl>(s.Q, op.lb0, op.lb1, T_out, n_act, tid);
      if constexpr (IP && AV) {
        if (sense) {
          __syncthreads();
          group_sensor<P, EPB, T, real>(a.sensor, ph, op.Vinv, s.Q, s.Fc, VS, s.sens, s_w, n_act, tid, nullptr, flat_g,
                                        [&](int le, double, double, bool, double g) {
                                          a.mu_next[e0 + le] = a.av_el[2 * size_t(e0 + le)] * g;
                                        });
        }
      }
    }
    b ^= 1;
    slot = next_slot;
  }
  if (a.resid) {
    __syncthreads();
    if (tid < 4) {
      unsigned long long m = 0ull;
      for (int w = 0; w < T / 32; ++w) m = s.mx[tid][w] > m ? s.mx[tid][w] : m;
      put_partial(a.resid, tid, __longlong_as_double((long long)m));
    }
  }
}

}  // namespace hg
