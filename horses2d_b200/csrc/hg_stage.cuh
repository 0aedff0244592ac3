// hg_stage.cuh -- the fused DGSEM stage kernel (Euler) for sm_100a.
//
// One launch = one Runge-Kutta stage (or one bare time derivative) over all elements, in place.  CTAs
// are persistent: each walks over groups of EPB consecutive elements, and while it works on one group
// the inputs of its next one travel into the other half of a double buffer (state, RK register, own
// traces, metrics and the side table of the group after it as bulk copies on an mbarrier; the
// neighbours' traces as 16-byte asynchronous copies, because their addresses come from the side table).
// Per group, with a barrier between the phases:
//   A  face nodes and volume nodes as one list of items over all threads (whole warps of each kind):
//      a face node takes its own and the neighbour's trace and solves the Riemann problem / boundary
//      state, x dS (ComputeRiemannSolver_*, DGSpatialDiscretizationMethods.f90:545-1511; projections
//      types 1-2, Mesh/QuadElement_EdgeProcedures.incf:749-1206); a volume node forms its contravariant
//      fluxes (Scalar_StdVolumeGreen, Approximation/DGWeakIntegrals.f90:111-181);
//   B  one thread per (variable, line of nodes, direction): the line's P fluxes in registers, contracted
//      with hatD and lifted with lbw at its two ends (Scalar_StdFace, DGWeakIntegrals.f90:183-266), back
//      in place; in float one thread per (variable, row of nodes) for both directions (row_sums);
//   C  per node: division by J (computeQDot :226-233), low-storage RK update G = a G + b QDot,
//      Q += c G (DGTimeIntegrator.f90:282-365); Gauss-Lobatto: the boundary nodes are the new traces;
//   D  Legendre-Gauss: one thread per (variable, line): the traces of the new state at the line's ends
//      (interpolateSolutionToBoundaries, :1520-1574) for the next launch (ping-pong buffer).
// What bounds it: latency, with 15 warps per SM in double (registers and shared memory), then the shared-memory
// pipe (58 %); in float instruction issue (70 %).  One thread per node with its loads where they were used (the form
// before) spent half of its warps' cycles on global loads and filled 62 % of the lanes of its face phase; measured
// with 512 x 512 elements, N = 4, Gauss-Lobatto, FP64: 0.81 ms a stage then, 0.33 ms now (1.17 GB of state, register
// and trace traffic: 3.6 TB/s); 16 x 16 elements: 20.5 -> 12.3 us a step.  Fewer or more elements to a group (4, 6)
// and 96 to 256 threads came out between equal and 25 % slower at N = 4.
// The Riemann flux of an interior face is evaluated by both of its elements with identical arguments
// (LEFT trace, RIGHT trace, LEFT's normal), so both see the same value and the face needs no separate
// launch or flux buffer.
//
// The nodal operators are kernel parameters: with the line loops unrolled their entries are constant-bank
// operands of the multiply-adds, so a line costs P shared loads and P stores for P^2 multiply-adds (one
// thread per node needs 2P loads for 2P multiply-adds).  Shared tiles are variable-major with rows of
// an odd number of nodes (PO) and a variable stride VS = 4 (8 in float) modulo the bank count: lanes that
// walk along rows, columns or (variable, line) pairs all touch different banks.
#pragma once
#include "hg_physics.cuh"
#include "hg_bc.cuh"

namespace hg {

// side kinds; SIDE_FLUX: a p-nonconforming or subdivided edge, whose lifted flux (projected to this
// element's side nodes, dS and sign applied) the mortar kernel has written to the NF buffer
enum { SIDE_LEFT = 0, SIDE_RIGHT = 1, SIDE_STATE = 2, SIDE_WALL = 3, SIDE_FLUX = 4 };
constexpr int SIDE_REVERSED = 16;

template <typename real>
struct StageArgs {
  int n_el;
  const int4* side;        // [n_el*4] {neighbour trace slot, flags, zone, per-node state row or -1}
  const real* side_geo;    // [n_el*4][P][3] (or [n_el*4][3] affine)  nx, ny, dS in this element's side order
  const real* vol_geo;     // element records of vol_geo_stride reals (below)
  const Zone* zones;
  const double* bq;        // per-node Dirichlet states [rows][P][4] (sides whose side.w >= 0)
  const real* FX;          // exact-solver face fluxes [n_el*4][P][4] of this stage (RIEMANN_EXACT faces)
  const real* NF;          // mortar fluxes [slots][P][4] of SIDE_FLUX sides (slot = side.x)
  double* Q;               // [n_el][P*P][4]
  real* G;                 // [n_el][P*P][4]
  const real* T_in;        // [n_el*4][P][4]
  real* T_out;
  double* QDot;            // optional output (time derivative only)
  double* resid;           // optional per-CTA max |QDot| per variable (put_partial)
  int* health;             // device health word {bits, element} (check_state), may be null
  int* health_host;        // mapped host flag set beside it, may be null
  int polls;               // limit of a wait for copies (mbar_wait)
  double a, b, c;          // G = a G + b QDot ; Q += c G
  int first;               // a == 0: do not read G
  int update;              // 1: RK update, 0: only QDot (and traces of the unchanged Q)
  int riemann;
  PhysConst pc;
};

// Bits of the health word (check_state; COPY: copies_failed).
enum { HEALTH_NONFINITE = 1, HEALTH_DENSITY = 2, HEALTH_PRESSURE = 4, HEALTH_COPY = 8 };

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int cmin(int a, int b) { return a < b ? a : b; }

// Metrics record of an element, a multiple of 16 bytes long in either precision.  Curved: [P*P][5] with
// Ja00 Ja01 Ja10 Ja11 1/J per node.  Affine (AFFINE_REC reals): those five, three unused, then nx ny dS of
// the four sides.
constexpr int AFFINE_REC = 20;
__host__ __device__ constexpr int vol_geo_stride(int P, bool affine) { return affine ? AFFINE_REC : (5 * P * P + 3) / 4 * 4; }

// Nodal operators of one order, passed by value (constant bank).
template <int P, typename real>
struct StageOps {
  real hatD[P * P], lb0[P], lb1[P], lbw0[P], lbw1[P];
};

// Elements per group: tiling variant 0 (large groups) and variant 1 (small groups: more CTAs in flight on
// small meshes); hg_autotune times both on the resident state and keeps the faster.
__host__ __device__ constexpr int epb_for(int P) { return P == 2 ? 16 : P <= 5 ? 8 : P <= 8 ? 4 : P <= 10 ? 2 : 1; }
__host__ __device__ constexpr int epb_small_for(int P) { return P <= 3 ? 4 : P <= 5 ? 2 : 1; }
__host__ __device__ constexpr int epb_stage(int P, int variant) { return variant ? epb_small_for(P) : epb_for(P); }
__host__ __device__ constexpr int block_of(int P, int EPB) { return ((P * P * EPB + 31) / 32) * 32; }
__host__ __device__ constexpr int block_for(int P) { return block_of(P, epb_for(P)); }
// Threads of a stage CTA: the group's face nodes in whole warps (the longest task, one round); small
// groups also hold a thread per volume node, so that phase A is a single round.
__host__ __device__ constexpr int stage_threads(int P, int variant) {
  const int nf = (4 * P * epb_stage(P, variant) + 31) / 32 * 32;
  return variant ? nf + block_of(P, epb_stage(P, variant)) : nf;
}

// Four consecutive values of a record that starts at a multiple of 4 values from a cudaMalloc'd base
// (16-byte aligned in float, 32-byte in double): one 128-bit access in float, two in double.
__device__ __forceinline__ void ld4(const float* p, float* o) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void ld4(const double* p, double* o) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
__device__ __forceinline__ void st4(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st4(double* p, const double* v) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

// W = 2 or 4 of them.
template <typename real, int W>
__device__ __forceinline__ void ld_w(const real* p, real (&o)[W]) {
  if constexpr (W == 4) {
    ld4(p, o);
  } else {
    const double2 v = *reinterpret_cast<const double2*>(p);
    o[0] = v.x; o[1] = v.y;
  }
}
template <typename real, int W>
__device__ __forceinline__ void st_w(real* p, const real (&v)[W]) {
  if constexpr (W == 4) st4(p, v);
  else *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}

// One value from global into shared memory as an asynchronous copy (4 or 8 bytes); the issuing thread
// sees it after cp_async_wait_all.
__device__ __forceinline__ void cp_async_real(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_real(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Four consecutive values from global into shared memory, 16 bytes at a time.
__device__ __forceinline__ void cp_async_4(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(dst))),
               "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_4(double* dst, const double* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + 16u), "l"(src + 2) : "memory");
}

// Bulk copies (both addresses and the size multiples of 16 bytes) that complete on an mbarrier.
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(bar))), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(dst))), "l"(src), "r"(bytes),
               "r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))) : "memory");
}
// Programmatic dependent launch: a kernel launched behind another one on the stream may start while that one
// still runs; what it reads or overwrites of the other's data comes after grid_wait.  A stage takes 4 us on a small
// mesh, a third of it between the last store of one kernel and the first load of the next.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Waits for the phase; gives up after a bounded number of polls (each suspends the thread for a while) and
// reports false.  The CTA's threads then leave together (copies_failed), before any of them reads what the copies
// should have brought: a copy that never lands ends the launch with a health bit instead of hanging it.
constexpr int COPY_POLLS = 1 << 20;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int polls) {
  const unsigned b = static_cast<unsigned>(__cvta_generic_to_shared(bar));
  for (int n = 0; n < polls; ++n) {
    unsigned done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(b), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}

// Of the CTA's threads that gave up waiting (any: uniform): the health bit, and a last bounded wait for the copies
// still in flight, which must not outlive the CTA's shared memory.
__device__ __forceinline__ void copies_failed(int* health, int* health_host, uint64_t* bar, unsigned parity) {
  if (health) atomicOr(health, HEALTH_COPY);
  if (health_host) *reinterpret_cast<volatile int*>(health_host) = 1;
  mbar_wait(bar, parity, COPY_POLLS);
}

// max that keeps NaN (a residual that is NaN must stay visible)
__device__ __forceinline__ double nanmax(double m, double v) { return (v > m || v != v) ? v : m; }

// Residual partials of a launch: {CTAs, -, -, -}, then a row of 4 maxima per CTA.  The count stands beside them because
// launches of one kernel differ in their CTAs (the network's weights take shared memory on the last stage of a step) and
// a replayed graph passes no host code that could note it.
__device__ __forceinline__ void put_partial(double* resid, int k, double m) {
  resid[4 + size_t(blockIdx.x) * 4 + k] = m;
  if (blockIdx.x == 0 && k == 0) resid[0] = double(gridDim.x);
}

// Per-CTA residual maxima from each lane's W variables (W = 2: even lanes 0 and 1, odd lanes 2 and 3); scratch holds
// W T values.
template <int W, int T>
__device__ __forceinline__ void residual_partial(const double* mx, double* scratch, double* resid, int tid) {
  __syncthreads();
#pragma unroll
  for (int k = 0; k < W; ++k) scratch[W * tid + k] = mx[k];
  __syncthreads();
  if (tid < 4) {
    double m = 0.0;
    for (int t = tid; t < W * T; t += 4) m = nanmax(m, scratch[t]);
    put_partial(resid, tid, m);
  }
}

// Max over the warp of non-negative values, as bits (ordered as the values are; NaN above all): two 32-bit
// reductions.
__device__ __forceinline__ unsigned long long warp_max_bits(double v) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(v);
  const unsigned hi = unsigned(u >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? unsigned(u) : 0u);
  return (static_cast<unsigned long long>(mh) << 32) | ml;
}

// Health of an updated node state.  The reference stops with "The simulation has crashed" when Q holds
// a NaN (DGTimeIntegrator.f90:224-233); here every RK update checks its node: bit 1 a non-finite value,
// bit 2 rho <= 0, bit 4 p <= 0 (tested as rho (rho E) - |rho u|^2 / 2 = rho p / (gamma - 1) <= 0, no
// division).  health = {bits, an offending element (the first to arrive)}; the mapped host flag tells
// the host without a synchronisation that the word is no longer clean.
__device__ __forceinline__ void check_state(int* health, int* health_host, double r, double ru, double rv,
                                            double rE, int e) {
  const bool finite = fabs(r) + fabs(ru) + fabs(rv) + fabs(rE) < 1.0e300;
  const double k = r * rE - 0.5 * (ru * ru + rv * rv);
  if (finite && r > 0.0 && k > 0.0) return;
  const int bits = !finite ? HEALTH_NONFINITE : (r > 0.0 ? HEALTH_PRESSURE : HEALTH_DENSITY);
  if (health) {
    atomicOr(health, bits);
    atomicCAS(health + 1, -1, e);
  }
  if (health_host) *reinterpret_cast<volatile int*>(health_host) = 1;
}

__host__ __device__ constexpr int face_node(int P, int side, int l, int kk) {
  return (side == 0 || side == 2) ? (l * P + kk) : (kk * P + l);
}

// In float (this kernel, and BR1's in hg_ns.cuh) a node's contraction and lift are one sum in one order: for l = 0 .. N
// the xi term, then the eta term, then the bottom, right, top and left sides.  A 32-bit time derivative of a smooth state
// is a difference of sums a thousand times as large, so another order gives it other digits from the fourth on (the two
// directions summed apart: 3e-4 in the 2-norm at N = 8, against 5e-13 in double, whose kernels do that: one line of one
// direction per thread).  The lanes of a row of nodes hold different rows j of hatD: a copy in shared memory, transposed.
// Against a line per thread: 128 vortex boxes 2.41 -> 2.54 ms for six steps.
template <int P, typename real, bool USED = sizeof(real) == 4>
struct SumOps {
  static constexpr bool ON = USED;
  real hatT[ON ? P * P : 1], lbw0[ON ? P : 1], lbw1[ON ? P : 1];
  template <typename Ops>
  __device__ __forceinline__ void fill(const Ops& op, int tid, int T) {
    if constexpr (ON) {
      for (int k = tid; k < P * P; k += T) hatT[(k % P) * P + k / P] = op.hatD[k];
      for (int k = tid; k < P; k += T) { lbw0[k] = op.lbw0[k]; lbw1[k] = op.lbw1[k]; }
    }
  }
};
// The sums of row j of an element, of one variable: Fc the row of xi fluxes, Gc the element's tile of eta fluxes (rows of
// PO nodes); face(side, k) the side's flux at its node k.  out replaces the row of xi fluxes.
template <int P, int PO, bool ENDS, typename Ops, typename real, typename Face>
__device__ __forceinline__ void row_sums(const Ops& op, const SumOps<P, real, true>& so, const real* Fc, const real* Gc, int j,
                                         Face face, real (&out)[P]) {
  real f[P], hj[P];
#pragma unroll
  for (int l = 0; l < P; ++l) {
    f[l] = Fc[l];
    hj[l] = so.hatT[l * P + j];
  }
  const real b0 = so.lbw0[j], b1 = so.lbw1[j], Fr = face(1, j), Fl = face(3, j);
#pragma unroll
  for (int i = 0; i < P; ++i) {
    real r = real(0);
#pragma unroll
    for (int l = 0; l < P; ++l) r = r + op.hatD[i * P + l] * f[l] + hj[l] * Gc[l * PO + i];
    if (!ENDS || j == 0) r = r - face(0, i) * b0;
    if (!ENDS || i == P - 1) r = r - Fr * op.lbw1[i];
    if (!ENDS || j == P - 1) r = r - face(2, i) * b1;
    if (!ENDS || i == 0) r = r - Fl * op.lbw0[i];
    out[i] = r;
  }
}
// Shared memory of a stage CTA.
template <int P, int V, typename real, bool AFFINE, bool LGL>
struct StageTiles {
  static constexpr int EPB = epb_stage(P, V), T = stage_threads(P, V);
  static constexpr int NP = P * P, FT = 4 * P, PO = P | 1, NN = EPB * NP, NF = EPB * FT, GS = vol_geo_stride(P, AFFINE);
  static constexpr int VM = sizeof(real) == 8 ? 16 : 32, V0 = EPB * P * PO;
  static constexpr int VS = V0 + (VM + VM / 4 - V0 % VM) % VM;   // = VM / 4 modulo VM
  struct In {                       // inputs of one group
    double Q[NN * 4];
    real G[NN * 4];
    real Tn[NF * 4];                // neighbours' traces (or mortar fluxes), in the task's node order
    real To[LGL ? 4 : NF * 4];      // own traces
    real vg[EPB * GS];
    real sg[AFFINE ? 4 : NF * 3];
  };
  alignas(16) In in[2];
  alignas(16) int4 side[3][EPB * 4];
  real Fc[4 * VS], Gc[4 * VS];      // contravariant fluxes, then their contractions; Fc then holds the new state
  real F[4 * NF];                   // face fluxes x dS (signed for a RIGHT side)
  SumOps<P, real> sum;
  uint64_t bar[2];
};

// AFFINE: metrics constant per element and normals / dS constant per side, as for parallelogram elements
// with straight edges.
// LGL: Gauss-Lobatto nodes, whose boundary interpolants are unit vectors (lb = e_0 / e_N): traces are
// node values and the lift touches only the line ends -- the same arithmetic as the dense form with its
// exact zeros left out.
template <int P, int V, typename real, bool AFFINE, bool LGL>
__global__ void __launch_bounds__(stage_threads(P, V))
    stage_kernel(const __grid_constant__ StageArgs<real> a, const __grid_constant__ StageOps<P, real> op) {
  using Tl = StageTiles<P, V, real, AFFINE, LGL>;
  constexpr int EPB = Tl::EPB, T = Tl::T, NP = Tl::NP, FT = Tl::FT, PO = Tl::PO, NF = Tl::NF, VS = Tl::VS, GS = Tl::GS;
  constexpr bool SUMS = SumOps<P, real>::ON;
  extern __shared__ __align__(16) unsigned char stage_smem[];
  Tl& s = *reinterpret_cast<Tl*>(stage_smem);
  const int tid = threadIdx.x;
  const int n_groups = (a.n_el + EPB - 1) / EPB;
  Phys<real> ph;
  ph.load(a.pc);

  const auto count = [&](int g) { return min(EPB, a.n_el - g * EPB); };
  // inputs of group g into half b, and the side table of the group after it (thread 0).  first: of the CTA's first
  // group, where the constant ones (tables, metrics) go ahead of the wait for the kernel before
  const auto issue_bulk = [&](int g, int b, bool first, int slot) {
    const int e0 = g * EPB, n = count(g), gn = g + gridDim.x;
    const bool rk = a.update && !a.first;
    typename Tl::In& in = s.in[b];
    const unsigned bq = n * NP * 32u, bg = rk ? n * NP * 4u * sizeof(real) : 0u, bt = LGL ? 0u : n * FT * 4u * sizeof(real);
    const unsigned bv = n * GS * unsigned(sizeof(real)), bs = AFFINE ? 0u : n * FT * 3u * sizeof(real);
    const unsigned b0 = first ? n * 64u : 0u, bn = gn < n_groups ? count(gn) * 64u : 0u;
    uint64_t* bar = &s.bar[b];
    mbar_expect(bar, bq + bg + bt + bv + bs + b0 + bn);
    if (b0) bulk_copy(s.side[slot], a.side + size_t(e0) * 4, b0, bar);
    bulk_copy(in.vg, a.vol_geo + size_t(e0) * GS, bv, bar);
    if (bs) bulk_copy(in.sg, a.side_geo + size_t(e0) * FT * 3, bs, bar);
    if (bn) bulk_copy(s.side[slot == 2 ? 0 : slot + 1], a.side + size_t(gn) * EPB * 4, bn, bar);
    if (first) grid_wait();
    bulk_copy(in.Q, a.Q + size_t(e0) * NP * 4, bq, bar);
    if (bt) bulk_copy(in.To, a.T_in + size_t(e0) * FT * 4, bt, bar);
    if (bg) bulk_copy(in.G, a.G + size_t(e0) * NP * 4, bg, bar);
  };
  // the neighbours' traces of group g into half b: a face task's copy is issued and read by one thread
  // (at0: the table entry of the thread's first task)
  const auto side_of = [&](const int4* side, int x) { return side[(x / FT) * 4 + (x % FT) / P]; };
  const auto issue_rows = [&](int g, int b, const int4* side, int4 at0) {
    const int n = count(g) * FT;
    for (int x = tid; x < n; x += T) {
      const int kk = x % P;
      const int4 sd = x == tid ? at0 : side_of(side, x);
      const int kind = sd.y & 15;
      if (kind == SIDE_LEFT || kind == SIDE_RIGHT)
        cp_async_4(&s.in[b].Tn[x * 4], a.T_in + (size_t(sd.x) * P + ((sd.y & SIDE_REVERSED) ? P - 1 - kk : kk)) * 4);
      else if (kind == SIDE_FLUX)
        cp_async_4(&s.in[b].Tn[x * 4], a.NF + (size_t(sd.x) * P + kk) * 4);
    }
    cp_async_commit();
  };

  s.sum.fill(op, tid, T);
  if (tid == 0) {
    mbar_init(&s.bar[0]);
    mbar_init(&s.bar[1]);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  const int4* side0 = a.side + size_t(blockIdx.x) * EPB * 4;
  const int4 at0 = tid < count(blockIdx.x) * FT ? side_of(side0, tid) : make_int4(0, 0, 0, 0);
  if (tid == 0) issue_bulk(blockIdx.x, 0, true, 0);
  else grid_wait();
  issue_rows(blockIdx.x, 0, side0, at0);
  constexpr int W = sizeof(real) == 8 ? 2 : 4;   // variables to a lane in phase C
  double mx[W] = {};                            // max |QDot| of this lane's variables
  __syncthreads();   // the barriers are initialised

  int b = 0, slot = 0;
  unsigned phase = 0u;
  for (int g = blockIdx.x; g < n_groups; g += gridDim.x) {
    const int e0 = g * EPB, n_act = count(g);
    const bool late = !mbar_wait(&s.bar[b], (phase >> b) & 1u, a.polls);
    cp_async_wait_all();
    // (the barrier: every thread is done with the previous group, its half and the work tiles are free)
    if (__syncthreads_or(late)) {
      if (tid == 0) copies_failed(a.health, a.health_host, &s.bar[b], (phase >> b) & 1u);
      return;
    }
    phase ^= 1u << b;
    const int next_slot = slot == 2 ? 0 : slot + 1;
    if (g + int(gridDim.x) < n_groups) {
      if (tid == 0) issue_bulk(g + gridDim.x, b ^ 1, false, next_slot);
      issue_rows(g + gridDim.x, b ^ 1, s.side[next_slot], tid < count(g + gridDim.x) * FT ? side_of(s.side[next_slot], tid) : at0);
    } else {
      grid_launch_next();   // the CTA's last group
    }
    const typename Tl::In& in = s.in[b];
    const int4* side = s.side[slot];

    // A: face fluxes and contravariant volume fluxes
    constexpr int NFR = (NF + 31) / 32 * 32;
    for (int x = tid; x < NFR + Tl::NN; x += T) {
      if (x < NFR) {
        const int le = x / FT, t = x % FT, sd_ = t / P, kk = t % P;
        if (x >= NF || le >= n_act) continue;
        const int4 sd = side[le * 4 + sd_];
        const int kind = sd.y & 15;
        real qn[4], F[4];
        if (kind == SIDE_LEFT || kind == SIDE_RIGHT || kind == SIDE_FLUX) ld4(&in.Tn[x * 4], qn);
        if (kind == SIDE_FLUX) {
#pragma unroll
          for (int k = 0; k < 4; ++k) s.F[k * NF + x] = qn[k];
          continue;
        }
        real qo[4];
        if (LGL) {
          double qd[4];
          ld4(&in.Q[(le * NP + face_node(P, sd_, (sd_ == 0 || sd_ == 3) ? 0 : P - 1, kk)) * 4], qd);
#pragma unroll
          for (int k = 0; k < 4; ++k) qo[k] = real(qd[k]);
        } else {
          ld4(&in.To[x * 4], qo);
        }
        const real* g3 = AFFINE ? &in.vg[le * GS + 8 + sd_ * 3] : &in.sg[x * 3];
        const real nx = g3[0], ny = g3[1], dS = g3[2];
        if (kind == SIDE_WALL) {
          euler_wall_flux(ph, qo, nx, ny, dS, F);
        } else {
          int solver = a.riemann;
          if (kind == SIDE_STATE) {
            const Zone& z = a.zones[sd.z];
            real us[4];
            bc_states(ph, z, qo, nx, ny, qn, us, sd.w >= 0 ? a.bq + (size_t(sd.w) * P + kk) * 4 : nullptr);
            if (z.riemann >= 0) solver = z.riemann;
          } else if (sd.z >= 0) {
            const int zr = a.zones[sd.z].riemann;
            if (zr >= 0) solver = zr;
          }
          const bool right = kind == SIDE_RIGHT;
          real qL[4], qR[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) { qL[k] = right ? qn[k] : qo[k]; qR[k] = right ? qo[k] : qn[k]; }
          face_riemann(solver, ph, qL, qR, nx, ny, a.FX, size_t(e0) * FT + x, F);
          const real sg = right ? -dS : dS;
#pragma unroll
          for (int k = 0; k < 4; ++k) F[k] *= sg;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) s.F[k * NF + x] = F[k];
      } else {
        const int m = x - NFR, le = m / NP, node = m % NP;
        if (le >= n_act) continue;
        double qd[4];
        ld4(&in.Q[m * 4], qd);
        const real q[4] = {real(qd[0]), real(qd[1]), real(qd[2]), real(qd[3])};
        const real* gp = AFFINE ? &in.vg[le * GS] : &in.vg[le * GS + node * 5];
        const real Ja00 = gp[0], Ja01 = gp[1], Ja10 = gp[2], Ja11 = gp[3];
        real f[4], gg[4];
        volume_flux(ph, q, f, gg);
        const int o = (le * P + node / P) * PO + node % P;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          s.Fc[k * VS + o] = f[k] * Ja00 + gg[k] * Ja10;   // F Ja(1,IX) + G Ja(2,IX)
          s.Gc[k * VS + o] = f[k] * Ja01 + gg[k] * Ja11;   // F Ja(1,IY) + G Ja(2,IY)
        }
      }
    }
    __syncthreads();

    // B: contraction and lift, one line of one variable per thread: rows of Fc between the left and right
    // sides, columns of Gc between the bottom and top ones
    const auto line = [&](real* U, const int st, const real F0, const real F1) {
      real in_[P], out[P];
#pragma unroll
      for (int l = 0; l < P; ++l) in_[l] = U[l * st];
#pragma unroll
      for (int i = 0; i < P; ++i) {
        real r = op.hatD[i * P] * in_[0];
#pragma unroll
        for (int l = 1; l < P; ++l) r += op.hatD[i * P + l] * in_[l];
        if (!LGL || i == 0) r -= F0 * op.lbw0[i];
        if (!LGL || i == P - 1) r -= F1 * op.lbw1[i];
        out[i] = r;
      }
#pragma unroll
      for (int l = 0; l < P; ++l) U[l * st] = out[l];
    };
    for (int x = tid; x < NF; x += T) {   // x = (variable, element, line)
      const int v = x / (P * EPB), le = (x / P) % EPB, m = x % P;
      if (le >= n_act) continue;
      const real* Fv = &s.F[v * NF + le * FT];
      real* Fc = &s.Fc[v * VS + (le * P + m) * PO];
      if constexpr (SUMS) {
        real r[P];
        row_sums<P, PO, LGL>(op, s.sum, Fc, &s.Gc[v * VS + le * P * PO], m, [&](int sd, int k) { return Fv[sd * P + k]; }, r);
#pragma unroll
        for (int l = 0; l < P; ++l) Fc[l] = r[l];
      } else {
        line(Fc, 1, Fv[3 * P + m], Fv[P + m]);
      }
    }
    if constexpr (!SUMS)
      for (int x = tid; x < NF; x += T) {
        const int v = x / (P * EPB), le = (x / P) % EPB, m = x % P;
        if (le >= n_act) continue;
        const real* Fv = &s.F[v * NF + le * FT];
        line(&s.Gc[v * VS + le * P * PO + m], PO, Fv[m], Fv[2 * P + m]);
      }
    __syncthreads();

    // C: time derivative and update, W variables of a node to a lane.  In double two lanes share a node: 16-byte
    // records side by side over the lanes, in shared memory as in HBM (16 x 16 elements 12 % less a step, orders 5
    // and 7 with mortars 5 %; in float, whose records are half as long, a lane per node is the faster one: 128 vortex
    // boxes 9 %)
    for (int x = tid; x < (4 / W * Tl::NN + 31) / 32 * 32; x += T) {
      const int m = x / (4 / W), h = x % (4 / W) * W;
      const bool on = m < n_act * NP;
      const int le = m / NP, node = m % NP, i = node % P, j = node / P, o = (m / P) * PO + node % P;
      const size_t off = (size_t(e0) * NP + m) * 4 + h;
      real qd[W] = {};
      if (on) {
        const real iJ = AFFINE ? in.vg[le * GS + 4] : in.vg[le * GS + node * 5 + 4];
#pragma unroll
        for (int k = 0; k < W; ++k)
          qd[k] = (SUMS ? s.Fc[(h + k) * VS + o] : s.Fc[(h + k) * VS + o] + s.Gc[(h + k) * VS + o]) * iJ;
        if (a.QDot) {
          double dq[W];
#pragma unroll
          for (int k = 0; k < W; ++k) dq[k] = double(qd[k]);
          st_w(a.QDot + off, dq);
        }
      }
      if (a.resid)
#pragma unroll
        for (int k = 0; k < W; ++k) mx[k] = nanmax(mx[k], fabs(double(qd[k])));
      if (a.update) {
        double q[W] = {};
        if (on) {
          real gn[W];
          if (a.first) {
#pragma unroll
            for (int k = 0; k < W; ++k) gn[k] = real(a.b) * qd[k];
          } else {
            ld_w(&in.G[m * 4 + h], gn);
#pragma unroll
            for (int k = 0; k < W; ++k) gn[k] = real(a.a) * gn[k] + real(a.b) * qd[k];
          }
          st_w(a.G + off, gn);
          ld_w(&in.Q[m * 4 + h], q);
#pragma unroll
          for (int k = 0; k < W; ++k) q[k] = q[k] + a.c * double(gn[k]);
          st_w(a.Q + off, q);
          real r[W];
#pragma unroll
          for (int k = 0; k < W; ++k) r[k] = real(q[k]);
          if (LGL) {
            real* tp = a.T_out + size_t(e0 + le) * FT * 4 + h;
            if (j == 0) st_w(tp + i * 4, r);
            if (i == P - 1) st_w(tp + (P + j) * 4, r);
            if (j == P - 1) st_w(tp + (2 * P + i) * 4, r);
            if (i == 0) st_w(tp + (3 * P + j) * 4, r);
          } else {
#pragma unroll
            for (int k = 0; k < W; ++k) s.Fc[(h + k) * VS + o] = r[k];
          }
        }
        if constexpr (W == 2) {   // the pair's other half, for the check of the whole state
          const double r0 = __shfl_xor_sync(0xffffffffu, q[0], 1), r1 = __shfl_xor_sync(0xffffffffu, q[1], 1);
          if (on && h == 0) check_state(a.health, a.health_host, q[0], q[1], r0, r1, e0 + le);
        } else {
          if (on) check_state(a.health, a.health_host, q[0], q[1], q[2], q[3], e0 + le);
        }
      }
    }

    // D: traces of the new state at both ends of every line; the variable runs fastest over the lanes, so
    // that four of them write one 4-value record
    if (!LGL && a.update) {
      __syncthreads();
      const auto ends = [&](const real* U, const int st, real* t0, real* t1) {
        real r0 = real(0), r1 = real(0);   // summed as trace_kernel does, bit for bit
#pragma unroll
        for (int l = 0; l < P; ++l) {
          const real u = U[l * st];
          r0 += op.lb0[l] * u;
          r1 += op.lb1[l] * u;
        }
        *t0 = r0;
        *t1 = r1;
      };
      for (int x = tid; x < n_act * FT; x += T) {   // x = (element, line, variable)
        const int v = x & 3, le = x / FT, m = (x >> 2) % P;
        real* tp = a.T_out + size_t(e0 + le) * FT * 4 + v;
        ends(&s.Fc[v * VS + (le * P + m) * PO], 1, tp + (3 * P + m) * 4, tp + (P + m) * 4);
        ends(&s.Fc[v * VS + le * P * PO + m], PO, tp + m * 4, tp + (2 * P + m) * 4);
      }
    }
    b ^= 1;
    slot = next_slot;
  }
  if (a.resid) residual_partial<W, T>(mx, reinterpret_cast<double*>(s.in), a.resid, tid);
  static_assert(sizeof(s.in) >= W * T * sizeof(double), "scratch of the residual maxima");
}

// Traces of the resident state (after hg_set_state).
// Summed in the order of the stage kernels, so that a state loaded from the host has the traces bit for bit that
// a stage left.  nodal: the Euler kernel's Gauss-Lobatto traces, the end nodes themselves.
template <int P, int EPB, typename real>
__global__ void __launch_bounds__(block_for(P)) trace_kernel(int n_el, const double* Q, const double* mats, real* T,
                                                             bool nodal) {
  constexpr int NP = P * P;
  constexpr int FT = 4 * P;
  __shared__ real s_lb[2 * P];
  __shared__ real s_Q[4][EPB][NP];
  const int flat = threadIdx.x;
  const int le = flat / NP, tid = flat - le * NP;
  for (int k = flat; k < 2 * P; k += blockDim.x) s_lb[k] = real(mats[NP + k]);
  const int e = blockIdx.x * EPB + le;
  const bool active = le < EPB && e < n_el;
  if (active)
#pragma unroll
    for (int k = 0; k < 4; ++k) s_Q[k][le][tid] = real(Q[(size_t(e) * NP + tid) * 4 + k]);
  __syncthreads();
  if (!active) return;
  for (int t = tid; t < FT; t += NP) {
    const int s = t / P, kk = t % P;
    const real* lbv = (s == 0 || s == 3) ? s_lb : s_lb + P;
    real tr[4] = {real(0), real(0), real(0), real(0)};
    if (nodal) {
#pragma unroll
      for (int k = 0; k < 4; ++k) tr[k] = s_Q[k][le][face_node(P, s, (s == 0 || s == 3) ? 0 : P - 1, kk)];
    } else {
      for (int l = 0; l < P; ++l)
#pragma unroll
        for (int k = 0; k < 4; ++k) tr[k] += s_Q[k][le][face_node(P, s, l, kk)] * lbv[l];
    }
    real* tp = T + ((size_t(e) * 4 + s) * P + kk) * 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) tp[k] = tr[k];
  }
}

// Max over the per-CTA residual partials (NaN kept).
static __global__ void residual_reduce_kernel(const double* resid, double* out) {
  const int nblocks = int(resid[0]);
  const double* part = resid + 4;
  __shared__ double s[4][256];
  double m[4] = {0.0, 0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < 4; ++k) m[k] = nanmax(m[k], part[size_t(b) * 4 + k]);
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k][threadIdx.x] = m[k];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
#pragma unroll
      for (int k = 0; k < 4; ++k) s[k][threadIdx.x] = nanmax(s[k][threadIdx.x], s[k][threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x < 4) out[threadIdx.x] = s[threadIdx.x][0];
}

}  // namespace hg
