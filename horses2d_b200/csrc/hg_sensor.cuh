// hg_sensor.cuh -- element shock sensors that set the artificial viscosity (device code).
//
// Three indicators feed the same viscosity law mu_e = Ceps sqrt(Volume)/(N+1) G (the law of
// JumpsBasedElementViscosity, Approximation/DGArtificialDissipation.f90:322-336):
//   jumps    the reference's interface-jumps indicator (jumps_kernel, hg_ns.cuh);
//   modal    modal decay (Persson-Peraire): s = max over rho, p of log10(E_N / E), E the energy of
//            the element's orthonormal-Legendre modal coefficients and E_N that of the modes whose
//            higher index is N; G = ramp(s; s0, kappa), the same sine ramp as the jumps indicator;
//   learned  an MLP 16 -> 32 -> 32 -> 1 (tanh hidden layers, sigmoid output) on 16 modal features
//            (for rho and p: log10 of the energy fraction in modal index k = 0..3 along xi and along
//            eta, higher indices folded into 3, floored at 1e-10); G = the sigmoid output y mapped
//            to max(0, (y - c) / (1 - c)), c = LEARNED_CUT (an exact zero below 5 % of the maximum
//            viscosity, as the modal ramp has below s0 - kappa: elements without viscosity skip the
//            dissipation's gradient work), or the modal G when a feature lies outside the box seen in
//            training (out-of-distribution fallback).
// No reference counterpart exists for modal and learned.
#pragma once
#include "hg_physics.cuh"

namespace hg {

enum { SENSOR_JUMPS = 0, SENSOR_MODAL = 1, SENSOR_LEARNED = 2 };
constexpr int MLP_IN = 16, MLP_H = 32;
constexpr int MLP_W1 = 0, MLP_B1 = MLP_W1 + MLP_H * MLP_IN, MLP_W2 = MLP_B1 + MLP_H, MLP_B2 = MLP_W2 + MLP_H * MLP_H,
              MLP_W3 = MLP_B2 + MLP_H, MLP_B3 = MLP_W3 + MLP_H, MLP_PARAMS = MLP_B3 + 1;

struct SensorArgs {
  int kind;            // SENSOR_*
  double s0, kappa;    // modal ramp centre and half width
  const float* mlp;    // [MLP_PARAMS] W1^T[16][32] b1 W2^T[32][32] b2 W3[32] b3 (hidden unit fastest)
  const float* lo;     // [16] feature box of the training set (with margin)
  const float* hi;     // [16]
};

// Scratch row of one warp (reals): the energies per modal index of rho and p along xi and eta (4P), the 16
// features and the first hidden layer (as floats); the latter two start at multiples of 16 bytes and are read
// with 16-byte loads.
__host__ __device__ constexpr int sr_ft(int P) { return 4 * P; }
__host__ __device__ constexpr int sr_h(int P) { return sr_ft(P) + MLP_IN; }
__host__ __device__ constexpr int sensor_scratch(int P) { return sr_h(P) + MLP_H; }

__device__ __forceinline__ double sensor_ramp(double s, double s0, double k) {
  if (s < s0 - k) return 0.0;
  if (s < s0 + k) return 0.5 * sin(0.5 * 3.141592653589793238462643 * (s - s0) / k) + 0.5;
  return 1.0;
}

__device__ __forceinline__ float mlp_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }
constexpr float LEARNED_CUT = 0.05f;
__device__ __forceinline__ float learned_g(float y) { return y > LEARNED_CUT ? (y - LEARNED_CUT) / (1.0f - LEARNED_CUT) : 0.0f; }

// smallest energy fraction a feature resolves (log10 floor -10: FP32 round-off, ~1e-14, stays below)
constexpr double SENSOR_FLOOR = 1e-10;
template <typename real> __device__ __forceinline__ real log10_r(real x);
template <> __device__ __forceinline__ double log10_r(double x) { return log10(x); }
template <> __device__ __forceinline__ float log10_r(float x) { return log10f(x); }
template <typename real> __device__ __forceinline__ real fmax_r(real a, real b) { return a > b ? a : b; }

// The network's weights into shared memory (16-byte aligned) as asynchronous copies: 16-byte chunks,
// the odd last float as a 4-byte copy.  They are visible after each thread's cp.async wait and a barrier.
__device__ __forceinline__ void sensor_weights_async(float* s_w, const float* g, int t, int nt) {
  constexpr int C16 = MLP_PARAMS / 4;
  const unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(s_w));
  for (int c = t; c < C16; c += nt)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(base + 16u * unsigned(c)), "l"(g + 4 * c)
                 : "memory");
  if (t == 0)
    for (int d = 4 * C16; d < MLP_PARAMS; ++d)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(base + 4u * unsigned(d)), "l"(g + d) : "memory");
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// 16 consecutive reals of a 16-byte aligned shared row as floats
__device__ __forceinline__ void load16(const float* r, float* f) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4 v = reinterpret_cast<const float4*>(r)[k];
    f[4 * k] = v.x; f[4 * k + 1] = v.y; f[4 * k + 2] = v.z; f[4 * k + 3] = v.w;
  }
}
__device__ __forceinline__ void load16(const double* r, float* f) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double2 v = reinterpret_cast<const double2*>(r)[k];
    f[2 * k] = float(v.x); f[2 * k + 1] = float(v.y);
  }
}

// G of the constant state as a warp has it: every constant-state element has the same features, so its network
// runs once per warp (the same inputs through the same code: the same bits).
struct FlatG {
  float g = 0.0f;
  bool known = false;
};

// Modal indicator and (if asked) the learned one for the n_act elements of a CTA's group; all T threads take
// part.  Q: the group's state tile, U: two variables' worth of free tile (variable stride VS, rows of PO
// nodes), scr: a scratch row per warp, s_w: the network's weights, complete and visible.
// emit(element, modal G, learned G, out-of-box verdict, G in use) runs in one lane per element.
//
// The modal transform runs as the stage kernels' contractions do, one thread per (variable, line) with Vinv
// in the constant bank.  From the modal energies on a warp works on an element by itself, without a barrier of
// the CTA: a lane per modal index, then a lane per feature (the out-of-box and constant-state tests are
// ballots), then a lane per hidden unit: the features and the first hidden layer are broadcast from the warp's
// scratch row, the 32-input sums of the second layer run as four interleaved partial sums, and the output unit
// is a warp shuffle tree.
template <int P, int EPB, int T, typename real, typename Emit>
__device__ __forceinline__ void group_sensor(const SensorArgs& sa, const Phys<real>& ph, const real* Vinv,
                                             const real* Q, real* U, int VS, real* scr, const float* s_w, int n_act,
                                             int tid, float* feat_out, FlatG& flat_g, Emit emit) {
  constexpr int N = P - 1, NP = P * P, PO = P | 1;
  const bool learned = sa.kind == SENSOR_LEARNED;
  for (int m = tid; m < n_act * NP; m += T) {
    const int o = (m / P) * PO + m % P;   // rows of all elements follow one another
    const real r = Q[o], ru = Q[VS + o], rv = Q[2 * VS + o], rE = Q[3 * VS + o];
    U[o] = r;
    U[VS + o] = ph.gm1 * (rE - real(0.5) * (ru * ru + rv * rv) / r);
  }
  const auto line = [&](real* u, const int st, const bool square) {
    real in[P], out[P];
#pragma unroll
    for (int l = 0; l < P; ++l) in[l] = u[l * st];
#pragma unroll
    for (int k = 0; k < P; ++k) {
      real c = real(0);
#pragma unroll
      for (int l = 0; l < P; ++l) c += Vinv[k * P + l] * in[l];
      out[k] = square ? c * c : c;
    }
#pragma unroll
    for (int l = 0; l < P; ++l) u[l * st] = out[l];
  };
  __syncthreads();
  for (int x = tid; x < 2 * P * EPB; x += T)
    if ((x / P) % EPB < n_act) line(U + (x / (P * EPB)) * VS + (x % (P * EPB)) * PO, 1, false);
  __syncthreads();
  for (int x = tid; x < 2 * P * EPB; x += T)   // the coefficients' squares: modal energies
    if ((x / P) % EPB < n_act) line(U + (x / (P * EPB)) * VS + ((x / P) % EPB) * P * PO + x % P, PO, true);
  __syncthreads();
  static_assert(MLP_H == 32, "one lane per hidden unit");
  const int lane = tid & 31;
  real* r = scr + (tid >> 5) * sensor_scratch(P);
  const real floor_f = log10_r(real(SENSOR_FLOOR));
  for (int le = tid >> 5; le < n_act; le += T / 32) {
    const real* c2 = U + le * P * PO;   // modal energies of rho; of p: + VS
    // energies per modal index: t = (v * 2 + dir) * P + k sums over the other index
    for (int t = lane; t < 4 * P; t += 32) {
      const int v = t / (2 * P), dir = (t / P) & 1, k = t % P;
      real a = real(0);
#pragma unroll
      for (int j = 0; j < P; ++j) a += c2[v * VS + (dir == 0 ? j * PO + k : k * PO + j)];
      r[t] = a;
    }
    __syncwarp();
    // lanes q < 16: features; lanes 16, 17: the modal-decay indicators of rho and p
    const int q = lane & 15, v = lane < MLP_IN ? q >> 3 : lane & 1;
    const real* sv = r + 2 * v * P;   // along xi: sv[m]; along eta: sv[P + n]
    real E = real(0), part = real(0), f = real(0);
#pragma unroll
    for (int m = 0; m < P; ++m) E += sv[m];
    bool ood = false, flat = true;
    if (lane < MLP_IN) {
      const int dir = (q >> 2) & 1, k = q & 3;
      if (k < 3) {
        if (k < P) part = sv[dir * P + k];
      } else {
        for (int m = 3; m < P; ++m) part += sv[dir * P + m];
      }
      // x / x is 1 exactly (also where the build's FP32 division is the approximate one)
      const real frac = E > real(0) ? (part == E ? real(1) : part / E) : real(0);
      f = log10_r(fmax_r(frac, real(SENSOR_FLOOR)));
      r[sr_ft(P) + q] = f;
      if (feat_out) feat_out[size_t(le) * MLP_IN + q] = float(f);
      ood = sa.lo && (float(f) < __ldg(sa.lo + q) || float(f) > __ldg(sa.hi + q));
      flat = f == ((q & 3) == 0 ? real(0) : floor_f);
    } else if (lane < MLP_IN + 2) {
      // the modes whose higher index is N: row N along eta plus column N below it
      const real* u = c2 + v * VS;
#pragma unroll
      for (int m = 0; m < P; ++m) part += u[N * PO + m];
#pragma unroll
      for (int n = 0; n < N; ++n) part += u[n * PO + N];
      f = (E > real(0) && part > real(0)) ? log10_r(part / E) : real(-1e30);
    }
    ood = __any_sync(0xffffffffu, ood);
    flat = __all_sync(0xffffffffu, flat);   // constant-state element: every energy in the mean mode
    const real p0 = __shfl_sync(0xffffffffu, f, MLP_IN), p1 = __shfl_sync(0xffffffffu, f, MLP_IN + 1);
    __syncwarp();
    float gl = 0.0f;
    if (learned && flat && flat_g.known) {
      gl = flat_g.g;
    } else if (learned) {
      float x[MLP_IN];
      load16(r + sr_ft(P), x);
      float z = s_w[MLP_B1 + lane];
#pragma unroll
      for (int k = 0; k < MLP_IN; ++k) z += s_w[MLP_W1 + k * MLP_H + lane] * x[k];
      float* h1 = reinterpret_cast<float*>(r + sr_h(P));
      h1[lane] = tanhf(z);
      __syncwarp();
      float zp[4] = {s_w[MLP_B2 + lane], 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int q4 = 0; q4 < MLP_H / 4; ++q4) {
        const float4 h = reinterpret_cast<const float4*>(h1)[q4];
        zp[0] += s_w[MLP_W2 + (4 * q4 + 0) * MLP_H + lane] * h.x;
        zp[1] += s_w[MLP_W2 + (4 * q4 + 1) * MLP_H + lane] * h.y;
        zp[2] += s_w[MLP_W2 + (4 * q4 + 2) * MLP_H + lane] * h.z;
        zp[3] += s_w[MLP_W2 + (4 * q4 + 3) * MLP_H + lane] * h.w;
      }
      const float h = tanhf((zp[0] + zp[1]) + (zp[2] + zp[3]));
      float y = s_w[MLP_W3 + lane] * h;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) y += __shfl_xor_sync(0xffffffffu, y, off);
      gl = learned_g(mlp_sigmoid(y + s_w[MLP_B3]));
      if (flat) { flat_g.g = gl; flat_g.known = true; }
    }
    if (lane == 0) {
      const double gm = sensor_ramp(double(p0 > p1 ? p0 : p1), sa.s0, sa.kappa);
      emit(le, gm, double(real(gl)), ood, learned && !ood ? double(real(gl)) : gm);
    }
    __syncwarp();
  }
}

}  // namespace hg
