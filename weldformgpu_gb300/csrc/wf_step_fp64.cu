// wf_step_fp64.cu — plain-FP64 form of the Fraser step.
//
// Compiled with -fmad=false, like the reference (--fmad=false,
// src/CMakeLists.txt:29): every multiply and add rounds separately, so with
// the same neighbour order the sums are bit-identical to the CPU oracle.
// Each kernel states the reference kernel(s) it replaces.
//
// What bounded these passes is the FP64 pipe (2 operations per clock and SM,
// 1/64 of the FP32 rate): ncu showed it 86-87 % busy in every pair pass at
// 170k particles, with 72 / 113 / 133 / 90 FP64 instructions a pair (density,
// stress, acceleration, heat), and memory and the integer pipes nearly idle.
// So
//   - whatever can be computed once is read back: the kernel factor GK and r^2
//     of each pair by the first pass that sees the positions, kept in two
//     arrays of the lists' layout for the other passes of the step (Work64);
//     m / rho and sigma / rho^2 once per particle;
//   - products, quotients and square roots run on the integer pipes (mul_int,
//     div_int, sqrt_int: wf_int64.cuh), additions on the FP64 pipe.
// 9 / 21 / 28 / 11 FP64 instructions a pair are left.  Times at 170k, in us,
// all on the FP64 pipe with nothing kept -> with the kept values -> now:
// density 1,066 -> 540 -> 247, stress 1,737 -> 1,070 -> 549, acceleration
// 2,178 -> 1,358 -> 577, heat 1,367 -> 1,354 -> 394 (it computes the geometry
// that the next step's density pass reads).  Stress and acceleration keep the
// FP64 pipe 79 % busy and the integer ALUs 47-51 %; density and heat the ALUs
// 61-63 % and FP64 64-71 %.
// Every value is rounded exactly as where it was computed on the FP64 pipe.
#include "wf_common.cuh"
#include "wf_heat.cuh"
#include "wf_int64.cuh"
#include "wf_lanes64.cuh"
#include "wf_mlp.cuh"
#include "wf_tensor.cuh"

namespace {

// |x| in [2^-kE, 2^kE], from the exponent bits (a comparison of doubles would
// run on the FP64 pipe); within: that, or zero
template <unsigned kE>
__device__ __forceinline__ bool in_range(double x) {
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - (1023u - kE) <= 2u * kE;
}
template <unsigned kE>
__device__ __forceinline__ bool within(double x) {
  return in_range<kE>(x) || (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) == 0u;
}

// Both forms of the pair terms: kInt on the integer pipes, else on the FP64 pipe.
template <bool kInt>
__device__ __forceinline__ double mul(double a, double b) {
  if constexpr (kInt) return mul_int(a, b);
  return a * b;
}
template <bool kInt>
__device__ __forceinline__ double quot(double a, double b) {
  if constexpr (kInt) return div_int(a, b);
  return a / b;
}
template <bool kInt>
__device__ __forceinline__ double root(double x) {
  if constexpr (kInt) return sqrt_int(x);
  return sqrt(x);
}
// A pair takes the integer form if it is tame: its loaded values are zero or
// within 2^+-kTame, so that every product and quotient of the pair, and every
// remainder of a sum in it, stays normal.  Any other pair takes the FP64 pipe.
constexpr unsigned kTame = 120;
// -0.5 x and 2 x: exact, so for zeros and tame values only the sign and exponent
// bits change (a select of the FP64 operation would still execute it: an
// eleventh of the stress pass's FP64 operations)
template <bool kInt>
__device__ __forceinline__ double neg_half(double x) {
  if constexpr (!kInt) return -0.5 * x;
  const int hi = __double2hiint(x);
  return __hiloint2double((hi ^ (int)0x80000000) - ((hi << 1) != 0 ? 0x00100000 : 0),
                          __double2loint(x));
}
template <bool kInt>
__device__ __forceinline__ double twice(double x) {
  if constexpr (!kInt) return x + x;
  const int hi = __double2hiint(x);
  return __hiloint2double(hi + ((hi << 1) != 0 ? 0x00100000 : 0), __double2loint(x));
}

// The cubic-spline gradient factor (Dim 3) with C = 1/(h^4 pi) hoisted: the
// reference recomputes C from h_ = (h_i + h_j)/2 = h for every pair
// (src/cuda/Functions.cu:76-88); with a uniform h the value is identical.  The
// division is shared by its two branches (so a warp whose lanes fall on both
// sides of q = 1 divides once) and the comparisons are on the bits of q >= 0.  q >= 2,
// infinite or NaN gives 0.
template <bool kInt>
__device__ __forceinline__ double spline64(double q, double h, double C) {
  const unsigned hi = (unsigned)__double2hiint(q);
  if (hi >= 0x40000000u) return 0.0;
  if ((hi | (unsigned)__double2loint(q)) == 0u) return C / h * (-3.0 + (9.0 / 2.0) * q);
  const bool in = hi < 0x3ff00000u;
  const double s = in ? q : 2.0 - q;
  const double c = mul<kInt>(mul<kInt>(in ? 9.0 / 4.0 : -3.0 / 4.0, s), s);
  const double d = in ? mul<kInt>(-3.0, q) + c : c;
  return mul<kInt>(quot<kInt>(C, mul<kInt>(q, h)), d);
}

// GK and RN(r r) of a pair from x_i - x_j
// (kIntSquares: with one lane the integer ALUs bound the passes that compute
// it, 67 % busy, and four of its products are better on the FP64 pipe: heat
// pass at 170k 427 -> 395 us; with eight lanes the other way, 114 -> 106 at
// 37k.)
template <bool kInt, bool kIntSquares = kInt>
__device__ __forceinline__ void pair_geometry(const StepParams& P, double xx, double xy, double xz,
                                              double& GK, double& r2) {
  const double rij = root<kInt>(mul<kIntSquares>(xx, xx) + mul<kIntSquares>(xy, xy) +
                               mul<kIntSquares>(xz, xz));
  GK = spline64<kInt>(quot<kInt>(rij, P.h), P.h, P.gkC);
  r2 = mul<kIntSquares>(rij, rij);
}

// Where the pair geometry of a pass comes from: computed (the work arrays
// could not be allocated), computed and kept for the passes behind it, or read.
enum { GEO_NONE = 0, GEO_STORE = 1, GEO_LOAD = 2 };

// GK is never positive, so the sign bit of a kept GK is free to say that the
// pair is tame: its position difference, GK and the neighbour's mass are zero
// or within 2^+-kTame (cleared: not, or GK = 0).
template <int kG, int kGeo>
__device__ __forceinline__ bool geometry(const StepParams& P, const Work64& W, int64_t e, double xx,
                                         double xy, double xz, double mj, double& GK, double& r2) {
  if constexpr (kGeo == GEO_LOAD) {
    const double k = __ldg(W.gk + e);
    r2 = __ldg(W.r2 + e);
    GK = __hiloint2double(__double2hiint(k) | (int)0x80000000, __double2loint(k));
    return __double2hiint(k) < 0;
  } else {
    bool tame = P.h_tame && within<kTame>(xx) && within<kTame>(xy) && within<kTame>(xz) &&
                within<kTame>(mj);
    if (kGeo != GEO_NONE && tame) pair_geometry<true, kG != 1>(P, xx, xy, xz, GK, r2);
    else pair_geometry<false>(P, xx, xy, xz, GK, r2);
    tame = tame && in_range<kTame>(GK) && in_range<2 * kTame>(r2);
    if constexpr (kGeo == GEO_STORE) {
      W.gk[e] = tame ? GK : fabs(GK);
      W.r2[e] = r2;
    }
    return tame;
  }
}

// ---- A: Domain_d::CalcDensInc + UpdateDensity ---------------------------
// src/cuda/InteractionAlt.cu:166-246, src/cuda/Mechanical.cu:198-203.
// Writes vd2 = (v, rho + dt*drho): the density the later passes of the step
// read, next to the velocity so one 32-byte load serves both; with the work
// arrays also m / rho of the new density.
template <bool kInt>
__device__ __forceinline__ double density_sum(double xx, double xy, double xz, double GK, double vx,
                                              double vy, double vz, double mj, double di,
                                              double dj) {
  const double temp1 = mul<kInt>(vx, mul<kInt>(xx, GK)) + mul<kInt>(vy, mul<kInt>(xy, GK)) +
                       mul<kInt>(vz, mul<kInt>(xz, GK));
  return mul<kInt>(mul<kInt>(mj, quot<kInt>(di, dj)), temp1);
}
template <int kG, int kGeo>
__device__ __forceinline__ double density_term(const StepParams& P, const Fields& F,
                                               const Work64& W, int64_t e, int j, const double4& xi,
                                               const double4& vi, bool pass) {
  const double4 xj = F.xm[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  const double mj = xj.w;
  double GK, r2;
  // kept for the other passes whatever the filter
  const bool tame = geometry<kG, kGeo>(P, W, e, xx, xy, xz, mj, GK, r2);
  if (!pass) return 0.0;
  const double4 vj = F.vd[j];
  const double di = vi.w, dj = vj.w;
  const double vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
  if constexpr (kGeo != GEO_NONE) {
    if (tame && within<kTame>(vx) && within<kTame>(vy) && within<kTame>(vz) &&
        in_range<kTame>(di) && in_range<kTame>(dj))
      return density_sum<true>(xx, xy, xz, GK, vx, vy, vz, mj, di, dj);
  }
  return density_sum<false>(xx, xy, xz, GK, vx, vy, vz, mj, di, dj);
}

template <int kG, int kGeo>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_density64(StepParams P, Fields F, Work64 W,
                                                   double4* __restrict__ vd2,
                                                   const int32_t* __restrict__ nb,
                                                   const int32_t* __restrict__ cnt) {
  __shared__ double sh[kG == 32 ? 32 : 1];
  int g;
  const int64_t i0 = slot64<kG>(g);
  if (kG == 1 && i0 >= P.n) return;
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : 0;
  const double4 xi = F.xm[i];
  const double4 vi = F.vd[i];
  const bool solid = valid && F.perm[i] < P.n_solid;
  const int32_t idi = F.id[i];
  const int c = solid ? cnt[i] : 0;
  double drho = 0.0;
  if constexpr (kG == 1) {
    for (int k = 0; k < c; k++) {
      const int64_t e = nb_at(P.npad, i, k);
      const int j = __ldg(nb + e);
      const bool pass = !P.contact || pass_ij(P, idi, F.id[j]);
      const double t = density_term<kG, kGeo>(P, F, W, e, j, xi, vi, pass);
      if (pass) drho += t;
    }
  } else {
    const int rounds = warp_rounds<kG>(c);
    for (int b = 0; b < rounds; b++) {
      double t = 0.0;
      if (kG * b + g < c) {
        const int64_t e = nb_at(P.npad, i, kG * b + g);
        const int j = __ldg(nb + e);
        const bool pass = !P.contact || pass_ij(P, idi, F.id[j]);
        t = density_term<kG, kGeo>(P, F, W, e, j, xi, vi, pass);
      }
      drho = add_in_order<kG>(sh, drho, t, c - kG * b);
    }
    if (!valid || g != 0) return;
  }
  double rho_new = vi.w;
  if (solid) {
    F.drho[i] = drho;
    rho_new = vi.w + P.dt * drho;
  }
  vd2[i] = make_double4(vi.x, vi.y, vi.z, rho_new);
  if (kGeo != GEO_NONE) W.mr[i] = xi.w / rho_new;
}

// ---- B: CalcRateTensors + PressureKernelExt + StressStrainOne -----------
// src/cuda/InteractionAlt.cu:262-383, src/cuda/Mechanical.cu:289-298 and
// :458-554.  The terms of one pair: D xx yy zz xy yz xz, W xy yz xz.
template <bool kInt>
__device__ __forceinline__ void rate_terms(double xx, double xy, double xz, double ax, double ay,
                                           double az, double GK, double mj_dj, double* t) {
  const double s = neg_half<kInt>(GK);
  // StrainRate (symmetric) scaled by -GK/2, then by mj/dj
  t[0] = mul<kInt>(mul<kInt>(mul<kInt>(twice<kInt>(ax), xx), s), mj_dj);
  t[1] = mul<kInt>(mul<kInt>(mul<kInt>(twice<kInt>(ay), xy), s), mj_dj);
  t[2] = mul<kInt>(mul<kInt>(mul<kInt>(twice<kInt>(az), xz), s), mj_dj);
  const double pxy = mul<kInt>(ax, xy), qxy = mul<kInt>(ay, xx), pxz = mul<kInt>(ax, xz),
               qxz = mul<kInt>(az, xx), pyz = mul<kInt>(ay, xz), qyz = mul<kInt>(az, xy);
  t[3] = mul<kInt>(mul<kInt>(pxy + qxy, s), mj_dj);
  t[4] = mul<kInt>(mul<kInt>(pyz + qyz, s), mj_dj);
  t[5] = mul<kInt>(mul<kInt>(pxz + qxz, s), mj_dj);
  // RotationRate with the reference's xz sign flip (zx left 0), :358-365
  t[6] = mul<kInt>(mul<kInt>(pxy - qxy, s), mj_dj);
  t[7] = mul<kInt>(mul<kInt>(pyz - qyz, s), mj_dj);
  t[8] = mul<kInt>(mul<kInt>(-(pxz - qxz), s), mj_dj);
}
template <int kG, int kGeo>
__device__ __forceinline__ void stress_terms(const StepParams& P, const Fields& F, const Work64& W,
                                             const double4* __restrict__ vd2, int64_t e, int j,
                                             const double4& xi, const double4& vi, double* t) {
  const double4 xj = F.xm[j];
  const double4 vj = vd2[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  const double ax = vi.x - vj.x, ay = vi.y - vj.y, az = vi.z - vj.z;
  double GK, r2, mj_dj;
  const bool tame = geometry<kG, kGeo>(P, W, e, xx, xy, xz, xj.w, GK, r2);
  if constexpr (kGeo == GEO_NONE) mj_dj = xj.w / vj.w;
  else mj_dj = __ldg(W.mr + j);
  if constexpr (kGeo != GEO_NONE) {
    if (tame && within<kTame>(ax) && within<kTame>(ay) && within<kTame>(az) &&
        within<kTame>(mj_dj)) {
      rate_terms<true>(xx, xy, xz, ax, ay, az, GK, mj_dj, t);
      return;
    }
  }
  rate_terms<false>(xx, xy, xz, ax, ay, az, GK, mj_dj, t);
}

// sigma / rho^2 of a slot (ai = 1 / rho^2), and whether all of it is tame
__device__ __forceinline__ void keep_sigma(const Work64& W, int64_t i, const double* sigma,
                                           double ai) {
  bool tame = true;
  for (int k = 0; k < 6; k++) {
    const double q = sigma[k] * ai;
    W.sa6[6 * i + k] = q;
    tame = tame && within<kTame>(q);
  }
  W.tame[i] = tame ? 1 : 0;
}

// The per-particle EOS and stress update from the particle's own rates
// (D xx yy zz xy yz xz, W xy yz xz); with the work arrays also sigma / rho^2
// for the acceleration pass.
__device__ __forceinline__ void stress_point(const StepParams& P, const Fields& F, const Work64& W,
                                             int64_t i, double rho, const double* r,
                                             int* __restrict__ status) {
  const double p = 0.0 + (P.Cs * P.Cs) * (rho - P.rho0);
  T3 SRS;
  SRS.xx = r[0]; SRS.yy = r[1]; SRS.zz = r[2];
  SRS.xy = SRS.yx = r[3]; SRS.yz = SRS.zy = r[4]; SRS.xz = SRS.zx = r[5];
  StressIn in;
  in.S = t3_from_sym(F.ss6 + 6 * i);
  in.D = SRS;
  in.Wflat[0] = 0.0; in.Wflat[1] = 0.0; in.Wflat[2] = 0.0;
  in.Wflat[3] = r[6]; in.Wflat[4] = r[7]; in.Wflat[5] = r[8];
  in.p = p;
  in.G = P.G;
  in.T = F.T[i];
  StressState st;
  st.eps_p = F.eps_p[i];
  st.sy = F.sy[i];
  st.pwn = F.pwn[i];
  StressOut out;
  stress_update_fp64(P, in, st, out);
  F.pwn[i] = st.pwn;
  F.eff[i] = out.eff;
  F.seq[i] = out.seq;
  F.eps_p[i] = st.eps_p;
  F.sy[i] = st.sy;
  F.dep[i] = out.dep;
  double* sg = F.sig6 + 6 * i;
  double* ss = F.ss6 + 6 * i;
  double* ep = F.eps6 + 6 * i;
  t3_store_flat(out.Sig, sg);
  t3_store_flat(out.S, ss);
  if (W.sa6) {
    const double ai = 1.0 / (rho * rho);
    const double q[6] = {out.Sig.xx, out.Sig.yy, out.Sig.zz, out.Sig.xy, out.Sig.yz, out.Sig.xz};
    keep_sigma(W, i, q, ai);
  }
  // strain += dt * D (the reference accumulates into an uninitialised local)
  ep[0] += SRS.xx * P.dt; ep[1] += SRS.yy * P.dt; ep[2] += SRS.zz * P.dt;
  ep[3] += SRS.xy * P.dt; ep[4] += SRS.yz * P.dt; ep[5] += SRS.xz * P.dt;
  if (P.log_cap > 0 && out.dep > 0.0 && P.mat.model == WF_JOHNSON_COOK && P.return_map == 1) {
    // (state, converged increment) pairs for training the warm-start MLP
    const unsigned long long slot = atomicAdd((unsigned long long*)P.log_count, 1ull);
    if (slot < (unsigned long long)P.log_cap) {
      float f[4];
      mlp_features((float)(out.st / out.sy0), st.eps_p - out.dep, (float)out.eff, (float)out.Th, f);
      P.log_x[slot] = make_float4(f[0], f[1], f[2], f[3]);
      P.log_y[slot] = (float)(out.dep / ((out.st - out.sy0) / (3.0 * P.G)));
    }
  }
  if (!isfinite(out.seq)) atomicOr(status, WF_STATUS_NAN);
  // Newton counters and the is_yielding flag (eps_p > 1e-6), one atomic per warp
  warp_count(status, (unsigned)out.newton_iters, out.newton_iters > 0 ? 1u : 0u, 0u,
             P.return_map == 1 && out.newton_iters >= P.newton_max_iter, st.eps_p > 1.e-6);
}


__device__ __forceinline__ void store_rates(const Fields& F, int64_t i, const double* r) {
  double* sr = F.sr6 + 6 * i;
  double* rr = F.rr6 + 6 * i;
  sr[0] = r[0]; sr[1] = r[1]; sr[2] = r[2]; sr[3] = r[3]; sr[4] = r[4]; sr[5] = r[5];
  rr[0] = 0.0; rr[1] = 0.0; rr[2] = 0.0; rr[3] = r[6]; rr[4] = r[7]; rr[5] = r[8];
}

// One lane per particle: the pair loop with the stress update behind it.
// Twelve blocks an SM (80 registers) hide the update's chains of operations:
// 170k particles 640 us with the 98 registers it would take, 604 with 80 (549
// now); the update as a kernel of its own, 624.
template <int kGeo>
__global__ void __launch_bounds__(64, 12) k_stress64(StepParams P, Fields F, Work64 W,
                                                     const double4* __restrict__ vd2,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt,
                                                     int* __restrict__ status) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double4 xi = F.xm[i];
  const double4 vi = vd2[i];
  // PressureKernelExt runs over every particle (EOS case 0, P0 = 0)
  F.p[i] = 0.0 + (P.Cs * P.Cs) * (vi.w - P.rho0);
  if (F.perm[i] >= P.n_solid) {
    if (W.sa6) keep_sigma(W, i, F.sig6 + 6 * i, 1.0 / (vi.w * vi.w));   // as stored
    return;
  }
  double r[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int c = cnt[i];
  for (int k = 0; k < c; k++) {
    const int64_t e = nb_at(P.npad, i, k);
    const int j = __ldg(nb + e);
    if (P.contact && !pass_j(P, F.id[j])) continue;
    double t[9];
    stress_terms<1, kGeo>(P, F, W, vd2, e, j, xi, vi, t);
#pragma unroll
    for (int a = 0; a < 9; a++) r[a] += t[a];
  }
  store_rates(F, i, r);
  stress_point(P, F, W, i, vi.w, r, status);
}

// Several lanes per particle: the pair loop alone (the rates go to sr6, rr6).
// The stress update is a kernel of its own, one lane per particle: behind the
// pair loop it would run on 1 to 4 of a warp's 32 lanes.
template <int kG, int kGeo>
__global__ void __launch_bounds__(32) k_rates64(StepParams P, Fields F, Work64 W,
                                                const double4* __restrict__ vd2,
                                                const int32_t* __restrict__ nb,
                                                const int32_t* __restrict__ cnt) {
  __shared__ double sh[32 * 9];
  int g;
  const int64_t i0 = slot64<kG>(g);
  const bool solid = i0 < P.n && F.perm[i0] < P.n_solid;
  const int64_t i = solid ? i0 : 0;
  const double4 xi = F.xm[i];
  const double4 vi = vd2[i];
  const int c = solid ? cnt[i] : 0;
  const int rounds = warp_rounds<kG>(c);
  double acc[2] = {0.0, 0.0};
  for (int b = 0; b < rounds; b++) {
    double t[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (kG * b + g < c) {
      const int64_t e = nb_at(P.npad, i, kG * b + g);
      const int j = __ldg(nb + e);
      if (!P.contact || pass_j(P, F.id[j])) stress_terms<kG, kGeo>(P, F, W, vd2, e, j, xi, vi, t);
    }
    add_in_order<kG, 9>(sh, t, g, acc, c - kG * b);
  }
  if (!solid) return;
  // accumulators 0-5 are D (sr6), 6-8 W (rr6 3-5); rr6 0-2 are zero
  if (g < 6) F.sr6[6 * i + g] = acc[0];
  else if (g < 9) F.rr6[6 * i + g - 3] = acc[0];
  if (kG < 9 && g == 0) F.rr6[6 * i + 5] = acc[1];
  if (g < 3) F.rr6[6 * i + g] = 0.0;
}

__global__ void __launch_bounds__(32) k_stress_point64(StepParams P, Fields F, Work64 W,
                                                       const double4* __restrict__ vd2,
                                                       int* __restrict__ status) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double rho = vd2[i].w;
  F.p[i] = 0.0 + (P.Cs * P.Cs) * (rho - P.rho0);
  if (F.perm[i] >= P.n_solid) {
    if (W.sa6) keep_sigma(W, i, F.sig6 + 6 * i, 1.0 / (rho * rho));   // as stored
    return;
  }
  const double* sr = F.sr6 + 6 * i;
  const double* rr = F.rr6 + 6 * i;
  const double r[9] = {sr[0], sr[1], sr[2], sr[3], sr[4], sr[5], rr[3], rr[4], rr[5]};
  stress_point(P, F, W, i, rho, r, status);
}

// ---- C: Domain_d::CalcAccel (src/cuda/InteractionAlt.cu:18-150) ---------
// si = sigma_i / rho_i^2 (xx yy zz xy yz xz)
template <bool kInt>
__device__ __forceinline__ void force_terms(double xx, double xy, double xz, double GK, double mj,
                                            const double* T, double* t) {
  const double gx = mul<kInt>(xx, GK), gy = mul<kInt>(xy, GK), gz = mul<kInt>(xz, GK);
  const double Mxx = mul<kInt>(T[0], mj), Myy = mul<kInt>(T[1], mj), Mzz = mul<kInt>(T[2], mj);
  const double Mxy = mul<kInt>(T[3], mj), Myz = mul<kInt>(T[4], mj), Mxz = mul<kInt>(T[5], mj);
  t[0] = mul<kInt>(Mxx, gx) + mul<kInt>(Mxy, gy) + mul<kInt>(Mxz, gz);
  t[1] = mul<kInt>(Mxy, gx) + mul<kInt>(Myy, gy) + mul<kInt>(Myz, gz);
  t[2] = mul<kInt>(Mxz, gx) + mul<kInt>(Myz, gy) + mul<kInt>(Mzz, gz);
}
// The artificial viscosity of a tame pair: false where a value in it leaves
// the range.
__device__ __forceinline__ bool viscosity_int(const StepParams& P, double xx, double xy, double xz,
                                              double vx, double vy, double vz, double r2, double di,
                                              double dj, double& PI) {
  const double vdx = mul_int(vx, xx) + mul_int(vy, xy) + mul_int(vz, xz);
  if (__double2hiint(vdx) >= 0) return true;
  const double den = r2 + P.visc_eps, aC = P.visc_ac;
  const double rho2 = di + dj;
  const double MU = div_int(mul_int(P.h, vdx), den);
  double num = mul_int(aC, MU);
  if (P.beta != 0.0) num = num + mul_int(mul_int(P.beta, MU), MU);
  PI = div_int(num, mul_int(0.5, rho2));
  return in_range<kTame>(MU) && within<kTame>(aC) && within<kTame>(P.beta) &&
         within<4 * kTame>(num) && in_range<kTame>(rho2) && in_range<2 * kTame>(den);
}
template <int kG, int kGeo>
__device__ __forceinline__ void accel_terms(const StepParams& P, const Fields& F, const Work64& W,
                                            const double4* __restrict__ vd2, int64_t e, int j,
                                            const double4& xi, const double4& vi, const double* si,
                                            bool tame_i, double* t) {
  const double4 xj = F.xm[j];
  const double4 vj = vd2[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  const double di = vi.w, dj = vj.w, mj = xj.w;
  const double vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
  double GK, r2;
  bool tame = geometry<kG, kGeo>(P, W, e, xx, xy, xz, mj, GK, r2) && tame_i;
  double2 s01, s23, s45;
  if constexpr (kGeo == GEO_NONE) {
    const double2* q = reinterpret_cast<const double2*>(F.sig6 + 6 * (int64_t)j);
    const double aj = 1.0 / (dj * dj);
    s01 = make_double2(q[0].x * aj, q[0].y * aj);
    s23 = make_double2(q[1].x * aj, q[1].y * aj);
    s45 = make_double2(q[2].x * aj, q[2].y * aj);
  } else {
    const double2* q = reinterpret_cast<const double2*>(W.sa6 + 6 * (int64_t)j);
    s01 = q[0]; s23 = q[1]; s45 = q[2];
    tame = tame && __ldg(W.tame + j) != 0;
  }
  // Si/di^2 + Sj/dj^2 + PI*I, times mj, then times GK*xij (tensor3.cu:225)
  double T[6] = {si[0] + s01.x, si[1] + s01.y, si[2] + s23.x,
                 si[3] + s23.y, si[4] + s45.x, si[5] + s45.y};
  if (P.alpha != 0.0 || P.beta != 0.0) {
    bool done = false;
    double PI = 0.0;
    if constexpr (kGeo != GEO_NONE) {
      if (tame && within<kTame>(vx) && within<kTame>(vy) && within<kTame>(vz))
        done = viscosity_int(P, xx, xy, xz, vx, vy, vz, r2, di, dj, PI);
    }
    if (!done) {
      const double vdx = vx * xx + vy * xy + vz * xz;
      PI = 0.0;
      if (vdx < 0) {
        const double MU = P.h * vdx / (r2 + 0.01 * P.h * P.h);
        const double Cij = 0.5 * (P.Cs + P.Cs);
        PI = (P.alpha * Cij * MU + P.beta * MU * MU) / (0.5 * (di + dj));
      }
    }
    // (adding the zero of a pair that moves apart changes no term)
    T[0] = T[0] + PI;
    T[1] = T[1] + PI;
    T[2] = T[2] + PI;
    tame = tame && within<kTame>(PI);
  }
  if (kGeo != GEO_NONE && tame) force_terms<true>(xx, xy, xz, GK, mj, T, t);
  else force_terms<false>(xx, xy, xz, GK, mj, T, t);
}

template <int kGeo>
__device__ __forceinline__ void own_sigma(const Fields& F, const Work64& W, int64_t i, double di,
                                          double* si) {
  if constexpr (kGeo == GEO_NONE) {
    const double* q = F.sig6 + 6 * i;
    const double ai = 1.0 / (di * di);
    for (int k = 0; k < 6; k++) si[k] = q[k] * ai;
  } else {
    for (int k = 0; k < 6; k++) si[k] = W.sa6[6 * i + k];
  }
}

template <int kG, int kGeo>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_accel64(StepParams P, Fields F, Work64 W,
                                                 const double4* __restrict__ vd2,
                                                 const int32_t* __restrict__ nb,
                                                 const int32_t* __restrict__ cnt) {
  __shared__ double sh[kG == 1 ? 1 : 32 * 3];
  int g;
  const int64_t i0 = slot64<kG>(g);
  const bool solid = i0 < P.n && F.perm[i0] < P.n_solid;
  if (kG == 1 && !solid) return;
  const int64_t i = solid ? i0 : 0;
  const double4 xi = F.xm[i];
  const double4 vi = vd2[i];
  const int32_t idi = F.id[i];
  double si[6];
  own_sigma<kGeo>(F, W, i, vi.w, si);
  const bool tame_i = kGeo != GEO_NONE && W.tame[i] != 0;
  const int c = solid ? cnt[i] : 0;
  double t[3];
  if constexpr (kG == 1) {
    double a[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < c; k++) {
      const int64_t e = nb_at(P.npad, i, k);
      const int j = __ldg(nb + e);
      if (P.contact && !pass_ij(P, idi, F.id[j])) continue;
      accel_terms<kG, kGeo>(P, F, W, vd2, e, j, xi, vi, si, tame_i, t);
      a[0] += t[0]; a[1] += t[1]; a[2] += t[2];
    }
    F.a[i] = make_double4(a[0], a[1], a[2], 0.0);
  } else {
    const int rounds = warp_rounds<kG>(c);
    double acc[2] = {0.0, 0.0};
    for (int b = 0; b < rounds; b++) {
      t[0] = t[1] = t[2] = 0.0;
      if (kG * b + g < c) {
        const int64_t e = nb_at(P.npad, i, kG * b + g);
        const int j = __ldg(nb + e);
        if (!P.contact || pass_ij(P, idi, F.id[j]))
          accel_terms<kG, kGeo>(P, F, W, vd2, e, j, xi, vi, si, tame_i, t);
      }
      add_in_order<kG, 3>(sh, t, g, acc, c - kG * b);
    }
    if (solid && g < 4) reinterpret_cast<double*>(F.a + i)[g] = acc[0];   // lane 3: 0
  }
}

// ---- heat: ThermalSolveKernel + plastic heat + CalcConvHeatKernel -------
// src/cuda/Thermal.cu:101-142 and :36-64, FP64 form: the reference's
// arithmetic in its order.  The mixed form's heat pass is k_heat32
// (wf_step_fp32.cu): pair flux in FP32 with the temperature difference taken
// from the (hi, lo) float pair; dT/dt and T stay FP64.  It runs behind the
// integration, so the geometry that it computes is that of the next step.
template <bool kInt>
__device__ __forceinline__ double heat_flux(double xx, double xy, double xz, double GK, double r2,
                                            double mj_dj, double kk, double dT) {
  return quot<kInt>(mul<kInt>(mul<kInt>(mj_dj, mul<kInt>(kk, dT)),
                              mul<kInt>(xx, mul<kInt>(xx, GK)) + mul<kInt>(xy, mul<kInt>(xy, GK)) +
                                  mul<kInt>(xz, mul<kInt>(xz, GK))), r2);
}
template <int kG, int kGeo>
__device__ __forceinline__ double heat_term(const StepParams& P, const Fields& F, const Work64& W,
                                            int64_t e, int j, const double4& xi, double Ti,
                                            double kk) {
  const double4 xj = F.xm[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  double GK, r2;
  const bool tame = geometry<kG, kGeo>(P, W, e, xx, xy, xz, xj.w, GK, r2);
  const double mj_dj = W.mr_heat ? __ldg(W.mr_heat + j) : xj.w / F.vd[j].w;
  const double dT = Ti - F.T[j];
  if constexpr (kGeo != GEO_NONE) {
    if (tame && within<kTame>(mj_dj) && within<kTame>(dT) && within<kTame>(kk))
      return heat_flux<true>(xx, xy, xz, GK, r2, mj_dj, kk, dT);
  }
  return heat_flux<false>(xx, xy, xz, GK, r2, mj_dj, kk, dT);
}

template <int kG, int kGeo>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_heat_rate(StepParams P, Fields F, Work64 W,
                                                   const int32_t* __restrict__ nb,
                                                   const int32_t* __restrict__ cnt,
                                                   int plastic_heat) {
  __shared__ double sh[kG == 32 ? 32 : 1];
  int g;
  const int64_t i0 = slot64<kG>(g);
  if (kG == 1 && i0 >= P.n) return;
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : 0;
  const double4 xi = F.xm[i];
  const double rhoi = F.vd[i].w;
  const double Ti = F.T[i], ki = F.kT[i];
  // the pair conductivity 4 k_i k_j / (k_i + k_j): the conductivity is one value for
  // every particle (wf_set_conductivity), so it is one value for every pair
  const double kk = 4.0 * ki * ki / (ki + ki);
  const int c = valid ? cnt[i] : 0;
  double s = 0.0;
  if constexpr (kG == 1) {
    for (int k = 0; k < c; k++) {
      const int64_t e = nb_at(P.npad, i, k);
      s += heat_term<kG, kGeo>(P, F, W, e, __ldg(nb + e), xi, Ti, kk);
    }
  } else {
    const int rounds = warp_rounds<kG>(c);
    for (int b = 0; b < rounds; b++) {
      double t = 0.0;
      if (kG * b + g < c) {
        const int64_t e = nb_at(P.npad, i, kG * b + g);
        t = heat_term<kG, kGeo>(P, F, W, e, __ldg(nb + e), xi, Ti, kk);
      }
      s = add_in_order<kG>(sh, s, t, c - kG * b);
    }
    if (!valid || g != 0) return;
  }
  F.dTdt[i] = heat_rate_fp64(P, F, i, s, rhoi, xi.w, Ti, plastic_heat);
}


// ---- ThermalSolve in FP64 (src/cuda/Thermal.cu:188-260) --------------------
// Positions, densities and lists do not change inside a heat solve, so what a
// pair contributes apart from the temperatures is computed once per solve:
// the product of the position difference with the kernel gradient and r^2 (two
// arrays of the lists' layout), m / rho, and the particle's own factors.  A
// step is then two FP64 operations, three integer products and a quotient a
// pair, and takes the leapfrog update with it; the neighbours' temperatures
// are read from one array while the new ones go to another.  64,000
// particles, 20 steps: 15.5 ms recomputing the pairs on the FP64 pipe, 1.88
// with the kept factors, 1.38 on the integer pipes, 1.2 with two lanes.
//
// Where the factor of entry k of particle i stands: with one or two lanes per
// particle (kRows) in row k of npad factors, so that a warp's reads and writes
// of an entry are whole lines (in the lists' blocks they are 16), else where
// the lists have it, so that a group's are.
template <bool kRows>
__device__ __forceinline__ int64_t factor_at(int64_t npad, int64_t i, int k) {
  return kRows ? k * npad + i : nb_at(npad, i, k);
}
template <bool kRows>
__global__ void __launch_bounds__(64) k_heat_pairs64(StepParams P, Fields F, HeatWork64 H,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double4 xi = F.xm[i];
  const double rhoi = F.vd[i].w, cp = F.cpT[i];
  H.mr[i] = xi.w / rhoi;
  H.scale[i] = 1. / (rhoi * cp);
  H.icp[i] = 1. / cp;
  H.conv[i] = F.bct[i] == 1 ? P.h_conv * pow(xi.w / rhoi, 0.666666666) : 0.0;
  H.fric[i] = F.qf && F.qf[i] > 0.0 ? F.qf[i] / (xi.w * cp) : 0.0;
  const int c = cnt[i];
  for (int k = 0; k < c; k++) {
    const int64_t e = factor_at<kRows>(P.npad, i, k);
    const double4 xj = F.xm[__ldg(nb + nb_at(P.npad, i, k))];
    const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
    double GK, r2;
    if (P.h_tame && within<kTame>(xx) && within<kTame>(xy) && within<kTame>(xz)) {
      pair_geometry<true, false>(P, xx, xy, xz, GK, r2);
      if (in_range<kTame>(GK)) {
        H.dot[e] = mul_int(xx, mul_int(xx, GK)) + mul_int(xy, mul_int(xy, GK)) +
                   mul_int(xz, mul_int(xz, GK));
        H.r2[e] = r2;
        continue;
      }
    }
    pair_geometry<false>(P, xx, xy, xz, GK, r2);
    H.dot[e] = xx * (xx * GK) + xy * (xy * GK) + xz * (xz * GK);
    H.r2[e] = r2;
  }
}

__device__ __forceinline__ double heat_step_term(double mr, double dT, double dot, double r2,
                                                 double kk) {
  if (within<kTame>(mr) && within<kTame>(dT) && within<kTame>(dot) && within<kTame>(kk) &&
      in_range<kTame>(r2))
    return div_int(mul_int(mul_int(mr, mul_int(kk, dT)), dot), r2);
  return mr * (kk * dT) * dot / r2;
}

template <int kG>
__global__ void __launch_bounds__(kG <= 2 ? 64 : 32) k_heat_step64(StepParams P, Fields F,
                                                     HeatWork64 H, const double* __restrict__ T,
                                                     double* __restrict__ T_out,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt, int first) {
  __shared__ double sh[kG == 32 ? 32 : 1];
  int g;
  const int64_t i0 = slot64<kG>(g);
  if (kG == 1 && i0 >= P.n) return;
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : 0;
  const double Ti = T[i], ki = F.kT[i];
  const double kk = 4.0 * ki * ki / (ki + ki);
  const int c = valid ? cnt[i] : 0;
  double s = 0.0;
  if constexpr (kG <= 2) {
    // Four entries a lane at a time, their loads in flight together; with two
    // lanes the terms of 8 b .. 8 b + 3 are lane 0's, and the sum goes from lane
    // to lane in list order.
    const int rounds = (kG == 1 ? c + 3 : __reduce_max_sync(0xffffffffu, c) + 7) / (4 * kG);
    for (int b = 0; b < rounds; b++) {
      const int k0 = 4 * (kG * b + g);
      double t[4] = {0.0, 0.0, 0.0, 0.0};
      if (k0 < c) {
        const int4 ja = __ldg(reinterpret_cast<const int4*>(nb + nb_at(P.npad, i, k0)));
        const int js[4] = {ja.x, ja.y, ja.z, ja.w};        // (past the list: the own slot)
        double mr[4], Tj[4], dot[4], r2[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int64_t e = factor_at<true>(P.npad, i, k0 + k);
          mr[k] = __ldg(H.mr + js[k]);
          Tj[k] = __ldg(T + js[k]);
          dot[k] = k0 + k < c ? __ldg(H.dot + e) : 0.0;
          r2[k] = k0 + k < c ? __ldg(H.r2 + e) : 1.0;
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (k0 + k < c) t[k] = heat_step_term(mr[k], Ti - Tj[k], dot[k], r2[k], kk);
      }
#pragma unroll
      for (int turn = 0; turn < kG; turn++) {
#pragma unroll
        for (int k = 0; k < 4; k++) s += t[k];
        if constexpr (kG == 2) s = __shfl_sync(0xffffffffu, s, turn, 2);
      }
    }
    if (!valid || g != 0) return;
  } else {
    const int rounds = warp_rounds<kG>(c);
    for (int b = 0; b < rounds; b++) {
      double t = 0.0;
      if (kG * b + g < c) {
        const int64_t e = factor_at<false>(P.npad, i, kG * b + g);
        const int j = __ldg(nb + e);
        t = heat_step_term(__ldg(H.mr + j), Ti - __ldg(T + j), __ldg(H.dot + e), __ldg(H.r2 + e), kk);
      }
      s = add_in_order<kG>(sh, s, t, c - kG * b);
    }
    if (!valid || g != 0) return;
  }
  // heat_rate_fp64 without plastic heat, from the kept factors
  s *= H.scale[i];
  const double fric = H.fric[i];
  if (fric > 0.0) s += fric;
  if (F.bct[i] == 1) s += H.icp[i] * (H.conv[i] * (P.T_inf - Ti) / F.xm[i].w);
  F.dTdt[i] = s;
  if (first) {
    F.Ta[i] = Ti - P.dt / 2.0 * s;
    T_out[i] = Ti;
    return;
  }
  const double ta = F.Ta[i];
  F.Tb[i] = ta;
  const double ta2 = ta + s * P.dt;
  F.Ta[i] = ta2;
  T_out[i] = (ta2 + ta) / 2.;
}

}  // namespace

static inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

// Lanes of the passes that have a form with four: in mid-sized domains four lanes
// hide more of a pair's chain of operations than one and spend fewer additions
// on the ordered sums than eight.  Pass, us, with 8 / 4 / 1 lanes: density
// 14,040 particles 38 / 35 / -, 50,560 112 / 95 / -, 86,592 - / 149 / 149,
// 169,680 - / 273 / 246; acceleration 10,752 52 / 55 / -, 14,040 69 / 62 / -,
// 50,560 201 / 186 / -, 169,680 - / 577 / 601, 401,920 - / 1,341 / 1,348,
// 786,000 - / 2,943 / 2,908; heat (and density, where they compute the
// geometry) 36,720 106 / 108 / -, 50,560 137 / 134 / -, 86,592 - / 210 / 227,
// 169,680 - / 389 / 384, 786,000 - / 1,705 / 1,505.
static int density_lanes(int64_t n) { return n >= 64000 ? 1 : n >= 12000 ? 4 : lanes64(n); }
static int accel_lanes(int64_t n) { return n >= 300000 ? 1 : n >= 12000 ? 4 : lanes64(n); }
static int geometry_lanes(int64_t n) { return n >= 130000 ? 1 : n >= 45000 ? 4 : lanes64(n); }

// Launches K<lanes, geometry>.
#define WF_LAUNCH64(LANES, K, GEO, ...)                                                        \
  do {                                                                                         \
    const int lanes = LANES, grid = blocks_for(P.n * lanes, lanes == 1 ? 64 : 32);             \
    if (lanes == 32) K<32, GEO><<<grid, 32, 0, s>>>(P, F, W, __VA_ARGS__);                     \
    else if (lanes == 16) K<16, GEO><<<grid, 32, 0, s>>>(P, F, W, __VA_ARGS__);                \
    else if (lanes == 8) K<8, GEO><<<grid, 32, 0, s>>>(P, F, W, __VA_ARGS__);                  \
    else if (lanes == 4) K<4, GEO><<<grid, 32, 0, s>>>(P, F, W, __VA_ARGS__);                  \
    else K<1, GEO><<<grid, 64, 0, s>>>(P, F, W, __VA_ARGS__);                                  \
  } while (0)

void launch_fp64_density(const StepParams& P, const Fields& F, const Work64& W, double4* vd2,
                         const NbBuffers& N, cudaStream_t s) {
  if (!W.gk) WF_LAUNCH64(density_lanes(P.n), k_density64, GEO_NONE, vd2, N.nb, N.cnt);
  else if (W.geo) WF_LAUNCH64(density_lanes(P.n), k_density64, GEO_LOAD, vd2, N.nb, N.cnt);
  else WF_LAUNCH64(geometry_lanes(P.n), k_density64, GEO_STORE, vd2, N.nb, N.cnt);
}
int launch_fp64_stress(const StepParams& P, const Fields& F, const Work64& W, const double4* vd2,
                       const NbBuffers& N, int* status, cudaStream_t s) {
  const int lanes = lanes64(P.n), grid = blocks_for(P.n * lanes, lanes == 1 ? 64 : 32);
  if (lanes == 1) {
    if (W.gk) k_stress64<GEO_LOAD><<<grid, 64, 0, s>>>(P, F, W, vd2, N.nb, N.cnt, status);
    else k_stress64<GEO_NONE><<<grid, 64, 0, s>>>(P, F, W, vd2, N.nb, N.cnt, status);
    return 1;
  }
  if (lanes == 32) {
    if (W.gk) k_rates64<32, GEO_LOAD><<<grid, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
    else k_rates64<32, GEO_NONE><<<grid, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
  } else if (lanes == 16) {
    if (W.gk) k_rates64<16, GEO_LOAD><<<grid, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
    else k_rates64<16, GEO_NONE><<<grid, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
  } else {
    if (W.gk) k_rates64<8, GEO_LOAD><<<grid, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
    else k_rates64<8, GEO_NONE><<<grid, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
  }
  k_stress_point64<<<blocks_for(P.n, 32), 32, 0, s>>>(P, F, W, vd2, status);
  return 2;
}
void launch_fp64_accel(const StepParams& P, const Fields& F, const Work64& W, const double4* vd2,
                       const NbBuffers& N, cudaStream_t s) {
  if (W.gk) WF_LAUNCH64(accel_lanes(P.n), k_accel64, GEO_LOAD, vd2, N.nb, N.cnt);
  else WF_LAUNCH64(accel_lanes(P.n), k_accel64, GEO_NONE, vd2, N.nb, N.cnt);
}
void launch_fp64_heat_rate(const StepParams& P, const Fields& F, const Work64& W,
                           const NbBuffers& N, int plastic_heat, cudaStream_t s) {
  if (W.gk) WF_LAUNCH64(geometry_lanes(P.n), k_heat_rate, GEO_STORE, N.nb, N.cnt, plastic_heat);
  else WF_LAUNCH64(geometry_lanes(P.n), k_heat_rate, GEO_NONE, N.nb, N.cnt, plastic_heat);
}
// Lanes of a particle in a heat solve's steps.  A step, us, with 1 / 2 lanes and
// four entries a lane in flight / the lanes of lanes64: n = 8,000 - / 18.5 /
// 16.4, 13,824 - / 20.4 / 22.6, 46,656 - / 34.9 / 66.6, 64,000 48.9 / 45.0 /
// 53.3, 85,184 61.4 / 59.8, 110,592 72.3 / 74.8, a million 500 / 529.
static int heat_lanes(int64_t n) { return n >= 100000 ? 1 : n >= 12000 ? 2 : lanes64(n); }

void launch_heat_pairs64(const StepParams& P, const Fields& F, const HeatWork64& H,
                         const NbBuffers& N, cudaStream_t s) {
  if (heat_lanes(P.n) <= 2) k_heat_pairs64<true><<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, H, N.nb, N.cnt);
  else k_heat_pairs64<false><<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, H, N.nb, N.cnt);
}
void launch_heat_step64(const StepParams& P, const Fields& F, const HeatWork64& H, double* T_out,
                        const NbBuffers& N, int first, cudaStream_t s) {
  const int lanes = heat_lanes(P.n), grid = blocks_for(P.n * lanes, lanes <= 2 ? 64 : 32);
  if (lanes == 32)
    k_heat_step64<32><<<grid, 32, 0, s>>>(P, F, H, F.T, T_out, N.nb, N.cnt, first);
  else if (lanes == 16)
    k_heat_step64<16><<<grid, 32, 0, s>>>(P, F, H, F.T, T_out, N.nb, N.cnt, first);
  else if (lanes == 8)
    k_heat_step64<8><<<grid, 32, 0, s>>>(P, F, H, F.T, T_out, N.nb, N.cnt, first);
  else if (lanes == 2)
    k_heat_step64<2><<<grid, 64, 0, s>>>(P, F, H, F.T, T_out, N.nb, N.cnt, first);
  else
    k_heat_step64<1><<<grid, 64, 0, s>>>(P, F, H, F.T, T_out, N.nb, N.cnt, first);
}
