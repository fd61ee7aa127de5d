// wf_step_fp64.cu — plain-FP64 form of the Fraser step.
//
// Compiled with -fmad=false, like the reference (--fmad=false,
// src/CMakeLists.txt:29): every multiply and add rounds separately, so with
// the same neighbour order the sums are bit-identical to the CPU oracle.
// Each kernel states the reference kernel(s) it replaces.
//
// What bounds these passes is the FP64 pipe (2 operations per clock and SM,
// 1/64 of the FP32 rate): ncu showed it 86-87 % busy in every pair pass at
// 170k particles with 72 / 113 / 133 / 90 FP64 instructions a pair (density,
// stress, acceleration, heat).  Memory is nearly idle there, so whatever can be
// computed once and read back is:
//   - the kernel factor GK and r^2 of each pair (a square root, a division by
//     h, a division by q h: about half of a density pass) by the first pass
//     that sees the positions, kept in two arrays of the lists' layout for the
//     other passes of the step (Work64);
//   - m / rho, 1 / rho and sigma / rho^2 once per particle instead of a
//     division per pair; the remaining rho_i / rho_j divides by a number whose
//     reciprocal is known (div_known).
// Every value is rounded exactly as where it was computed per pair.
#include "wf_common.cuh"
#include "wf_heat.cuh"
#include "wf_mlp.cuh"
#include "wf_tensor.cuh"

namespace {

// a / b, correctly rounded, from y = 1 / b correctly rounded: one
// multiplication and two fused multiply-adds (Brisebarre, Muller and Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", IEEE Trans. Computers 53(8), 2004; the last step is
// Markstein's).  Needs a, b and a / b well inside the normal range.
__device__ __forceinline__ double div_known(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
// |x| in [2^-400, 2^400], from the exponent bits (a comparison of doubles
// would run on the FP64 pipe)
__device__ __forceinline__ bool mid_range(double x) {
  return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 623u <= 800u;
}
// -0.5 x and 2 x: exact, so only the sign and exponent bits change (zeros,
// subnormals and the ends of the range take the multiplication)
__device__ __forceinline__ double neg_half(double x) {
  const int hi = __double2hiint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  if (e - 2u < 2045u) return __hiloint2double((hi ^ (int)0x80000000) - 0x00100000, __double2loint(x));
  return -0.5 * x;
}
__device__ __forceinline__ double twice(double x) {
  const int hi = __double2hiint(x);
  const unsigned e = ((unsigned)hi >> 20) & 0x7ffu;
  if (e - 1u < 2045u) return __hiloint2double(hi + 0x00100000, __double2loint(x));
  return x + x;
}

// The cubic-spline gradient factor of gradK64, bit for bit, with the division
// shared by its two branches (so a warp whose lanes fall on both sides of
// q = 1 divides once) and the comparisons on the bits of q >= 0.  q >= 2,
// infinite or NaN gives 0.
__device__ __forceinline__ double spline64(double q, double h, double C) {
  const unsigned hi = (unsigned)__double2hiint(q);
  if (hi >= 0x40000000u) return 0.0;
  if ((hi | (unsigned)__double2loint(q)) == 0u) return C / h * (-3.0 + (9.0 / 2.0) * q);
  const bool in = hi < 0x3ff00000u;
  const double s = in ? q : 2.0 - q;
  const double c = ((in ? 9.0 / 4.0 : -3.0 / 4.0) * s) * s;
  return C / (q * h) * (in ? -3.0 * q + c : c);
}

// GK and RN(r r) of a pair from x_i - x_j
__device__ __forceinline__ void pair_geometry(const StepParams& P, double xx, double xy, double xz,
                                              double& GK, double& r2) {
  const double rij = sqrt(xx * xx + xy * xy + xz * xz);
  GK = spline64(P.h_known ? div_known(rij, P.h, P.invh) : rij / P.h, P.h, P.gkC);
  r2 = rij * rij;
}

// Where the pair geometry of a pass comes from: computed (the work arrays
// could not be allocated), computed and kept for the passes behind it, or read.
enum { GEO_NONE = 0, GEO_STORE = 1, GEO_LOAD = 2 };

template <int kGeo>
__device__ __forceinline__ void geometry(const StepParams& P, const Work64& W, int64_t e, double xx,
                                         double xy, double xz, double& GK, double& r2) {
  if constexpr (kGeo == GEO_LOAD) {
    GK = __ldg(W.gk + e);
    r2 = __ldg(W.r2 + e);
  } else {
    pair_geometry(P, xx, xy, xz, GK, r2);
    if constexpr (kGeo == GEO_STORE) {
      W.gk[e] = GK;
      W.r2[e] = r2;
    }
  }
}

// ---- lanes of a particle ---------------------------------------------------
// kG = 1: one thread per particle walks its list.  kG = 8: eight lanes per
// particle, lane g takes entry 8 b + g of list block b (one coalesced read of
// the block's indices and geometry), and the block's terms are added in list
// order, term by term, so the sums round as in the walk.  Eight lanes spread a
// small domain over the chip (540 particles are 5 blocks of 128 threads, 135
// warps with eight lanes each) and shorten the chain of dependent pairs; the
// ordered sums cost up to 8 additions per list block and accumulator set, so
// a domain that fills the SMs is faster with one lane.
constexpr int kLanes64 = 8;

// this thread's slot, lane and list length; threads past the end or without a
// list keep c = 0 and stay for the warp's shuffles
template <int kG>
__device__ __forceinline__ int64_t slot64(int& g) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  g = (int)(t & (kG - 1));
  return t / kG;
}
// list blocks the warp walks together (eight lanes per particle)
__device__ __forceinline__ int warp_blocks(int c) {
  return (__reduce_max_sync(0xffffffffu, c) + WF_NB_BLK - 1) / WF_NB_BLK;
}
// acc + t_0 + ... + t_7 over the lanes of a group, in lane order, on every lane
__device__ __forceinline__ double add_in_order(double acc, double t) {
#pragma unroll
  for (int k = 0; k < kLanes64; k++) acc += __shfl_sync(0xffffffffu, t, k, kLanes64);
  return acc;
}
// The same for kA accumulators through shared memory (32 rows of kA doubles,
// kA odd: no bank conflicts): lane a of the group adds accumulator a, lane
// a - 8 accumulator a >= 8.
template <int kA>
__device__ __forceinline__ void add_in_order(double* sh, const double* t, int g, double* acc) {
  static_assert(kA % 2 == 1 && kA <= 2 * kLanes64, "accumulators of a group");
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < kA; a++) sh[lane * kA + a] = t[a];
  __syncwarp();
  const double* row = sh + (lane - g) * kA;
  if (g < kA)
#pragma unroll
    for (int k = 0; k < kLanes64; k++) acc[0] += row[k * kA + g];
  if (kA > kLanes64 && g < kA - kLanes64)
#pragma unroll
    for (int k = 0; k < kLanes64; k++) acc[1] += row[k * kA + g + kLanes64];
  __syncwarp();
}

// ---- A: Domain_d::CalcDensInc + UpdateDensity ---------------------------
// src/cuda/InteractionAlt.cu:166-246, src/cuda/Mechanical.cu:198-203.
// Writes vd2 = (v, rho + dt*drho): the density the later passes of the step
// read, next to the velocity so one 32-byte load serves both; with the work
// arrays also m / rho and 1 / rho of the new density.
template <int kGeo>
__device__ __forceinline__ double density_term(const StepParams& P, const Fields& F,
                                               const Work64& W, int64_t e, int j, const double4& xi,
                                               const double4& vi, bool known_i, bool pass) {
  const double4 xj = F.xm[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  double GK, r2;
  geometry<kGeo>(P, W, e, xx, xy, xz, GK, r2);   // kept for the other passes whatever the filter
  if (!pass) return 0.0;
  const double4 vj = F.vd[j];
  const double di = vi.w, dj = vj.w, mj = xj.w;
  const double vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
  const double temp1 = vx * (xx * GK) + vy * (xy * GK) + vz * (xz * GK);
  double ratio;
  if (kGeo != GEO_NONE && known_i) {
    const double y = __ldg(W.rr + j);
    ratio = mid_range(y) ? div_known(di, dj, y) : di / dj;
  } else {
    ratio = di / dj;
  }
  return mj * ratio * temp1;
}

template <int kG, int kGeo>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_density64(StepParams P, Fields F, Work64 W,
                                                   double4* __restrict__ vd2,
                                                   const int32_t* __restrict__ nb,
                                                   const int32_t* __restrict__ cnt) {
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
  const bool known_i = W.recip && mid_range(vi.w);
  double drho = 0.0;
  if constexpr (kG == 1) {
    for (int k = 0; k < c; k++) {
      const int64_t e = nb_at(P.npad, i, k);
      const int j = __ldg(nb + e);
      const bool pass = !P.contact || pass_ij(P, idi, F.id[j]);
      const double t = density_term<kGeo>(P, F, W, e, j, xi, vi, known_i, pass);
      if (pass) drho += t;
    }
  } else {
    const int blocks = warp_blocks(c);
    for (int b = 0; b < blocks; b++) {
      double t = 0.0;
      if (WF_NB_BLK * b + g < c) {
        const int64_t e = nb_at(P.npad, i, WF_NB_BLK * b + g);
        const int j = __ldg(nb + e);
        const bool pass = !P.contact || pass_ij(P, idi, F.id[j]);
        t = density_term<kGeo>(P, F, W, e, j, xi, vi, known_i, pass);
      }
      drho = add_in_order(drho, t);
    }
    if (!valid || g != 0) return;
  }
  double rho_new = vi.w;
  if (solid) {
    F.drho[i] = drho;
    rho_new = vi.w + P.dt * drho;
  }
  vd2[i] = make_double4(vi.x, vi.y, vi.z, rho_new);
  if (kGeo != GEO_NONE) {
    W.mr[i] = xi.w / rho_new;
    W.rr_out[i] = 1.0 / rho_new;
  }
}

// ---- B: CalcRateTensors + PressureKernelExt + StressStrainOne -----------
// src/cuda/InteractionAlt.cu:262-383, src/cuda/Mechanical.cu:289-298 and
// :458-554.  The terms of one pair: D xx yy zz xy yz xz, W xy yz xz.
template <int kGeo>
__device__ __forceinline__ void stress_terms(const StepParams& P, const Fields& F, const Work64& W,
                                             const double4* __restrict__ vd2, int64_t e, int j,
                                             const double4& xi, const double4& vi, double* t) {
  const double4 xj = F.xm[j];
  const double4 vj = vd2[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  const double ax = vi.x - vj.x, ay = vi.y - vj.y, az = vi.z - vj.z;
  double GK, mj_dj;
  if constexpr (kGeo == GEO_NONE) {
    double r2;
    pair_geometry(P, xx, xy, xz, GK, r2);
    mj_dj = xj.w / vj.w;
  } else {
    GK = __ldg(W.gk + e);
    mj_dj = __ldg(W.mr + j);
  }
  const double s = neg_half(GK);
  // StrainRate (symmetric) scaled by -GK/2, then by mj/dj
  t[0] = (twice(ax) * xx) * s * mj_dj;
  t[1] = (twice(ay) * xy) * s * mj_dj;
  t[2] = (twice(az) * xz) * s * mj_dj;
  const double pxy = ax * xy, qxy = ay * xx, pxz = ax * xz, qxz = az * xx, pyz = ay * xz,
               qyz = az * xy;
  t[3] = (pxy + qxy) * s * mj_dj;
  t[4] = (pyz + qyz) * s * mj_dj;
  t[5] = (pxz + qxz) * s * mj_dj;
  // RotationRate with the reference's xz sign flip (zx left 0), :358-365
  t[6] = (pxy - qxy) * s * mj_dj;
  t[7] = (pyz - qyz) * s * mj_dj;
  t[8] = (-(pxz - qxz)) * s * mj_dj;
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
    double* sa = W.sa6 + 6 * i;
    sa[0] = out.Sig.xx * ai; sa[1] = out.Sig.yy * ai; sa[2] = out.Sig.zz * ai;
    sa[3] = out.Sig.xy * ai; sa[4] = out.Sig.yz * ai; sa[5] = out.Sig.xz * ai;
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

// sigma / rho^2 of a slot that the stress update skips (a rigid one), as stored
__device__ __forceinline__ void keep_sigma(const Fields& F, const Work64& W, int64_t i, double rho) {
  if (!W.sa6) return;
  const double ai = 1.0 / (rho * rho);
  for (int k = 0; k < 6; k++) W.sa6[6 * i + k] = F.sig6[6 * i + k] * ai;
}

// One lane per particle: the pair loop with the stress update behind it.
template <int kGeo>
__global__ void __launch_bounds__(64) k_stress64(StepParams P, Fields F, Work64 W,
                                                  const double4* __restrict__ vd2,
                                                  const int32_t* __restrict__ nb,
                                                  const int32_t* __restrict__ cnt,
                                                  int* __restrict__ status) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double4 xi = F.xm[i];
  const double4 vi = vd2[i];
  // PressureKernelExt runs over every particle (EOS case 0, P0 = 0)
  F.p[i] = 0.0 + (P.Cs * P.Cs) * (vi.w - P.rho0);
  if (F.perm[i] >= P.n_solid) {
    keep_sigma(F, W, i, vi.w);
    return;
  }
  double r[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int c = cnt[i];
  for (int k = 0; k < c; k++) {
    const int64_t e = nb_at(P.npad, i, k);
    const int j = __ldg(nb + e);
    if (P.contact && !pass_j(P, F.id[j])) continue;
    double t[9];
    stress_terms<kGeo>(P, F, W, vd2, e, j, xi, vi, t);
#pragma unroll
    for (int a = 0; a < 9; a++) r[a] += t[a];
  }
  store_rates(F, i, r);
  stress_point(P, F, W, i, vi.w, r, status);
}

// Eight lanes per particle: the pair loop alone (the rates go to sr6, rr6).
// The stress update is a kernel of its own, one lane per particle: behind the
// pair loop it would run on 4 of a warp's 32 lanes.
template <int kGeo>
__global__ void __launch_bounds__(32) k_rates64(StepParams P, Fields F, Work64 W,
                                                const double4* __restrict__ vd2,
                                                const int32_t* __restrict__ nb,
                                                const int32_t* __restrict__ cnt) {
  __shared__ double sh[32 * 9];
  int g;
  const int64_t i0 = slot64<kLanes64>(g);
  const bool solid = i0 < P.n && F.perm[i0] < P.n_solid;
  const int64_t i = solid ? i0 : 0;
  const double4 xi = F.xm[i];
  const double4 vi = vd2[i];
  const int c = solid ? cnt[i] : 0;
  const int blocks = warp_blocks(c);
  double acc[2] = {0.0, 0.0};
  for (int b = 0; b < blocks; b++) {
    double t[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (WF_NB_BLK * b + g < c) {
      const int64_t e = nb_at(P.npad, i, WF_NB_BLK * b + g);
      const int j = __ldg(nb + e);
      if (!P.contact || pass_j(P, F.id[j])) stress_terms<kGeo>(P, F, W, vd2, e, j, xi, vi, t);
    }
    add_in_order<9>(sh, t, g, acc);
  }
  if (!solid) return;
  // accumulators 0-5 are D (sr6), 6-8 W (rr6 3-5); rr6 0-2 are zero
  if (g < 6) F.sr6[6 * i + g] = acc[0];
  else F.rr6[6 * i + g - 3] = acc[0];
  if (g == 0) F.rr6[6 * i + 5] = acc[1];
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
    keep_sigma(F, W, i, rho);
    return;
  }
  const double* sr = F.sr6 + 6 * i;
  const double* rr = F.rr6 + 6 * i;
  const double r[9] = {sr[0], sr[1], sr[2], sr[3], sr[4], sr[5], rr[3], rr[4], rr[5]};
  stress_point(P, F, W, i, rho, r, status);
}

// ---- C: Domain_d::CalcAccel (src/cuda/InteractionAlt.cu:18-150) ---------
// si = sigma_i / rho_i^2 (xx yy zz xy yz xz)
template <int kGeo>
__device__ __forceinline__ void accel_terms(const StepParams& P, const Fields& F, const Work64& W,
                                            const double4* __restrict__ vd2, int64_t e, int j,
                                            const double4& xi, const double4& vi, const double* si,
                                            double* t) {
  const double4 xj = F.xm[j];
  const double4 vj = vd2[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  const double di = vi.w, dj = vj.w, mj = xj.w;
  const double vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
  double GK, r2;
  double2 s01, s23, s45;
  if constexpr (kGeo == GEO_NONE) {
    pair_geometry(P, xx, xy, xz, GK, r2);
    const double2* q = reinterpret_cast<const double2*>(F.sig6 + 6 * (int64_t)j);
    const double aj = 1.0 / (dj * dj);
    s01 = make_double2(q[0].x * aj, q[0].y * aj);
    s23 = make_double2(q[1].x * aj, q[1].y * aj);
    s45 = make_double2(q[2].x * aj, q[2].y * aj);
  } else {
    GK = __ldg(W.gk + e);
    r2 = __ldg(W.r2 + e);
    const double2* q = reinterpret_cast<const double2*>(W.sa6 + 6 * (int64_t)j);
    s01 = q[0]; s23 = q[1]; s45 = q[2];
  }
  // Si/di^2 + Sj/dj^2 + PI*I, times mj, then times GK*xij (tensor3.cu:225)
  double Txx = si[0] + s01.x, Tyy = si[1] + s01.y, Tzz = si[2] + s23.x;
  const double Txy = si[3] + s23.y, Tyz = si[4] + s45.x, Txz = si[5] + s45.y;
  if (P.alpha != 0.0 || P.beta != 0.0) {
    const double vdx = vx * xx + vy * xy + vz * xz;
    if (vdx < 0) {
      const double MU = P.h * vdx / (r2 + 0.01 * P.h * P.h);
      const double Cij = 0.5 * (P.Cs + P.Cs);
      const double PI = (P.alpha * Cij * MU + P.beta * MU * MU) / (0.5 * (di + dj));
      Txx = Txx + PI;
      Tyy = Tyy + PI;
      Tzz = Tzz + PI;
    }
  }
  const double gx = xx * GK, gy = xy * GK, gz = xz * GK;
  const double Mxx = Txx * mj, Myy = Tyy * mj, Mzz = Tzz * mj;
  const double Mxy = Txy * mj, Myz = Tyz * mj, Mxz = Txz * mj;
  t[0] = Mxx * gx + Mxy * gy + Mxz * gz;
  t[1] = Mxy * gx + Myy * gy + Myz * gz;
  t[2] = Mxz * gx + Myz * gy + Mzz * gz;
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
  const int c = solid ? cnt[i] : 0;
  double t[3];
  if constexpr (kG == 1) {
    double a[3] = {0.0, 0.0, 0.0};
    for (int k = 0; k < c; k++) {
      const int64_t e = nb_at(P.npad, i, k);
      const int j = __ldg(nb + e);
      if (P.contact && !pass_ij(P, idi, F.id[j])) continue;
      accel_terms<kGeo>(P, F, W, vd2, e, j, xi, vi, si, t);
      a[0] += t[0]; a[1] += t[1]; a[2] += t[2];
    }
    F.a[i] = make_double4(a[0], a[1], a[2], 0.0);
  } else {
    const int blocks = warp_blocks(c);
    double acc[2] = {0.0, 0.0};
    for (int b = 0; b < blocks; b++) {
      t[0] = t[1] = t[2] = 0.0;
      if (WF_NB_BLK * b + g < c) {
        const int64_t e = nb_at(P.npad, i, WF_NB_BLK * b + g);
        const int j = __ldg(nb + e);
        if (!P.contact || pass_ij(P, idi, F.id[j]))
          accel_terms<kGeo>(P, F, W, vd2, e, j, xi, vi, si, t);
      }
      add_in_order<3>(sh, t, g, acc);
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
template <int kGeo>
__device__ __forceinline__ double heat_term(const StepParams& P, const Fields& F, const Work64& W,
                                            int64_t e, int j, const double4& xi, double Ti,
                                            double kk) {
  const double4 xj = F.xm[j];
  const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
  double GK, r2;
  geometry<kGeo>(P, W, e, xx, xy, xz, GK, r2);
  const double mj_dj = W.mr_heat ? __ldg(W.mr_heat + j) : xj.w / F.vd[j].w;
  return mj_dj * (kk * (Ti - F.T[j])) *
         (xx * (xx * GK) + xy * (xy * GK) + xz * (xz * GK)) / r2;
}

template <int kG, int kGeo>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_heat_rate(StepParams P, Fields F, Work64 W,
                                                   const int32_t* __restrict__ nb,
                                                   const int32_t* __restrict__ cnt,
                                                   int plastic_heat) {
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
      s += heat_term<kGeo>(P, F, W, e, __ldg(nb + e), xi, Ti, kk);
    }
  } else {
    const int blocks = warp_blocks(c);
    for (int b = 0; b < blocks; b++) {
      double t = 0.0;
      if (WF_NB_BLK * b + g < c) {
        const int64_t e = nb_at(P.npad, i, WF_NB_BLK * b + g);
        t = heat_term<kGeo>(P, F, W, e, __ldg(nb + e), xi, Ti, kk);
      }
      s = add_in_order(s, t);
    }
    if (!valid || g != 0) return;
  }
  F.dTdt[i] = heat_rate_fp64(P, F, i, s, rhoi, xi.w, Ti, plastic_heat);
}


// ---- ThermalSolve in FP64 (src/cuda/Thermal.cu:188-260) --------------------
// Positions, densities and lists do not change inside a heat solve, so what a
// pair contributes apart from the temperatures is computed once per solve:
// the product of the position difference with the kernel gradient, r^2 and
// its reciprocal (three arrays of the lists' layout), m / rho, and the
// particle's own factors.  A step is then eight FP64 operations a pair instead
// of 90 (the FP64 pipe bounds both: 64,000 particles 761 -> 68 us a step, 80 %
// of the pipe's peak; the factors take 364 us a solve) and takes the leapfrog
// update with it; the neighbours' temperatures are read
// from one array while the new ones go to another.
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
    const int64_t e = nb_at(P.npad, i, k);
    const double4 xj = F.xm[__ldg(nb + e)];
    const double xx = xi.x - xj.x, xy = xi.y - xj.y, xz = xi.z - xj.z;
    double GK, r2;
    pair_geometry(P, xx, xy, xz, GK, r2);
    H.dot[e] = xx * (xx * GK) + xy * (xy * GK) + xz * (xz * GK);
    H.r2[e] = r2;
    H.ir2[e] = 1.0 / r2;
  }
}

__device__ __forceinline__ double heat_step_term(const HeatWork64& H, const double* __restrict__ T,
                                                 int64_t e, int j, double Ti, double kk) {
  const double num = __ldg(H.mr + j) * (kk * (Ti - __ldg(T + j))) * __ldg(H.dot + e);
  const double r2 = __ldg(H.r2 + e), y = __ldg(H.ir2 + e);
  // zero and the middle of the range divide by the known reciprocal
  const bool easy = mid_range(num) || ((__double2hiint(num) << 1) | __double2loint(num)) == 0;
  return easy && mid_range(y) ? div_known(num, r2, y) : num / r2;
}

template <int kG>
__global__ void __launch_bounds__(kG == 1 ? 64 : 32) k_heat_step64(StepParams P, Fields F,
                                                     HeatWork64 H, const double* __restrict__ T,
                                                     double* __restrict__ T_out,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt, int first) {
  int g;
  const int64_t i0 = slot64<kG>(g);
  if (kG == 1 && i0 >= P.n) return;
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : 0;
  const double Ti = T[i], ki = F.kT[i];
  const double kk = 4.0 * ki * ki / (ki + ki);
  const int c = valid ? cnt[i] : 0;
  double s = 0.0;
  if constexpr (kG == 1) {
    for (int k = 0; k < c; k++) {
      const int64_t e = nb_at(P.npad, i, k);
      s += heat_step_term(H, T, e, __ldg(nb + e), Ti, kk);
    }
  } else {
    const int blocks = warp_blocks(c);
    for (int b = 0; b < blocks; b++) {
      double t = 0.0;
      if (WF_NB_BLK * b + g < c) {
        const int64_t e = nb_at(P.npad, i, WF_NB_BLK * b + g);
        t = heat_step_term(H, T, e, __ldg(nb + e), Ti, kk);
      }
      s = add_in_order(s, t);
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

// Below this many particles eight lanes share one (see kLanes64).
constexpr int64_t kWide64 = 24000;

// Launches K<lanes, geometry> with one or eight lanes per particle.
#define WF_LAUNCH64(K, GEO, ...)                                                               \
  do {                                                                                         \
    if (P.n < kWide64)                                                                         \
      K<kLanes64, GEO><<<blocks_for(P.n * kLanes64, 32), 32, 0, s>>>(P, F, W, __VA_ARGS__);    \
    else                                                                                       \
      K<1, GEO><<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, W, __VA_ARGS__);                      \
  } while (0)

void launch_fp64_density(const StepParams& P, const Fields& F, const Work64& W, double4* vd2,
                         const NbBuffers& N, cudaStream_t s) {
  if (!W.gk) WF_LAUNCH64(k_density64, GEO_NONE, vd2, N.nb, N.cnt);
  else if (W.geo) WF_LAUNCH64(k_density64, GEO_LOAD, vd2, N.nb, N.cnt);
  else WF_LAUNCH64(k_density64, GEO_STORE, vd2, N.nb, N.cnt);
}
int launch_fp64_stress(const StepParams& P, const Fields& F, const Work64& W, const double4* vd2,
                       const NbBuffers& N, int* status, cudaStream_t s) {
  if (P.n < kWide64) {
    const int blocks = blocks_for(P.n * kLanes64, 32);
    if (W.gk) k_rates64<GEO_LOAD><<<blocks, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
    else k_rates64<GEO_NONE><<<blocks, 32, 0, s>>>(P, F, W, vd2, N.nb, N.cnt);
    k_stress_point64<<<blocks_for(P.n, 32), 32, 0, s>>>(P, F, W, vd2, status);
    return 2;
  }
  if (W.gk) k_stress64<GEO_LOAD><<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, W, vd2, N.nb, N.cnt, status);
  else k_stress64<GEO_NONE><<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, W, vd2, N.nb, N.cnt, status);
  return 1;
}
void launch_fp64_accel(const StepParams& P, const Fields& F, const Work64& W, const double4* vd2,
                       const NbBuffers& N, cudaStream_t s) {
  if (W.gk) WF_LAUNCH64(k_accel64, GEO_LOAD, vd2, N.nb, N.cnt);
  else WF_LAUNCH64(k_accel64, GEO_NONE, vd2, N.nb, N.cnt);
}
void launch_fp64_heat_rate(const StepParams& P, const Fields& F, const Work64& W,
                           const NbBuffers& N, int plastic_heat, cudaStream_t s) {
  if (W.gk) WF_LAUNCH64(k_heat_rate, GEO_STORE, N.nb, N.cnt, plastic_heat);
  else WF_LAUNCH64(k_heat_rate, GEO_NONE, N.nb, N.cnt, plastic_heat);
}
void launch_heat_pairs64(const StepParams& P, const Fields& F, const HeatWork64& H,
                         const NbBuffers& N, cudaStream_t s) {
  k_heat_pairs64<<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, H, N.nb, N.cnt);
}
void launch_heat_step64(const StepParams& P, const Fields& F, const HeatWork64& H, double* T_out,
                        const NbBuffers& N, int first, cudaStream_t s) {
  if (P.n < kWide64)
    k_heat_step64<kLanes64><<<blocks_for(P.n * kLanes64, 32), 32, 0, s>>>(P, F, H, F.T, T_out,
                                                                          N.nb, N.cnt, first);
  else
    k_heat_step64<1><<<blocks_for(P.n, 64), 64, 0, s>>>(P, F, H, F.T, T_out, N.nb, N.cnt, first);
}
