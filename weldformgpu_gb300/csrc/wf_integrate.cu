// wf_integrate.cu — per-particle integration and heat conduction kernels.
//
// Compiled with -fmad=false: the FP64 leapfrog, position and temperature
// updates round exactly like the reference (--fmad=false).
#include "wf_common.cuh"
#include "wf_heat.cuh"
#include "wf_integrate.cuh"

namespace {

// ---- D: BC, UpdatePosFraser, UpdateVel, BC, CalcIntEnergy ---------------
// GeneralAfter/ApplyBCVel (src/WeldFormGPU.cu:103-106, src/cuda/Mechanical.cu:572-584),
// UpdatePosFraser (:179-187), UpdateVel (:142-148), CalcIntEnergy
// (src/cuda/Energy.cu:5-19), in SolverFraser.cu:273-287 order.
// The blocks behind the particles' move the rigid meshes' nodes (nothing here
// reads them), which saves a launch per mesh.
__global__ void __launch_bounds__(256) k_integrate(StepParams P, Fields F,
                                                   const double4* __restrict__ vd2,
                                                   const float4* __restrict__ a32) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) {
    int b = (int)blockIdx.x - (int)((P.n + blockDim.x - 1) / blockDim.x);
    if (b < 0) return;
    for (int m = 0; m < P.ncsid; m++) {
      const int blocks = (P.mesh[m].nn + (int)blockDim.x - 1) / (int)blockDim.x;
      if (b < blocks) return mesh_move_one(P.mesh[m], P.dt, b * (int)blockDim.x + (int)threadIdx.x);
      b -= blocks;
    }
    return;
  }
  if (a32) {
    // rigid (non-solid) slots keep the acceleration the BCs left (zero)
    const float4 af = F.perm[i] < P.n_solid ? a32[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    integrate_mixed_one(P, F, vd2, i, af);
    return;
  }
  double4 xm = F.xm[i];
  const double4 v4 = vd2[i];
  const double4 a4 = F.a[i];
  const int32_t id = F.id[i];
  double vx = v4.x, vy = v4.y, vz = v4.z, ax = a4.x, ay = a4.y, az = a4.z;
  record_bc_force(P, i, id, xm.w, ax, ay, az);
  apply_bc(P, id, vx, vy, vz, ax, ay, az);
  const double dt = P.dt;
  const double ux = vx * dt + ((ax * 0.5) * dt) * dt;
  const double uy = vy * dt + ((ay * 0.5) * dt) * dt;
  const double uz = vz * dt + ((az * 0.5) * dt) * dt;
  xm.x = xm.x + ux; xm.y = xm.y + uy; xm.z = xm.z + uz;
  double4 u = F.u[i];
  u.x = u.x + ux; u.y = u.y + uy; u.z = u.z + uz;
  vx = vx + ax * dt; vy = vy + ay * dt; vz = vz + az * dt;
  apply_bc(P, id, vx, vy, vz, ax, ay, az);
  // energy_mode 0 reads particle 0's tensors for every particle, like the
  // reference; mode 1 uses each particle's own.
  const bool own = P.energy_mode != 0;
  if (!own || F.perm[i] < P.n_solid) {
    const double* ss = F.ss6 + 6 * (own ? i : (int64_t)P.inv[0]);
    const double* sr = F.sr6 + 6 * (own ? i : (int64_t)P.inv[0]);
    const double de = xm.w / v4.w *
                      (ss[0] * sr[0] + ss[1] * sr[1] + ss[2] * sr[2] +
                       2.0 * (ss[3] * sr[3] + ss[4] * sr[4] + ss[5] * sr[5]));
    F.eint[i] += de * dt;
  }
  F.xm[i] = xm;
  F.vd[i] = make_double4(vx, vy, vz, v4.w);
  F.u[i] = u;
  F.a[i] = make_double4(ax, ay, az, 0.0);
}

// TempCalcLeapfrogFirst / TempCalcLeapfrog (src/cuda/Thermal.cu:16-31)
__global__ void __launch_bounds__(256) k_heat_leapfrog(StepParams P, Fields F, int first,
                                                       int mixed) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double T = heat_leapfrog_one(P, F, i, F.dTdt[i], first);
  if (mixed && !first) {
    const float thi = (float)T;
    F.pv[i].v.w = thi;
    F.tl32[i] = (float)(T - (double)thi);
  }
}

}  // namespace

static inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }
// Threads of a block: one warp in domains that give no SM two blocks of 256,
// so that their few FP64 operations run on every SM (540 particles: integration
// 7.5 -> 6.3 us).
static inline int threads64(int64_t n) { return n < 77824 ? 32 : 256; }

void launch_integrate(const StepParams& P, const Fields& F, const double4* vd2,
                      const float4* a32, cudaStream_t s) {
  const int t = threads64(P.n);
  int grid = blocks_for(P.n, t);
  for (int m = 0; P.contact && m < P.ncsid; m++) grid += blocks_for(P.mesh[m].nn, t);
  k_integrate<<<grid, t, 0, s>>>(P, F, vd2, a32);
}

void launch_thermal(const StepParams& P, const Fields& F, const Work64& W, const NbBuffers& N,
                    int first, int plastic_heat, int mixed, cudaStream_t s) {
  if (mixed) launch_fp32_heat(P, F, N, plastic_heat, s);
  else launch_fp64_heat_rate(P, F, W, N, plastic_heat, s);
  const int t = threads64(P.n);
  k_heat_leapfrog<<<blocks_for(P.n, t), t, 0, s>>>(P, F, first, mixed);
}
