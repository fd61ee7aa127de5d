// wf_step_fp32.cu — mixed-precision form of the Fraser step.
//
// Pair loops, the Jaumann/J2 stress update and the heat flux run in FP32 with
// FP32 accumulation in the fixed neighbour order.  Kept in FP64 (they sum
// ~1e-7 s increments over long runs): positions, displacements, velocities
// and their update, density accumulation, equivalent plastic strain, yield
// stress and the Newton residual, and every reduction.  The gathered
// neighbour data are 32-byte FP32 records (Rec32): pv = (x, m/rho | v, T_hi) with
// T_lo beside it, written by the integration, for the density + heat pass;
// pvb = (x, m | v, rho_new), written by the density pass, for the stress and
// acceleration passes; sig = stress / rho^2, written by the stress pass.
// All FP32 constants arrive precomputed in StepParams: on GB300 a per-thread
// FP64 division or conversion costs as much as the whole FP32 pair loop.
#include "wf_common.cuh"
#include "wf_heat.cuh"
#include "wf_integrate.cuh"
#include "wf_mlp.cuh"
#include "wf_tensor.cuh"
#include "wf_tiles.cuh"

namespace {

struct T3f {
  float xx, xy, xz, yx, yy, yz, zx, zy, zz;
};

// operator*(tensor3, tensor3) of src/cuda/tensor3.cu:241-256 in FP32
__device__ __forceinline__ T3f mul_ref_f(const T3f& a, const T3f& b) {
  T3f r;
  r.xx = a.xx * b.xx + a.xy * b.yx + a.xz * b.zx;
  r.xy = a.xx * b.yx + a.xy * b.yy + a.xz * b.yz;
  r.xz = a.xx * b.zx + a.xy * b.zy + a.xz * b.zz;
  r.yx = a.yx * b.xx + a.yy * b.yx + a.yz * b.zx;
  r.yy = a.yx * b.yx + a.yy * b.yy + a.yz * b.yz;
  r.yz = a.yx * b.zx + a.yy * b.zy + a.yz * b.zz;
  r.zx = a.zx * b.xx + a.zy * b.yx + a.zz * b.zx;
  r.zy = a.zx * b.yx + a.zy * b.yy + a.zz * b.yz;
  r.zz = a.zx * b.zx + a.zy * b.zy + a.zz * b.zz;
  return r;
}

// Neighbour records by slot from global memory or by halo rank from a staged
// tile's shared memory.
struct RecGlobal {
  const Rec32* r;
  __device__ __forceinline__ Rec32 get(int j) const { return rec_load(r + j); }
};
struct RecShared {
  const float4* p;
  const float4* v;
  __device__ __forceinline__ Rec32 get(int j) const { return Rec32{p[j], v[j]}; }
};

// ---- A32: density rate + update (InteractionAlt.cu:166-246, Mechanical.cu:198) --
// Lane groups of the pair passes: kLanes consecutive lanes share one particle;
// lane g of the group takes entries [8b + g W, 8b + (g + 1) W) of every list
// block b (W = 8 / kLanes, the list readers' sub<W>), and the lanes' partial
// sums are combined by an xor-shuffle tree, which gives every lane of the
// group the same value.  A warp then covers fewer particles and its gathers
// touch fewer L1 lines (the neighbours of consecutive sorted particles
// overlap), and each lane's chain of dependent gathers is shorter.

// lane group of G lanes (a power of two) that share one particle
template <int G>
__device__ __forceinline__ unsigned group_mask() {
  if constexpr (G == 32) return 0xffffffffu;
  return ((1u << G) - 1u) << ((threadIdx.x & 31u) & ~(unsigned)(G - 1));
}

// Blocks per SM that a pass is compiled for (kWide: few blocks, so many
// registers per thread and the compiler keeps more loads in flight; else many
// blocks).  A grid of at most four blocks per SM runs in one wave whatever the
// bound, and what it waits for is each thread's own chain of loads: 10,752
// particles 14.5 -> 12.5 us stress, 16.9 -> 14.8 acceleration, 46.3 -> 42.4 a
// step, while 50,560 (more than one wave of the acceleration pass's two lanes
// per particle) lose 27 -> 35 us there.
constexpr int kWideBlocks = 4;

// Density + heat pass: one lane per particle (786k particles: 0.199 ms with
// one lane and 6 blocks per SM, 0.202-0.213 ms with 2 or 4 lanes).
constexpr int kDensLanes = 1;
constexpr int kDensMinBlocks = 6;
constexpr int kDensBatch = 4;

// ---- A32 + heat: the previous step's heat pass fused into this density pass.
// Heat at the end of step n (ThermalSolveKernel + plastic heat + convection +
// leapfrog, src/cuda/Thermal.cu:16-142) and the density pass of step n+1 read
// the same positions x^{n+1}, velocities and densities, so one walk over the
// neighbour list serves both.  Neighbour temperatures come from the th32
// mirror (T^n, written by the integration kernel), so each thread may update
// its own FP64 temperature in place.  After a rebuild at the start of step
// n+1 the heat flux of step n uses the new list (built for these positions).
// The pair loop of the density + heat pass over the neighbour list L: its
// entries are slots (NbList32 / NbList16: records gathered from the global
// arrays) or ranks in the tile's halo (NbListS: the arrays are its
// shared-memory copies).
template <bool kFilter, bool kHeat, class L, class R>
__device__ __forceinline__ void density_heat_pairs(const StepParams& P, const Fields& F,
                                                   const R& rec, const float* __restrict__ gt,
                                                   const L& list, int g, int c, float4 pi,
                                                   float4 vi, float2 ti,
                                                   bool solid, int32_t idi, float& drho_out,
                                                   float& sf_out) {
  constexpr int W = WF_NB_BLK / kDensLanes;
  constexpr int NB = W < kDensBatch ? W : kDensBatch;   // neighbours gathered per batch
  const float invh = P.invhf, C = P.Cf, Ch = P.Chf;
  float drho = 0.0f, sf = 0.0f;
  int nx[W];
  if (c > 0) list.template sub<W>(0, g, nx);
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    int js[W];
#pragma unroll
    for (int q = 0; q < W; q++) js[q] = nx[q];
    const int m = c - WF_NB_BLK * b - g * W;   // entries of this lane's sub-block in the list
    if (P.nb_pf && c > WF_NB_BLK * (b + P.nb_pf)) list.prefetch(b + P.nb_pf, kDensLanes);
    if (c > WF_NB_BLK * (b + 1)) list.template sub<W>(b + 1, g, nx);
#pragma unroll
    for (int h = 0; h < W; h += NB) {
      float4 pj[NB], vj[NB];
      float tj[NB];
#pragma unroll
      for (int q = 0; q < NB; q++) {
        const Rec32 r = rec.get(js[h + q]);
        pj[q] = r.p;
        vj[q] = r.v;
        if constexpr (kHeat) tj[q] = gt[js[h + q]];
      }
#pragma unroll
      for (int q = 0; q < NB; q++) {
        // Entries past the count are the particle's own slot (list padding):
        // r^2 = 0 gives GK = 0 exactly (gk32_r2), so they add exact zeros and
        // need no test, except under the zone filter.
        if (kFilter && h + q >= m) continue;
        const float xx = pi.x - pj[q].x, xy = pi.y - pj[q].y, xz = pi.z - pj[q].z;
        const float GK = gk32_r2(xx * xx + xy * xy + xz * xz, invh, Ch, C);
        // m_j / rho_j GK, shared by both sums
        const float mg = pj[q].w * GK;
        // heat flux (every particle, no contact filter); the pair
        // conductivity 4 k_i k_j / (k_i + k_j) = 2k multiplies the sum
        if constexpr (kHeat) {
          const float dT = (ti.x - vj[q].w) + (ti.y - tj[q]);
          sf += mg * dT;
        }
        // density rate (solid particles, contact filter); rho_i multiplies the sum
        bool pass = solid;
        if constexpr (kFilter) pass = pass && pass_ij(P, idi, F.id[js[h + q]]);
        if (pass) {
          const float vx = vi.x - vj[q].x, vy = vi.y - vj[q].y, vz = vi.z - vj[q].z;
          drho += mg * (vx * xx + vy * xy + vz * xz);
        }
      }
    }
  }
  drho_out = drho;             // rho_i multiplies it (caller)
  sf_out = sf;
}

// ---- A32: the density pass without a heat pass to fuse (a call's first
// step; every step when heat is off): the density sum of density_heat_pairs.
template <bool kWide>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : kDensMinBlocks) k_density32(StepParams P, Fields F,
                                                                  double4* __restrict__ vd2,
                                                                  Rec32* __restrict__ pvb,
                                                                  const int32_t* __restrict__ nb,
                                                                  const int32_t* __restrict__ cnt,
                                                                  const List16 L16) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const bool solid = F.perm[i] < P.n_solid;
  if (P.state_pf) prefetch_l2(F.vd + i);
  if (P.pf_ahead > 0) {
    const int64_t ia = i + P.pf_ahead;      // the slot this thread's successor will take
    if (ia < P.n) {
      prefetch_l2(F.pv + ia); prefetch_l2(cnt + ia);
      prefetch_l2(F.perm + ia);
      for (int b = 0; b < P.wave_pf && b < WF_NB_BLOCKS; b++) nb_prefetch(nb, P.npad, ia, b, 4);
    }
  }
  const Rec32 own = rec_load(F.pv + i);
  const float4 pi = own.p, vi = own.v;
  const int c = solid ? cnt[i] : 0;
  const int32_t idi = F.id[i];
  float drho = 0.0f, sf = 0.0f;
  const int b16 = L16.base ? L16.base[i / WF_TILE] : -1;     // uniform over the block
  const float2 t0 = make_float2(0.f, 0.f);
  const RecGlobal rec{F.pv};
  const NbList32 list{nb, P.npad, i};
  if (zone_filter(P))
    density_heat_pairs<true, false>(P, F, rec, nullptr, list, 0, c, pi, vi, t0, solid, idi, drho, sf);
  else if (b16 >= 0)
    density_heat_pairs<false, false>(P, F, rec, nullptr, NbList16{L16.off, P.npad, i, b16}, 0, c, pi,
                                     vi, t0, solid, idi, drho, sf);
  else
    density_heat_pairs<false, false>(P, F, rec, nullptr, list, 0, c, pi, vi, t0, solid, idi, drho,
                                     sf);
  const double4 vdi = F.vd[i];
  drho *= (float)vdi.w;
  double rho_new = vdi.w;
  if (solid) {
    F.drho[i] = (double)drho;
    rho_new = vdi.w + P.dt * (double)drho;
  }
  vd2[i] = make_double4(vdi.x, vdi.y, vdi.z, rho_new);
  pvb[i] = Rec32{make_float4(pi.x, pi.y, pi.z, F.m32[i]),
                 make_float4(vi.x, vi.y, vi.z, (float)rho_new)};
}

template <bool kWide>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : kDensMinBlocks) k_density_heat32(StepParams P, Fields F,
                                                        double4* __restrict__ vd2,
                                                        Rec32* __restrict__ pvb,
                                                        const int32_t* __restrict__ nb,
                                                        const int32_t* __restrict__ cnt,
                                                        int first, int plastic_heat,
                                                        const TileHalo T, const List16 L16) {
  // tile staging (one lane per particle: a block of 128 threads is one tile)
  extern __shared__ __align__(16) uint8_t sdh[];
  float4* sp = reinterpret_cast<float4*>(sdh);
  float4* sv = sp + T.cap;
  float* st = reinterpret_cast<float*>(sv + T.cap);
  uint16_t* sl = reinterpret_cast<uint16_t*>(sdh + density_lists_at(T.cap));
  int staged = -1;
  if (kDensLanes == 1 && T.cap > 0) {
    const float4* src = reinterpret_cast<const float4*>(F.pv);
    const int H = T.hcnt[blockIdx.x];
    if (H >= 0 && H <= T.cap) {                 // uniform over the block
      const int32_t* hs = T.halo + T.hoff[blockIdx.x];
      for (int k = threadIdx.x; k < H; k += blockDim.x) {
        const int s = hs[k];
        cp_async16(sp + k, src + 2 * (int64_t)s);
        cp_async16(sv + k, src + 2 * (int64_t)s + 1);
        cp_async4(st + k, F.tl32 + s);
      }
      stage_lists(T.nbl, P.npad, blockIdx.x, sl);
      cp_async_wait_all();
      __syncthreads();
      staged = H;
    }
  }
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int g = (int)(t & (kDensLanes - 1));
  const int64_t i = t / kDensLanes;
  if (i >= P.n) return;
  const Rec32 own = rec_load(F.pv + i);
  const float4 pi = own.p, vi = own.v;
  const float2 ti = make_float2(vi.w, F.tl32[i]);
  const bool solid = F.perm[i] < P.n_solid;
  const int32_t idi = F.id[i];
  if (P.state_pf && g == 0) {
    prefetch_l2(F.vd + i); prefetch_l2(F.T + i); prefetch_l2(F.cpT + i);
    prefetch_l2(F.dep + i); prefetch_l2(F.sy + i); prefetch_l2(F.Ta + i);
  }
  if (P.pf_ahead > 0 && g == 0) {
    const int64_t ia = i + P.pf_ahead;      // the slot this thread's successor will take
    if (ia < P.n) {
      prefetch_l2(F.pv + ia); prefetch_l2(F.tl32 + ia);
      prefetch_l2(cnt + ia); prefetch_l2(F.perm + ia);
      for (int b = 0; b < P.wave_pf && b < WF_NB_BLOCKS; b++) nb_prefetch(nb, P.npad, ia, b, 4);
    }
  }
  float drho, sf;
  const int c = cnt[i];
  const int b16 = L16.base ? L16.base[i / WF_TILE] : -1;     // uniform over the block
  const RecGlobal rec{F.pv};
  const NbList32 list{nb, P.npad, i};
  if (zone_filter(P))
    density_heat_pairs<true, true>(P, F, rec, F.tl32, list, g, c, pi, vi, ti, solid, idi, drho, sf);
  else if (staged >= 0)
    density_heat_pairs<false, true>(P, F, RecShared{sp, sv}, st, NbListS{sl, (int)threadIdx.x}, g, c,
                                    pi, vi, ti, solid, idi, drho, sf);
  else if (b16 >= 0)
    density_heat_pairs<false, true>(P, F, rec, F.tl32, NbList16{L16.off, P.npad, i, b16}, g, c, pi,
                                    vi, ti, solid, idi, drho, sf);
  else
    density_heat_pairs<false, true>(P, F, rec, F.tl32, list, g, c, pi, vi, ti, solid, idi, drho, sf);
  if constexpr (kDensLanes > 1) {
    const unsigned mask = group_mask<kDensLanes>();
#pragma unroll
    for (int o = 1; o < kDensLanes; o <<= 1) {
      sf += __shfl_xor_sync(mask, sf, o, kDensLanes);
      drho += __shfl_xor_sync(mask, drho, o, kDensLanes);
    }
  }
  if (g != 0) return;
  const double4 vdi = F.vd[i];
  drho *= (float)vdi.w;
  // heat of the previous step: rate and leapfrog, own particle only
  const double dTdt = heat_rate_mixed(P, F, i, P.k2f * sf, vdi.w, (double)F.m32[i], F.T[i],
                                      plastic_heat);
  F.dTdt[i] = dTdt;
  heat_leapfrog_one(P, F, i, dTdt, first);
  // density of this step
  double rho_new = vdi.w;
  if (solid) {
    F.drho[i] = (double)drho;
    rho_new = vdi.w + P.dt * (double)drho;
  }
  vd2[i] = make_double4(vdi.x, vdi.y, vdi.z, rho_new);
  pvb[i] = Rec32{make_float4(pi.x, pi.y, pi.z, F.m32[i]),
                 make_float4(vi.x, vi.y, vi.z, (float)rho_new)};
}

// ---- the heat pass alone (ThermalSolveKernel, src/cuda/Thermal.cu:101-142) --
// A call's last heat pass and every step of the mixed ThermalSolve: the heat
// sum of density_heat_pairs, the same operations in the same neighbour order
// (so a separate pass gives the fused pass's sum and dT/dt bit for bit; the
// temperature update behind it, k_heat_leapfrog, is compiled without FMA
// contraction, so some temperatures differ from the fused pass's in the last bit).
template <class L>
__device__ __forceinline__ float heat_pairs(const StepParams& P, const Rec32* __restrict__ pv,
                                            const float* __restrict__ gt, const L& list, int c,
                                            float4 pi, float2 ti) {
  constexpr int NB = kDensBatch;
  const float invh = P.invhf, C = P.Cf, Ch = P.Chf;
  float sf = 0.0f;
  int nx[WF_NB_BLK];
  if (c > 0) list.block(0, nx);
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    int js[WF_NB_BLK];
#pragma unroll
    for (int q = 0; q < WF_NB_BLK; q++) js[q] = nx[q];
    if (P.nb_pf && c > WF_NB_BLK * (b + P.nb_pf)) list.prefetch(b + P.nb_pf, 1);
    if (c > WF_NB_BLK * (b + 1)) list.block(b + 1, nx);
#pragma unroll
    for (int h = 0; h < WF_NB_BLK; h += NB) {
      float4 pj[NB];
      float2 tj[NB];
#pragma unroll
      for (int q = 0; q < NB; q++) {
        const Rec32 r = rec_load(pv + js[h + q]);
        pj[q] = r.p;
        tj[q] = make_float2(r.v.w, gt[js[h + q]]);
      }
#pragma unroll
      for (int q = 0; q < NB; q++) {
        // padding entries (the particle's own slot) add exact zeros (gk32_r2)
        const float xx = pi.x - pj[q].x, xy = pi.y - pj[q].y, xz = pi.z - pj[q].z;
        const float GK = gk32_r2(xx * xx + xy * xy + xz * xz, invh, Ch, C);
        const float mg = pj[q].w * GK;
        const float dT = (ti.x - tj[q].x) + (ti.y - tj[q].y);
        sf += mg * dT;
      }
    }
  }
  return sf;
}

__global__ void __launch_bounds__(128, kDensMinBlocks) k_heat32(StepParams P, Fields F,
                                                               const int32_t* __restrict__ nb,
                                                               const int32_t* __restrict__ cnt,
                                                               int plastic_heat) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  if (P.state_pf) {
    prefetch_l2(F.vd + i); prefetch_l2(F.xm + i); prefetch_l2(F.T + i); prefetch_l2(F.cpT + i);
    prefetch_l2(F.dep + i); prefetch_l2(F.sy + i);
  }
  if (P.pf_ahead > 0) {
    const int64_t ia = i + P.pf_ahead;      // the slot this thread's successor will take
    if (ia < P.n) {
      prefetch_l2(F.pv + ia); prefetch_l2(F.tl32 + ia); prefetch_l2(cnt + ia);
      for (int b = 0; b < P.wave_pf && b < WF_NB_BLOCKS; b++) nb_prefetch(nb, P.npad, ia, b, 4);
    }
  }
  const Rec32 own = rec_load(F.pv + i);
  const float4 pi = own.p;
  const float2 ti = make_float2(own.v.w, F.tl32[i]);
  const int c = cnt[i];
  const float sf = heat_pairs(P, F.pv, F.tl32, NbList32{nb, P.npad, i}, c, pi, ti);
  F.dTdt[i] = heat_rate_mixed(P, F, i, P.k2f * sf, F.vd[i].w, F.xm[i].w, F.T[i], plastic_heat);
}

// ---- ThermalSolve in the mixed form (src/cuda/Thermal.cu:188-260) ---------
// Positions, densities and lists do not change inside a heat solve, so the
// pair factor m_j / rho_j GK of heat_pairs is computed once per solve (one
// float per list entry, padding entries 0) and a step gathers 8 bytes a
// neighbour, its temperature, instead of 28; the particle's own factors are
// kept too (heat_rate_mixed), and the leapfrog update rides in the same pass:
// the neighbours' temperatures are read from one mirror while the new ones go
// to another.  T, Tb and dT/dt feed nothing inside a solve and are written by
// its last step only.  Same operations in the same order as k_heat32 and
// k_heat_leapfrog.
// A step streams the lists and factors and is bound by HBM, so the lists are
// kept as 16-bit offsets from the tile's smallest slot where they span no more
// than 65,536 (in cell order a tile's lists reach one cell layer down and up:
// boxes up to ~115 particles a side; other tiles keep the 32-bit lists):
// 428 bytes a particle instead of 556, a million particles 80 -> 75 us a step
// (70 with lists and factors read past L1; 48 registers, and a bound that
// forces fewer spills: 12 blocks an SM 88 us; blocks of 256 72 us).
__global__ void __launch_bounds__(128) k_heat_pairs32(StepParams P, Fields F, HeatWork32 H,
                                                      const int32_t* __restrict__ nb,
                                                      const int32_t* __restrict__ cnt) {
  static_assert(WF_TILE == 128, "a block is a tile");
  __shared__ int s_lo[4], s_hi[4];
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : P.n - 1;
  const int c = valid ? cnt[i] : 0;
  const NbList32 list{nb, P.npad, i};
  // the tile's smallest and largest slot
  int lo = (int)i, hi = (int)i;
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    int js[WF_NB_BLK];
    list.block(b, js);
#pragma unroll
    for (int q = 0; q < WF_NB_BLK; q++) {
      lo = min(lo, js[q]);
      hi = max(hi, js[q]);
    }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) { s_lo[threadIdx.x >> 5] = lo; s_hi[threadIdx.x >> 5] = hi; }
  __syncthreads();
  for (int w = 0; w < 4; w++) { lo = min(lo, s_lo[w]); hi = max(hi, s_hi[w]); }
  const bool near = hi - lo < 65536;
  if (threadIdx.x == 0) H.base[blockIdx.x] = near ? lo : -1;
  if (!valid) return;
  const float4 pi = F.pv[i].p;
  const float invh = P.invhf, C = P.Cf, Ch = P.Chf;
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    int js[WF_NB_BLK];
    float mg[WF_NB_BLK];
    list.block(b, js);
    if (near)
      *reinterpret_cast<uint4*>(H.off + ((int64_t)b * P.npad + i) * WF_NB_BLK) =
          make_uint4((unsigned)(js[0] - lo) | (unsigned)(js[1] - lo) << 16,
                     (unsigned)(js[2] - lo) | (unsigned)(js[3] - lo) << 16,
                     (unsigned)(js[4] - lo) | (unsigned)(js[5] - lo) << 16,
                     (unsigned)(js[6] - lo) | (unsigned)(js[7] - lo) << 16);
#pragma unroll
    for (int q = 0; q < WF_NB_BLK; q++) {
      const float4 pj = __ldg(&F.pv[js[q]].p);
      const float xx = pi.x - pj.x, xy = pi.y - pj.y, xz = pi.z - pj.z;
      const float GK = gk32_r2(xx * xx + xy * xy + xz * xz, invh, Ch, C);
      mg[q] = pj.w * GK;
    }
    float4* out = reinterpret_cast<float4*>(H.mg + ((int64_t)b * P.npad + i) * WF_NB_BLK);
    out[0] = make_float4(mg[0], mg[1], mg[2], mg[3]);
    out[1] = make_float4(mg[4], mg[5], mg[6], mg[7]);
  }
  const float rf = (float)F.vd[i].w, cpf = (float)F.cpT[i], mf = (float)F.xm[i].w;
  float conv = 0.0f, fric = 0.0f;
  if (F.bct[i] == 1) conv = P.h_convf * powf(mf / rf, 0.666666666f);
  if (F.qf && F.qf[i] > 0.0) fric = (float)F.qf[i] / (mf * cpf);
  H.own[i] = make_float4(rf * cpf, conv, mf * cpf, fric);
}

// four values read once: past L1
__device__ __forceinline__ void ld_stream4(const float* p, float* v) {
  asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
      : "l"(p));
}
// the heat sum from the kept factors over the list L
template <class L>
__device__ __forceinline__ float heat_step_pairs(const float* __restrict__ factors,
                                                 const float2* __restrict__ th, const L& list,
                                                 int64_t npad, int64_t i, int c, float2 ti) {
  float sf = 0.0f;
  int nx[WF_NB_BLK];
  if (c > 0) list.block(0, nx);
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    float2 tj[WF_NB_BLK];
#pragma unroll
    for (int q = 0; q < WF_NB_BLK; q++) tj[q] = __ldg(th + nx[q]);
    float mg[WF_NB_BLK];
    const float* f = factors + ((int64_t)b * npad + i) * WF_NB_BLK;
    ld_stream4(f, mg);
    ld_stream4(f + 4, mg + 4);
    if (c > WF_NB_BLK * (b + 1)) list.block(b + 1, nx);
#pragma unroll
    for (int q = 0; q < WF_NB_BLK; q++) {
      const float dT = (ti.x - tj[q].x) + (ti.y - tj[q].y);
      sf += mg[q] * dT;
    }
  }
  return sf;
}

constexpr int kHeatStepThreads = 128;
__global__ void __launch_bounds__(kHeatStepThreads) k_heat_step32(StepParams P, Fields F, HeatWork32 H,
                                                     const float2* __restrict__ th,
                                                     float2* __restrict__ th_out,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt, int first,
                                                     int last) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const float2 ti = th[i];
  const int c = cnt[i];
  const int b16 = H.base[i / WF_TILE];         // uniform over the warp
  const float sf =
      b16 >= 0 ? heat_step_pairs(H.mg, th, NbList16{H.off, P.npad, i, b16}, P.npad, i, c, ti)
               : heat_step_pairs(H.mg, th, NbList32{nb, P.npad, i}, P.npad, i, c, ti);
  const float4 own = H.own[i];
  float sm = P.k2f * sf / own.x;
  if (own.w > 0.0f) sm += own.w;
  if (own.y != 0.0f) sm += own.y * (P.T_inff - ti.x) / own.z;
  const double rate = (double)sm, dt = P.dt;
  if (first) {
    F.Ta[i] = __dsub_rn(F.T[i], __dmul_rn(dt / 2.0, rate));
    if (last) F.dTdt[i] = rate;
    th_out[i] = ti;
    return;
  }
  const double ta = F.Ta[i];
  const double ta2 = __dadd_rn(ta, __dmul_rn(rate, dt));
  F.Ta[i] = ta2;
  const double T = __dmul_rn(__dadd_rn(ta2, ta), 0.5);
  const float thi = (float)T;
  th_out[i] = make_float2(thi, (float)(T - (double)thi));
  if (last) {
    F.T[i] = T;
    F.Tb[i] = ta;
    F.dTdt[i] = rate;
  }
}

// Johnson-Cook consistent return map of the mixed form, solved for the
// increment.  With the cached power pwn = ep^n and u = dl / ep,
//   f(dl) = d0 - 3G dl - B RT pwn ((1 + u)^n - 1),   d0 = st - (A + B pwn) RT,
// is the same residual as st - 3G dl - (A + B (ep + dl)^n) RT, but every term
// is of the size of the overshoot d0, so FP32 resolves the root to ~1e-7 of dl
// (st itself is an FP32 value).  The written form subtracts numbers ~1e3 times
// larger than d0 and needs FP64, which GB300 issues at 1/64 of the FP32 rate.
// Valid while the bracket [0, d0 / 3G] keeps u below 0.05: the 5-term binomial
// series of (1 + u)^n - 1 then has a relative truncation error of about
// |C(n,6)|/n u^5 (1.7e-8 for n = 0.42, below FP32 rounding; 0.05^5/6 = 5e-8 for
// any n <= 1).  Returns false otherwise (first yield, large increments, a power
// refresh step) and the caller takes the FP64 form.  On success pwn is advanced
// to (ep + dl)^n in FP64.
__device__ __forceinline__ bool jc_return_inc32(const StepParams& P, float st, float RT,
                                                double ep, double& pwn, float dl_ratio,
                                                float* dl_out, float* sy_out, int* iters) {
  if (!(pwn >= 0.0) || P.refresh_pow || !(ep > 0.0)) return false;
  const float pw = (float)pwn;
  const float BRp = P.jcBf * RT * pw;
  const float sy0 = P.jcAf * RT + BRp;
  const float d0 = st - sy0;
  *iters = 0;
  if (!(d0 > 0.0f)) {
    *dl_out = 0.0f;
    *sy_out = sy0;
    return true;
  }
  const float epf = (float)ep;
  float hi = d0 / P.G3f, lo = 0.0f;
  if (!(hi < 0.05f * epf)) return false;
  const float inv_ep = 1.0f / epf;
  const float b0 = P.binf[0], b1 = P.binf[1], b2 = P.binf[2], b3 = P.binf[3], b4 = P.binf[4];
  const float tol = fmaxf((float)P.newton_rtol * st, 16.0f * 1.1920929e-7f * d0);
  float dl = (dl_ratio > 0.0f && dl_ratio <= 1.0f) ? dl_ratio * hi : hi;
  int it = 0;
  for (; it < P.newton_max_iter; it++) {
    const float u = dl * inv_ep;
    const float ser = u * (b0 + u * (b1 + u * (b2 + u * (b3 + u * b4))));
    const float f = d0 - P.G3f * dl - BRp * ser;
    if (fabsf(f) <= tol) break;
    if (f > 0.0f) lo = dl; else hi = dl;
    // f'(dl) = -3G - B RT pwn n (1 + u)^(n - 1) / ep
    const float dser =
        inv_ep * (b0 + u * (2.0f * b1 + u * (3.0f * b2 + u * (4.0f * b3 + u * 5.0f * b4))));
    float dn = dl + f / (P.G3f + BRp * dser);
    if (!(dn > lo && dn < hi)) dn = 0.5f * (lo + hi);
    dl = dn;
  }
  const float u = dl * inv_ep;
  const float ser = u * (b0 + u * (b1 + u * (b2 + u * (b3 + u * b4))));
  *iters = it;
  *dl_out = dl;
  *sy_out = sy0 + BRp * ser;
  pwn += pwn * (double)ser;
  return true;
}

// ---- B32: rate tensors + EOS + stress (InteractionAlt.cu:262-383,
//      Mechanical.cu:289-298, :458-554), energy (Energy.cu:5-19, own tensors)
// neighbours gathered per batch in the stress pass (position and velocity)
constexpr int kStressBatch = 4;
// hardening slope over 3G above which the warm-start network is asked: the
// radial start's relative overshoot must exceed the network's error (~1e-2)
constexpr float kMlpSteep = 0.02f;

// The rate-tensor pair loop of the stress pass (CalcRateTensors,
// InteractionAlt.cu:262-383, in FP32) over the neighbour list L (slots into
// the global array, or ranks into the tile's halo in shared memory).
// acc = D xx yy zz xy yz xz, W xy yz xz, with the off-diagonal sums doubled
// (halved by the caller).  The off-diagonal terms of a pair are a + b (D) and
// a - b (W) of two products a = s_k x_l, b = s_l x_k: their two sums are
// accumulated (one FMA each) and combined once after the loop.
template <bool kFilter, class L, class R>
__device__ __forceinline__ void stress_pairs(const StepParams& P, const Fields& F, const R& rec,
                                             const L& list, int c,
                                             float4 pi, float4 vi, float* acc) {
  const float invh = P.invhf, C = P.Cf, Ch = P.Chf;
  float Dxx = 0.f, Dyy = 0.f, Dzz = 0.f;
  float Axy = 0.f, Bxy = 0.f, Axz = 0.f, Bxz = 0.f, Ayz = 0.f, Byz = 0.f;
  int nx[8];
  if (c > 0) list.block(0, nx);
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    int js[8];
#pragma unroll
    for (int q = 0; q < 8; q++) js[q] = nx[q];
    const int m = c - WF_NB_BLK * b;
    if (P.nb_pf && m > P.nb_pf * WF_NB_BLK) list.prefetch(b + P.nb_pf, 1);
    if (m > WF_NB_BLK) list.block(b + 1, nx);
#pragma unroll
    for (int h = 0; h < WF_NB_BLK; h += kStressBatch) {
      float4 pj[kStressBatch], vj[kStressBatch];
#pragma unroll
      for (int q = 0; q < kStressBatch; q++) {
        const Rec32 r = rec.get(js[h + q]);
        pj[q] = r.p;
        vj[q] = r.v;
      }
#pragma unroll
      for (int q = 0; q < kStressBatch; q++) {
        // Entries past the count are the particle's own slot (list padding):
        // r^2 = 0 gives GK = 0 exactly (gk32_r2), so they add exact zeros and
        // need no test, except under the zone filter.
        if constexpr (kFilter) {
          if (h + q >= m || !pass_j(P, F.id[js[h + q]])) continue;
        }
        const float xx = pi.x - pj[q].x, xy = pi.y - pj[q].y, xz = pi.z - pj[q].z;
        // w = 2 s of the reference's s = -GK m_j / (2 rho_j); the off-diagonal
        // sums carry the factor 2 and are halved after the loop
        const float w = -gk32_r2(xx * xx + xy * xy + xz * xz, invh, Ch, C) *
                        __fdividef(pj[q].w, vj[q].w);
        const float sa = (vi.x - vj[q].x) * w, sb = (vi.y - vj[q].y) * w,
                    sc = (vi.z - vj[q].z) * w;
        Dxx += sa * xx;
        Dyy += sb * xy;
        Dzz += sc * xz;
        Axy += sa * xy;
        Bxy += sb * xx;
        Axz += sa * xz;
        Bxz += sc * xx;
        Ayz += sb * xz;
        Byz += sc * xy;
      }
    }
  }
  acc[0] = Dxx; acc[1] = Dyy; acc[2] = Dzz;
  acc[3] = Axy + Bxy; acc[4] = Ayz + Byz; acc[5] = Axz + Bxz;
  acc[6] = Axy - Bxy; acc[7] = Ayz - Byz; acc[8] = Bxz - Axz;
}

// Copies the tile's halo records and local lists into shared memory (every
// thread of the block takes part; asynchronous 16-byte copies, then one
// barrier).  Returns the halo size, or -1 when the tile is not staged (the
// block then gathers from global memory): sp[k], sv[k] = the two halves of
// rec[halo[k]]; the lists go to sl.
__device__ __forceinline__ int stage_halo16(const TileHalo& T, int64_t npad, int tile, float4* sp,
                                            float4* sv, const Rec32* rec, uint16_t* sl) {
  const int H = T.cap > 0 ? T.hcnt[tile] : -1;
  if (H < 0 || H > T.cap) return -1;        // uniform over the block
  const int32_t* hs = T.halo + T.hoff[tile];
  for (int k = threadIdx.x; k < H; k += blockDim.x) {
    const float4* src = reinterpret_cast<const float4*>(rec + hs[k]);
    cp_async16(sp + k, src);
    cp_async16(sv + k, src + 1);
  }
  stage_lists(T.nbl, npad, tile, sl);
  cp_async_wait_all();
  __syncthreads();
  return H;
}

// The stress pass, with the warm-start network compiled in (kMlp: kernel
// k_stress32_mlp) or without it (k_stress32); both held to 80 registers for
// 6 blocks per SM (786k particles: 0.222 -> 0.213 ms without the network;
// with it, 6 blocks gained nothing while the network took 25 KB of shared
// memory per block, and 0.2335 -> 0.226 ms once it took 17 KB).
template <bool kMlp>
__device__ __forceinline__ void stress32_body(StepParams P, Fields F,
                                                  const Rec32* __restrict__ pvb,
                                                  const Sig32 sig,
                                                  const int32_t* __restrict__ nb,
                                                  const int32_t* __restrict__ cnt,
                                                  int* __restrict__ status,
                                                  const uint4* __restrict__ mlp,
                                                  const MlpL1 l1, const TileHalo T,
                                                  const List16 L16) {
  // The MLP runs on the tensor cores (tcgen05) for the block's 128 particles
  // at once: every thread of the block must reach it, so out-of-range and
  // non-solid threads are predicated rather than returned before that point.
  // Dynamic shared memory: the network's region (when it runs), then the
  // tile's halo records (positions, velocities) when the tile is staged.
  extern __shared__ __align__(1024) uint8_t smlp[];
  if constexpr (kMlp) mlp_umma_begin(smlp, mlp);
  float4* sp = reinterpret_cast<float4*>(smlp + (kMlp ? WF_UMMA_SMEM : 0));
  float4* sv = sp + T.cap;
  uint16_t* sl = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(sp) + stress_lists_at(T.cap));
  const int staged = stage_halo16(T, P.npad, blockIdx.x, sp, sv, pvb, sl);
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : 0;
  const Rec32 own = rec_load(pvb + i);
  const float4 pi = own.p, vi = own.v;
  const double rho_new = F.vd[i].w + P.dt * F.drho[i];
  const double p = 0.0 + (P.Cs * P.Cs) * (rho_new - P.rho0);   // FP64: small density change
  if (valid) F.p[i] = p;
  const bool solid = valid && F.perm[i] < P.n_solid;
  if (!kMlp && !solid) return;
  if (P.state_pf && solid) {
    prefetch_l2(F.ss32 + 6 * i); prefetch_l2(F.eps_p + i); prefetch_l2(F.sy + i);
    prefetch_l2(F.pwn + i); prefetch_l2(F.T + i); prefetch_l2(F.eint + i);
  }
  if (P.pf_ahead > 0) {
    const int64_t ia = i0 + P.pf_ahead;     // the slot this thread's successor will take
    if (ia < P.n) {
      prefetch_l2(pvb + ia); prefetch_l2(F.vd + ia);
      prefetch_l2(F.drho + ia); prefetch_l2(cnt + ia); prefetch_l2(F.perm + ia);
      for (int b = 0; b < P.wave_pf && b < WF_NB_BLOCKS; b++) nb_prefetch(nb, P.npad, ia, b, 4);
    }
  }
  const int c = solid ? cnt[i] : 0;
  float acc[9];
  const int b16 = L16.base ? L16.base[i0 / WF_TILE] : -1;    // uniform over the block
  const RecGlobal rec{pvb};
  const NbList32 list{nb, P.npad, i};
  if (zone_filter(P))
    stress_pairs<true>(P, F, rec, list, c, pi, vi, acc);
  else if (staged >= 0)
    stress_pairs<false>(P, F, RecShared{sp, sv}, NbListS{sl, (int)threadIdx.x}, c, pi, vi, acc);
  else if (b16 >= 0)
    stress_pairs<false>(P, F, rec, NbList16{L16.off, P.npad, i, b16}, c, pi, vi, acc);
  else
    stress_pairs<false>(P, F, rec, list, c, pi, vi, acc);
  float Dxx = acc[0], Dyy = acc[1], Dzz = acc[2], Dxy = acc[3], Dyz = acc[4], Dxz = acc[5];
  float Wxy = acc[6], Wyz = acc[7], Wxz = acc[8];
  Dxy *= 0.5f; Dxz *= 0.5f; Dyz *= 0.5f;
  Wxy *= 0.5f; Wxz *= 0.5f; Wyz *= 0.5f;
  // Jaumann update with the reference's product
  float2* ssp = reinterpret_cast<float2*>(F.ss32 + 6 * i);
  const float2 s01 = ssp[0], s23 = ssp[1], s45 = ssp[2];
  T3f S;
  S.xx = s01.x; S.yy = s01.y; S.zz = s23.x;
  S.xy = S.yx = s23.y; S.yz = S.zy = s45.x; S.xz = S.zx = s45.y;
  T3f W;
  W.xx = W.yy = W.zz = 0.f;
  W.xy = Wxy; W.yz = Wyz; W.xz = Wxz; W.yx = -Wxy; W.zy = -Wyz; W.zx = -Wxz;
  T3f WT;
  WT.xx = WT.yy = WT.zz = 0.f;
  WT.xy = W.yx; WT.xz = W.zx; WT.yx = W.xy; WT.yz = W.zy; WT.zx = W.xz; WT.zy = W.yz;
  const T3f SRT = mul_ref_f(S, WT);
  const T3f RS = mul_ref_f(W, S);
  const float G2 = P.G2f, dt = P.dtf;
  const float tr3 = (1.0f / 3.0f) * (Dxx + Dyy + Dzz);
  T3f Sn;
  Sn.xx = dt * (G2 * (Dxx - tr3) + SRT.xx + RS.xx) + S.xx;
  Sn.yy = dt * (G2 * (Dyy - tr3) + SRT.yy + RS.yy) + S.yy;
  Sn.zz = dt * (G2 * (Dzz - tr3) + SRT.zz + RS.zz) + S.zz;
  Sn.xy = dt * (G2 * Dxy + SRT.xy + RS.xy) + S.xy;
  Sn.yx = dt * (G2 * Dxy + SRT.yx + RS.yx) + S.yx;
  Sn.xz = dt * (G2 * Dxz + SRT.xz + RS.xz) + S.xz;
  Sn.zx = dt * (G2 * Dxz + SRT.zx + RS.zx) + S.zx;
  Sn.yz = dt * (G2 * Dyz + SRT.yz + RS.yz) + S.yz;
  Sn.zy = dt * (G2 * Dyz + SRT.zy + RS.zy) + S.zy;
  const float eff = sqrtf(0.5f * ((Dxx - Dyy) * (Dxx - Dyy) + (Dyy - Dzz) * (Dyy - Dzz) +
                                  (Dzz - Dxx) * (Dzz - Dxx)) +
                          3.0f * (Dxy * Dxy + Dyz * Dyz + Dxz * Dxz));
  const float J2 = 0.5f * (Sn.xx * Sn.xx + 2.0f * Sn.xy * Sn.yx + 2.0f * Sn.xz * Sn.zx +
                           Sn.yy * Sn.yy + 2.0f * Sn.yz * Sn.zy + Sn.zz * Sn.zz);
  const float st = sqrtf(3.0f * J2);
  double eps_p = F.eps_p[i], sy = F.sy[i];
  double dep = 0.0, seq = st;
  float scale = 1.0f;
  const MatParams& M = P.mat;
  // rate and thermal factors of the JC law in FP32 (mixed form)
  float Th = 0.0f, RTf = 1.0f;
  double pwn = F.pwn[i];
  const bool jc_newton = P.return_map == 1 && M.model == WF_JOHNSON_COOK;
  if (jc_newton) {
    Th = ((float)F.T[i] - P.jcTtf) * P.jcinvdTf;
    if (P.clamp_homologous) Th = fminf(fmaxf(Th, 0.0f), 0.999f);
    const float sr = eff == 0.0f ? 1.0e-5f : eff;
    RTf = (1.0f + P.jcCf * __logf(sr * P.jcinveps0f)) * (1.0f - __powf(Th, P.jcmf));
  }
  double ratio = -1.0;
  if constexpr (kMlp) {
    // warm start: sigma_y0 from the cached power (FP32 suffices for the features).
    // The network can only improve on the radial start where that start is
    // poor: it overshoots the increment by about H' / (3G + H'), with the
    // hardening slope H' = n B RT eps_p^(n - 1) = n B RT pwn / eps_p.  Where
    // that is below the network's own prediction error (~1e-2) the radial
    // start is the better one, and Newton needs one iteration from either.
    const float sy0f = ((float)M.A + (float)M.B * (float)fmax(pwn, 0.0)) * RTf;
    const bool steep = !(eps_p > 0.0) || !(pwn > 0.0) ||
                       P.jcnf * P.jcBf * RTf * __fdividef((float)pwn, (float)eps_p) >
                           kMlpSteep * P.G3f;
    const bool want = solid && jc_newton && st > sy0f && steep;
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    if (want) mlp_features(st / sy0f, eps_p, eff, Th, f);
    const float y = mlp_umma_cta(smlp, mlp, f, want, status, l1);
    const float yc = mlp_accept(y);
    if (want && yc > 0.0f) ratio = (double)yc;
    if (!solid) return;
  }
  unsigned n_it = 0u, n_call = 0u, n_mlp = 0u;   // this particle's return-map counters
  bool capped = false;                            // Newton stopped at newton_max_iter
  if (P.return_map == 0) {
    // reference one-shot radial return (Mechanical.cu:503-536)
    if (sy < (double)st) scale = (float)(sy / (double)st);
    if (M.model == WF_HOLLOMON) sy = hollomon_yield(M, eps_p);
    else if (M.model == WF_JOHNSON_COOK) sy = jc_yield_ref(M, eps_p, (double)eff, F.T[i]);
    if ((double)st > sy) {
      dep = ((double)st - sy) / (3.0 * P.G);
      eps_p += dep;
      seq = sy;
      if (M.model == WF_BILINEAR) sy += dep * M.Ep;
    }
  } else if (jc_newton) {
    // consistent return map: FP32 Newton on the increment where the series
    // form holds, else the FP64 residual with the cached power
    int it = 0;
    double sy1;
    float dlf, sy1f;
    const bool inc32 = jc_return_inc32(P, st, RTf, eps_p, pwn, (float)ratio, &dlf, &sy1f, &it);
    if (inc32) {
      dep = (double)dlf;
      sy1 = (double)sy1f;
    } else {
      jc_return_cached(P, (double)st, 3.0 * P.G, eps_p, pwn, (double)RTf, ratio, &dep, &sy1,
                       &it);
    }
    F.pwn[i] = pwn;
    capped = it >= P.newton_max_iter;
    if (dep > 0.0) {
      scale = inc32 ? sy1f / st : (float)(sy1 / (double)st);
      eps_p += dep;
      seq = sy1;
      n_it = (unsigned)it;
      n_call = 1u;
      n_mlp = ratio > 0.0 ? 1u : 0u;
    }
    sy = sy1;
  } else {
    // bilinear / Hollomon consistent return map in FP64
    Hard H;
    H.model = M.model; H.R = 1.0; H.Th = 1.0; H.sy_cur = sy; H.Ep = M.Ep;
    double sy0, dsy0;
    hard_eval(M, H, eps_p, 0.0, &sy0, &dsy0);
    if ((double)st > sy0) {
      const double G3 = 3.0 * P.G;
      int it = 0;
      dep = newton_return(P, H, (double)st, G3, eps_p, sy0, ((double)st - sy0) / G3, &it);
      capped = it >= P.newton_max_iter;
      double sy1, dsy1;
      hard_eval(M, H, eps_p, dep, &sy1, &dsy1);
      scale = (float)(sy1 / (double)st);
      eps_p += dep;
      sy = sy1;
      seq = sy1;
      n_it = (unsigned)it;
      n_call = 1u;
    } else {
      sy = sy0;
    }
  }
  Sn.xx *= scale; Sn.yy *= scale; Sn.zz *= scale;
  Sn.xy *= scale; Sn.yz *= scale; Sn.xz *= scale;
  ssp[0] = make_float2(Sn.xx, Sn.yy);
  ssp[1] = make_float2(Sn.zz, Sn.xy);
  ssp[2] = make_float2(Sn.yz, Sn.xz);
  // stress / rho^2 for the acceleration pass
  const float pf = (float)p;
  const float rf = vi.w;
  const float ir2 = 1.0f / (rf * rf);
  sig.a[i] = make_float4((Sn.xx - pf) * ir2, (Sn.yy - pf) * ir2, (Sn.zz - pf) * ir2, Sn.xy * ir2);
  sig.b[i] = make_float2(Sn.yz * ir2, Sn.xz * ir2);
  F.eps_p[i] = eps_p;
  F.sy[i] = sy;
  F.seq[i] = seq;
  F.dep[i] = dep;
  F.eff[i] = (double)eff;
  // CalcIntEnergy, accumulated in FP64: energy_mode 1 with the particle's own
  // tensors; energy_mode 0 (the reference's, Energy.cu:270-276) with particle
  // 0's for every particle: its S:D goes to *P.e0 and the integration adds
  // m/rho S0:D0 dt to each particle
  const float sd = Sn.xx * Dxx + Sn.yy * Dyy + Sn.zz * Dzz +
                   2.0f * (Sn.xy * Dxy + Sn.yz * Dyz + Sn.xz * Dxz);
  if (P.energy_mode != 0) {
    const float def = __fdividef(pi.w, rf) * sd;
    F.eint[i] += (double)def * P.dt;
  } else if (i == (int64_t)P.inv[0]) {
    *P.e0 = (double)sd;
  }
  if (P.max_dep && dep > 0.0) {
    // the largest strain since the last rebuild (k_max_dep's maximum, kept up as
    // the strains grow); most warps see that it is larger than theirs
    const double v = eps_p - F.eps_rb[i];
    if (v > 0.0) {
      const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
      if (bits > *(volatile unsigned long long*)P.max_dep) atomicMax(P.max_dep, bits);
    }
  }
  warp_count(status, n_it, n_call, n_mlp, capped, eps_p > 1.e-6);
  if (!isfinite(st)) atomicOr(status, WF_STATUS_NAN);
}

template <bool kWide>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : 6) k_stress32_mlp(StepParams P, Fields F,
                                                      const Rec32* __restrict__ pvb,
                                                      const Sig32 sig,
                                                      const int32_t* __restrict__ nb,
                                                      const int32_t* __restrict__ cnt,
                                                      int* __restrict__ status,
                                                      const uint4* __restrict__ mlp,
                                                      const MlpL1 l1, const TileHalo T,
                                                      const List16 L16) {
  stress32_body<true>(P, F, pvb, sig, nb, cnt, status, mlp, l1, T, L16);
}
template <bool kWide>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : 6) k_stress32(StepParams P, Fields F,
                                                     const Rec32* __restrict__ pvb,
                                                     const Sig32 sig,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt,
                                                     int* __restrict__ status,
                                                     const TileHalo T, const List16 L16) {
  stress32_body<false>(P, F, pvb, sig, nb, cnt, status, nullptr, MlpL1{}, T, L16);
}

// ---- C32: acceleration + Monaghan viscosity (InteractionAlt.cu:18-150) ----
// Lane groups of kAccelLanes (see nb_sub).  Neighbours are gathered in batches
// of kAccelBatch, 56 bytes each (position, velocity, stress/rho^2).  Compiled
// for 8 blocks per SM (kTight) the neighbours of a batch are kept apart by
// tests that never hold (P.pair_fence, always 0): without them the compiler
// overlaps them, needs more than the 64 registers that 8 blocks leave and
// spills (786k particles: 286 us; 231 with the tests, 240 with 6 blocks and
// without them).  786k particles with records of 16 bytes: 0.278 ms with one
// lane per particle, 0.272 with two, 0.31-0.39 with four.
constexpr int kAccelLanes = 2;
constexpr int kAccelBatch = 2;
static_assert(WF_NB_BLK / kAccelLanes >= kAccelBatch, "batch within the lane's sub-block");

// Neighbour records of the acceleration pass, from global memory (the slot
// arrays) or from the tile's halo in shared memory (indexed by local list).
template <class R>
struct AccelSrc {
  R rec;
  const float4* sa;
  const float2* sb;
};

template <bool kFilter, bool kTight, class L, class R>
__device__ __forceinline__ float4 accel_value(const StepParams& P, const Fields& F,
                                              const Rec32* __restrict__ pvb,
                                              const Sig32 sig,
                                              const int32_t* __restrict__ cnt, int64_t i, int g,
                                              const AccelSrc<R>& src, const L& list) {
  constexpr int W = WF_NB_BLK / kAccelLanes;
  const Rec32 own = rec_load(pvb + i);
  const float4 pi = own.p, vi = own.v;
  const int32_t idi = F.id[i];
  const float4 s0 = sig.a[i];
  const float2 s1 = sig.b[i];
  const float invh = P.invhf, C = P.Cf, Ch = P.Chf;
  const float h = P.hf, Cs = P.Csf, alpha = P.alphaf, beta = P.betaf, eps = P.epsf;
  const bool av = alpha != 0.0f || beta != 0.0f;
  float ax = 0.f, ay = 0.f, az = 0.f;
  const int c = cnt[i];
  int nx[W];
  if (c > 0) list.template sub<W>(0, g, nx);
  for (int b = 0; WF_NB_BLK * b < c; b++) {
    int js[W];
#pragma unroll
    for (int q = 0; q < W; q++) js[q] = nx[q];
    const int m = c - WF_NB_BLK * b - g * W;   // entries of this lane's sub-block in the list
    if (P.nb_pf && c > WF_NB_BLK * (b + P.nb_pf)) list.prefetch(b + P.nb_pf, kAccelLanes);
    if (c > WF_NB_BLK * (b + 1)) list.template sub<W>(b + 1, g, nx);
#pragma unroll
    for (int hh = 0; hh < W; hh += kAccelBatch) {
      float4 pj[kAccelBatch], vj[kAccelBatch], t0[kAccelBatch];
      float2 t1[kAccelBatch];
#pragma unroll
      for (int q = 0; q < kAccelBatch; q++) {
        const int j = js[hh + q];
        const Rec32 r = src.rec.get(j);
        pj[q] = r.p;
        vj[q] = r.v;
        t0[q] = src.sa[j];
        t1[q] = src.sb[j];
      }
#pragma unroll
      for (int q = 0; q < kAccelBatch; q++) {
        // Entries past the count are the particle's own slot (list padding):
        // r^2 = 0 gives GK = 0 exactly (gk32_r2), so they add exact zeros and
        // need no test, except under the zone filter.
        if constexpr (kTight && !kFilter) {
          if (P.pair_fence && hh + q >= m) continue;
          if (P.pair_fence && !pass_ij(P, idi, F.id[js[hh + q]])) continue;
        }
        if constexpr (kFilter) {
          if (hh + q >= m || !pass_ij(P, idi, F.id[js[hh + q]])) continue;
        }
        const float xx = pi.x - pj[q].x, xy = pi.y - pj[q].y, xz = pi.z - pj[q].z;
        const float r2 = xx * xx + xy * xy + xz * xz;
        const float GK = gk32_r2(r2, invh, Ch, C) * pj[q].w;
        float PI = 0.f;
        if (av) {
          const float vdx =
              (vi.x - vj[q].x) * xx + (vi.y - vj[q].y) * xy + (vi.z - vj[q].z) * xz;
          if (vdx < 0.f) {
            const float MU = __fdividef(h * vdx, r2 + eps);
            PI = __fdividef(alpha * Cs * MU + beta * MU * MU, 0.5f * (vi.w + vj[q].w));
          }
        }
        const float Txx = s0.x + t0[q].x + PI, Tyy = s0.y + t0[q].y + PI,
                    Tzz = s0.z + t0[q].z + PI;
        const float Txy = s0.w + t0[q].w, Tyz = s1.x + t1[q].x, Txz = s1.y + t1[q].y;
        const float gx = xx * GK, gy = xy * GK, gz = xz * GK;
        ax += Txx * gx + Txy * gy + Txz * gz;
        ay += Txy * gx + Tyy * gy + Tyz * gz;
        az += Txz * gx + Tyz * gy + Tzz * gz;
      }
    }
  }
  if constexpr (kAccelLanes > 1) {
    const unsigned mask = group_mask<kAccelLanes>();
#pragma unroll
    for (int o = 1; o < kAccelLanes; o <<= 1) {
      ax += __shfl_xor_sync(mask, ax, o, kAccelLanes);
      ay += __shfl_xor_sync(mask, ay, o, kAccelLanes);
      az += __shfl_xor_sync(mask, az, o, kAccelLanes);
    }
  }
  return make_float4(ax, ay, az, 0.f);
}

// thread -> (slot, lane within the slot's group)
__device__ __forceinline__ int64_t accel_slot(int& g) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  g = (int)(t & (kAccelLanes - 1));
  return t / kAccelLanes;
}

template <bool kWide>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : 8) k_accel32(StepParams P, Fields F,
                                                 const Rec32* __restrict__ pvb,
                                                 const Sig32 sig,
                                                 float4* __restrict__ a32,
                                                 const int32_t* __restrict__ nb,
                                                 const int32_t* __restrict__ cnt) {
  int g;
  const int64_t i = accel_slot(g);
  if (i >= P.n) return;
  if (P.pf_ahead > 0 && g == 0) {
    const int64_t ia = i + P.pf_ahead;      // the slot this thread's successor will take
    if (ia < P.n) {
      prefetch_l2(pvb + ia); prefetch_l2(sig.a + ia); prefetch_l2(sig.b + ia);
      prefetch_l2(cnt + ia); prefetch_l2(F.perm + ia);
      prefetch_l2(F.id + ia);
      for (int b = 0; b < P.wave_pf && b < WF_NB_BLOCKS; b++)
        nb_prefetch(nb, P.npad, ia, b, 2 * kAccelLanes);
    }
  }
  if (F.perm[i] >= P.n_solid) return;
  const AccelSrc<RecGlobal> src{{pvb}, sig.a, sig.b};
  const NbList32 list{nb, P.npad, i};
  const float4 af = zone_filter(P)
                        ? accel_value<true, !kWide>(P, F, pvb, sig, cnt, i, g, src, list)
                        : accel_value<false, !kWide>(P, F, pvb, sig, cnt, i, g, src, list);
  if (g == 0) a32[i] = af;
}

// What follows the acceleration of a slot: with contact law 1 the few slots near
// a tool go to the list, all others are integrated.
template <bool kLaw1>
__device__ __forceinline__ void accel_tail(const StepParams& P, const Fields& F,
                                           const Rec32* __restrict__ pvb,
                                           const double4* __restrict__ vd2, float4* a32, int64_t i,
                                           float4 af) {
  if constexpr (kLaw1) {
    if (F.perm[i] < P.n_solid) {
      const float4 p = pvb[i].p;
      if (law1_near(P, p.x, p.y, p.z) && law1_triangles(P, F.xm[i])) {
        a32[i] = af;
        const unsigned mask = __activemask();
        const int lead = __ffs(mask) - 1, lane = threadIdx.x & 31;
        int base = 0;
        if (lane == lead) base = atomicAdd(P.near_count, __popc(mask));
        base = __shfl_sync(mask, base, lead);
        P.near_list[base + __popc(mask & ((1u << lane) - 1u))] = (int32_t)i;
        return;
      }
      F.cf[i] = make_double4(0.0, 0.0, 0.0, 0.0);
      F.qf[i] = 0.0;
      P.ccnt[i] = 0;
    }
  }
  integrate_mixed_one(P, F, vd2, i, af);
}

// The acceleration pass with the integration of the same slot behind it
// (no contact stage in between): one pass instead of two, the integration's
// FP64 work and traffic overlapping the other warps' neighbour gathers.
// Neighbours are read from pvb (the density pass's copy of the mirrors) while
// the new mirrors go to F.pv and th32, which this pass does not read.
// kLaw1 (contact law 1): only the slots whose cell of a tool's bins lists a
// triangle take part in the contact, so all others are integrated here as well,
// and those few leave their
// acceleration in a32 and their number in the list that k_contact_law1_list
// (wf_contact.cu) works through, contact and integration.  The separate passes
// read and wrote every slot again (500k particles: 68 us for the contact and 39
// for the integration; now 34 for the listed slots).
// Whole warps run that part, the block's first two for its 64 slots: as one of
// two lanes per slot it issued its ~35 FP64 operations, 16 cycles of an SM each
// whatever the lanes, twice as often (FP64 pipe 41 % busy at 786k; 50,560
// particles 31.6 -> 27.5 us, 500k with law 1 0.5 % of a step).
template <bool kLaw1, bool kWide>
__global__ void __launch_bounds__(128, kWide ? kWideBlocks : 8) k_accel_int32(StepParams P, Fields F,
                                                     const Rec32* __restrict__ pvb,
                                                     const Sig32 sig,
                                                     const double4* __restrict__ vd2,
                                                     float4* __restrict__ a32,
                                                     const int32_t* __restrict__ nb,
                                                     const int32_t* __restrict__ cnt, const List16 L16) {
  __shared__ float4 s_af[128 / kAccelLanes];
  int g;
  const int64_t i0 = accel_slot(g);
  const bool valid = i0 < P.n;
  const int64_t i = valid ? i0 : P.n - 1;
  const AccelSrc<RecGlobal> src{{pvb}, sig.a, sig.b};
  if (P.state_pf && g == 0) {
    prefetch_l2(F.xm + i); prefetch_l2(vd2 + i); prefetch_l2(F.u + i); prefetch_l2(F.T + i);
  }
  if (P.pf_ahead > 0 && g == 0) {
    const int64_t ia = i + P.pf_ahead;      // the slot this thread's successor will take
    if (ia < P.n) {
      prefetch_l2(pvb + ia); prefetch_l2(sig.a + ia); prefetch_l2(sig.b + ia);
      prefetch_l2(cnt + ia); prefetch_l2(F.perm + ia);
      prefetch_l2(F.id + ia);
      for (int b = 0; b < P.wave_pf && b < WF_NB_BLOCKS; b++) nb_prefetch(nb, P.npad, ia, b, 2 * kAccelLanes);
    }
  }
  // rigid (non-solid) slots: zero acceleration, moved by their BCs
  float4 af = make_float4(0.f, 0.f, 0.f, 0.f);
  if (valid && F.perm[i] < P.n_solid) {
    const int b16 = L16.base ? L16.base[i / WF_TILE] : -1;   // uniform over the block
    const NbList32 list{nb, P.npad, i};
    if (kLaw1 && zone_filter(P))
      af = accel_value<true, !kWide>(P, F, pvb, sig, cnt, i, g, src, list);
    else if (b16 >= 0)
      af = accel_value<false, !kWide>(P, F, pvb, sig, cnt, i, g, src,
                                      NbList16{L16.off, P.npad, i, b16});
    else
      af = accel_value<false, !kWide>(P, F, pvb, sig, cnt, i, g, src, list);
  }
  if (g == 0) s_af[threadIdx.x / kAccelLanes] = af;
  __syncthreads();
  if (threadIdx.x >= 128 / kAccelLanes) return;
  const int64_t k = blockIdx.x * (int64_t)(128 / kAccelLanes) + threadIdx.x;
  if (k >= P.n) return;
  accel_tail<kLaw1>(P, F, pvb, vd2, a32, k, s_af[threadIdx.x]);
}

// The same pass for staged tiles: a block of 2 x 128 threads is one tile;
// it copies the halo's positions, velocities and stress / rho^2 records into
// shared memory, then reads the neighbours from there through the local
// lists.  Tiles that are not staged gather from global memory.
__global__ void __launch_bounds__(2 * WF_TILE, 3) k_accel_int32_tiles(
    StepParams P, Fields F, const Rec32* __restrict__ pvb, const Sig32 sig,
    const double4* __restrict__ vd2, const int32_t* __restrict__ nb,
    const int32_t* __restrict__ cnt, const TileHalo T) {
  static_assert(kAccelLanes == 2, "one tile per block of 2 lanes per slot");
  extern __shared__ __align__(16) uint8_t sac[];
  float4* sp = reinterpret_cast<float4*>(sac);
  float4* sv = sp + T.cap;
  float4* ssa = sv + T.cap;
  float2* ssb = reinterpret_cast<float2*>(ssa + T.cap);
  uint16_t* sl = reinterpret_cast<uint16_t*>(sac + accel_lists_at(T.cap));
  int staged = -1;
  {
    const int H = T.cap > 0 ? T.hcnt[blockIdx.x] : -1;
    if (H >= 0 && H <= T.cap) {                 // uniform over the block
      const int32_t* hs = T.halo + T.hoff[blockIdx.x];
      for (int k = threadIdx.x; k < H; k += blockDim.x) {
        const int s = hs[k];
        const float4* rec = reinterpret_cast<const float4*>(pvb + s);
        cp_async16(sp + k, rec);
        cp_async16(sv + k, rec + 1);
        cp_async16(ssa + k, sig.a + s);
        cp_async8(ssb + k, sig.b + s);
      }
      stage_lists(T.nbl, P.npad, blockIdx.x, sl);
      cp_async_wait_all();
      __syncthreads();
      staged = H;
    }
  }
  int g;
  const int64_t i = accel_slot(g);
  if (i >= P.n) return;
  float4 af = make_float4(0.f, 0.f, 0.f, 0.f);   // rigid (non-solid) slots: moved by their BCs
  if (F.perm[i] < P.n_solid) {
    if (staged >= 0) {
      const AccelSrc<RecShared> src{{sp, sv}, ssa, ssb};
      af = accel_value<false, false>(P, F, pvb, sig, cnt, i, g, src, NbListS{sl, (int)(threadIdx.x >> 1)});
    } else {
      const AccelSrc<RecGlobal> src{{pvb}, sig.a, sig.b};
      af = accel_value<false, false>(P, F, pvb, sig, cnt, i, g, src, NbList32{nb, P.npad, i});
    }
  }
  if (g == 0) integrate_mixed_one(P, F, vd2, i, af);
}

}  // namespace

static inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

// Slots one resident wave ahead for `kernel` (SMs x resident blocks x threads
// per block / lanes per slot): block b + (resident blocks) starts about when
// block b ends, so the prologue a block prefetches for the slots that far on
// is in L2 when their block starts.  Cached per dynamic shared memory size.
template <class K>
static int64_t wave_slots(K kernel, int threads, size_t smem, int lanes, size_t* c_smem,
                          int64_t* c_val) {
  if (*c_val > 0 && *c_smem == smem) return *c_val;
  int dev = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem) != cudaSuccess)
    return 0;
  *c_smem = smem;
  *c_val = (int64_t)sms * per * threads / lanes;
  return *c_val;
}

// Does a grid run in one wave at kWideBlocks blocks per SM?  (1 or 0; the SM
// count is that of the device the process first asked about.)
static int one_wave(int blocks) {
  static const int sms = [] {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return 0;
    return v;
  }();
  return blocks <= kWideBlocks * sms ? 1 : 0;
}

void launch_fp32_density(const StepParams& P, const Fields& F, double4* vd2, Rec32* pvb,
                         const NbBuffers& N, const List16& L16, cudaStream_t s) {
  static size_t c_smem[2] = {0, 0};
  static int64_t c_val[2] = {0, 0};
  const int blocks = blocks_for(P.n, 128), w = one_wave(blocks);
  const auto kernel = w ? k_density32<true> : k_density32<false>;
  StepParams Q = P;
  Q.pf_ahead = !P.wave_pf ? 0 : (int64_t)(P.wave_dist * (double)wave_slots(
      kernel, 128, 0, 1, &c_smem[w], &c_val[w]));
  kernel<<<blocks, 128, 0, s>>>(Q, F, vd2, pvb, N.nb, N.cnt, L16);
}
void launch_fp32_density_heat(const StepParams& P, const Fields& F, double4* vd2, Rec32* pvb,
                              const NbBuffers& N, int first, int plastic_heat, const TileHalo& T,
                              const List16& L16, cudaStream_t s) {
  TileHalo Tl = T;
  if (kDensLanes != 1) Tl.cap = 0;
  const size_t smem = Tl.cap > 0 ? density_lists_at(Tl.cap) + WF_TILE_LIST_BYTES : 0;
  static size_t opted[2][64] = {};  // per variant and device: dynamic shared memory opted in so far
  static size_t c_smem[2] = {0, 0};
  static int64_t c_val[2] = {0, 0};
  const int blocks = blocks_for(P.n * kDensLanes, 128), w = one_wave(blocks);
  const auto kernel = w ? k_density_heat32<true> : k_density_heat32<false>;
  opt_in_smem(kernel, smem, opted[w]);
  StepParams Q = P;
  Q.pf_ahead = !P.wave_pf ? 0 : (int64_t)(P.wave_dist * (double)wave_slots(
      kernel, 128, smem, kDensLanes, &c_smem[w], &c_val[w]));
  kernel<<<blocks, 128, smem, s>>>(
      Q, F, vd2, pvb, N.nb, N.cnt, first, plastic_heat, Tl, L16);
}
void launch_fp32_heat(const StepParams& P, const Fields& F, const NbBuffers& N, int plastic_heat,
                      cudaStream_t s) {
  static size_t c_smem = 0;
  static int64_t c_val = 0;
  StepParams Q = P;
  Q.pf_ahead = !P.wave_pf ? 0 : (int64_t)(P.wave_dist * (double)wave_slots(
      k_heat32, 128, 0, 1, &c_smem, &c_val));
  k_heat32<<<blocks_for(P.n, 128), 128, 0, s>>>(Q, F, N.nb, N.cnt, plastic_heat);
}
void launch_heat_pairs32(const StepParams& P, const Fields& F, const HeatWork32& H,
                         const NbBuffers& N, cudaStream_t s) {
  k_heat_pairs32<<<blocks_for(P.n, 128), 128, 0, s>>>(P, F, H, N.nb, N.cnt);
}
void launch_heat_step32(const StepParams& P, const Fields& F, const HeatWork32& H, float2* th_out,
                        const NbBuffers& N, int first, int last, cudaStream_t s) {
  k_heat_step32<<<blocks_for(P.n, kHeatStepThreads), kHeatStepThreads, 0, s>>>(P, F, H, F.th32, th_out, N.nb, N.cnt, first,
                                                     last);
}
void launch_fp32_stress(const StepParams& P, const Fields& F, const Rec32* pvb, const Sig32& sig,
                        const NbBuffers& N, int* status, const void* mlp_packed,
                        const MlpL1* mlp_l1, const TileHalo& T, const List16& L16,
                        cudaStream_t s) {
  const uint4* W = reinterpret_cast<const uint4*>(mlp_packed);
  const MlpL1 l1 = (W && mlp_l1) ? *mlp_l1 : MlpL1{};
  static_assert(WF_UMMA_SMEM % 16 == 0, "the halo records behind the network's region");
  const size_t smem = (W ? WF_UMMA_SMEM : 0) +
                      (T.cap > 0 ? stress_lists_at(T.cap) + WF_TILE_LIST_BYTES : 0);
  static size_t opted[2][2][64] = {};  // per variant and device: dynamic shared memory opted in
  static size_t c_smem[2][2] = {};
  static int64_t c_val[2][2] = {};
  const int blocks = blocks_for(P.n, 128), w = one_wave(blocks), m = W ? 1 : 0;
  StepParams Q = P;
  const auto run = [&](auto kernel, auto... args) {
    opt_in_smem(kernel, smem, opted[m][w]);
    Q.pf_ahead = !P.wave_pf ? 0 : (int64_t)(P.wave_dist * (double)wave_slots(
        kernel, 128, smem, 1, &c_smem[m][w], &c_val[m][w]));
    kernel<<<blocks, 128, smem, s>>>(Q, F, pvb, sig, N.nb, N.cnt, status, args...);
  };
  if (W) run(w ? k_stress32_mlp<true> : k_stress32_mlp<false>, W, l1, T, L16);
  else run(w ? k_stress32<true> : k_stress32<false>, T, L16);
}
void launch_fp32_accel(const StepParams& P, const Fields& F, const Rec32* pvb,
                       const Sig32& sig, float4* a32, const NbBuffers& N, cudaStream_t s) {
  static size_t c_smem[2] = {0, 0};
  static int64_t c_val[2] = {0, 0};
  const int blocks = blocks_for(P.n * kAccelLanes, 128), w = one_wave(blocks);
  const auto kernel = w ? k_accel32<true> : k_accel32<false>;
  StepParams Q = P;
  Q.pf_ahead = !P.wave_pf ? 0 : (int64_t)(P.wave_dist * (double)wave_slots(
      kernel, 128, 0, kAccelLanes, &c_smem[w], &c_val[w]));
  kernel<<<blocks, 128, 0, s>>>(Q, F, pvb, sig, a32, N.nb, N.cnt);
}
void launch_fp32_accel_integrate(const StepParams& P, const Fields& F, const Rec32* pvb,
                                 const Sig32& sig, const double4* vd2, float4* a32,
                                 const NbBuffers& N, const TileHalo& T, const List16& L16, cudaStream_t s) {
  if (T.cap > 0) {
    const size_t smem = accel_lists_at(T.cap) + WF_TILE_LIST_BYTES;
    static size_t opted[64] = {};
    opt_in_smem(k_accel_int32_tiles, smem, opted);
    k_accel_int32_tiles<<<blocks_for(P.n * kAccelLanes, 2 * WF_TILE), 2 * WF_TILE, smem, s>>>(
        P, F, pvb, sig, vd2, N.nb, N.cnt, T);
    return;
  }
  static size_t c_smem[2][2] = {};
  static int64_t c_val[2][2] = {};
  const int blocks = blocks_for(P.n * kAccelLanes, 128), w = one_wave(blocks);
  const int law1 = P.near_count ? 1 : 0;
  const auto kernel = law1 ? (w ? k_accel_int32<true, true> : k_accel_int32<true, false>)
                           : (w ? k_accel_int32<false, true> : k_accel_int32<false, false>);
  StepParams Q = P;
  Q.pf_ahead = !P.wave_pf ? 0 : (int64_t)(P.wave_dist * (double)wave_slots(
      kernel, 128, 0, kAccelLanes, &c_smem[law1][w], &c_val[law1][w]));
  kernel<<<blocks, 128, 0, s>>>(Q, F, pvb, sig, vd2, a32, N.nb, N.cnt, L16);
}
