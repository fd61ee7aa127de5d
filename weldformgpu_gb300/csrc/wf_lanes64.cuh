// wf_lanes64.cuh — how many lanes share a particle in the FP64 passes over the
// neighbour lists, and sums in list order over those lanes.
//
// kG = 1: one thread per particle walks its list.  kG = 4, 8, 16 or 32: so many
// lanes per particle, lane g takes entry kG b + g in round b (one coalesced
// read of the round's indices and geometry), and the round's terms are added
// in list order, term by term, so the sums round as in the walk.  More lanes
// spread a small domain over the chip (800 particles: 13 blocks of 64 threads,
// 800 of a warp) and shorten the chain of dependent loads and pairs, 27-57
// deep in the walk and one or two rounds with a warp; the ordered sums use
// fewer lanes for the more additions (8 lanes: up to 8 a round and accumulator
// set).  Step with the heat pass, us, with 32 / 16 / 8 / 1 lanes: n = 800 74 /
// 87 / 111 / -, 2,184 99 / 97 / 111 / -, 3,328 127 / 110 / 121 / -, 6,320 201
// / 157 / 144 / -, 36,720 - / - / 528 / 584, 86,592 - / - / 1,174 / 1,150:
// the lines of lanes64().
#pragma once
#include "wf_common.cuh"

// Lanes of a particle for a domain of n
static inline int lanes64(int64_t n) {
  return n >= 64000 ? 1 : n >= 5000 ? 8 : n >= 2000 ? 16 : 32;
}

// This thread's slot, lane and list length; threads past the end or without a
// list keep c = 0 and stay for the warp's shuffles
template <int kG>
__device__ __forceinline__ int64_t slot64(int& g) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  g = (int)(t & (kG - 1));
  return t / kG;
}
// rounds of kG entries that the warp walks together
template <int kG>
__device__ __forceinline__ int warp_rounds(int c) {
  return (__reduce_max_sync(0xffffffffu, c) + kG - 1) / kG;
}
// acc + t_0 + ... over the lanes of a group, in lane order: on every lane of
// eight; of a warp, on lane 0, through shared memory (32 doubles).  m: terms
// of the round (a warp's are all its own particle's)
template <int kG>
__device__ __forceinline__ double add_in_order(double* sh, double acc, double t, int m) {
  if constexpr (kG == 32) {
    const int lane = threadIdx.x & 31;
    sh[lane] = t;
    __syncwarp();
    if (lane == 0)
#pragma unroll
      for (int b = 0; b < kG; b += 8) {
        if (b >= m) break;
#pragma unroll
        for (int k = 0; k < 8; k++) acc += sh[b + k];
      }
    __syncwarp();
  } else {
#pragma unroll
    for (int k = 0; k < kG; k++) acc += __shfl_sync(0xffffffffu, t, k, kG);
  }
  return acc;
}
// The same for kA accumulators through shared memory (32 rows of kA doubles,
// kA odd: no bank conflicts): lane a of the group adds accumulator a, lane
// a - kG accumulator a >= kG.
template <int kG, int kA>
__device__ __forceinline__ void add_in_order(double* sh, const double* t, int g, double* acc,
                                             int m) {
  static_assert(kA % 2 == 1 && kA <= 2 * kG, "accumulators of a group");
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < kA; a++) sh[lane * kA + a] = t[a];
  __syncwarp();
  const double* row = sh + (lane - g) * kA;
#pragma unroll
  for (int b = 0; b < kG; b += 8) {
    if (kG == 32 && b >= m) break;
    if (g < kA)
#pragma unroll
      for (int k = 0; k < (kG < 8 ? kG : 8); k++) acc[0] += row[(b + k) * kA + g];
    if (kA > kG && g < kA - kG)
#pragma unroll
      for (int k = 0; k < (kG < 8 ? kG : 8); k++) acc[1] += row[(b + k) * kA + g + kG];
  }
  __syncwarp();
}
