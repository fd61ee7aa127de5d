// wf_nsearch.cu — neighbour search with cuNSearch's float32 rule, cell sort
// and physical reorder of every per-particle array.
//
// Rule (src/cuNSearch/src/cuNSearchKernels.cu:41-234, cuNSearchDeviceData.cu:
// 27-174): search radius r = float(2 h); cell = floor((p - GridMin) *
// GridDelta) in float; candidates from the 27 cells in z, y, x order;
// accept j when the float squared distance is < r*r and > 0; at most 70.
// The distance is computed with round-to-nearest intrinsics, so no fused
// multiply-add can change which pairs pass.
//
// Layout: particles are counting-sorted by linear cell index (z-major), ties
// by original id, and all state is gathered into the new order.  The three
// x-adjacent cells of a row are then one contiguous slot range, so a
// particle's candidates are 9 ranges, visited in the reference's order.
// Lists are stored in blocks of 8 entries (nb_at in wf_common.cuh): a thread
// reads 8 entries with two 16-byte loads and a warp reads contiguous memory.
#include <algorithm>
#include <type_traits>

#include "wf_common.cuh"
#include "wf_nsearch.cuh"

namespace {

__device__ __forceinline__ int cell_coord(float p, float gmin, float gdelta) {
  return (int)floorf(__fmul_rn(__fsub_rn(p, gmin), gdelta));
}

// Cell bounds of the particles, floor(p / r) per axis (kComputeMinMax), as six
// unsigned maxima that start at zero: mm[a] of the complement (so of the
// minimum), mm[3 + a] of the value, both with the sign bit flipped.
__device__ __forceinline__ unsigned bound_code(int c) { return (unsigned)c ^ 0x80000000u; }

// One thread's bounds into mm: warp, block, one atomic per block and axis.
__device__ __forceinline__ void reduce_bounds(const unsigned* lo, const unsigned* hi,
                                              unsigned* mm) {
  __shared__ unsigned smx[6][32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int a = 0; a < 3; a++) {
    const unsigned u = __reduce_max_sync(0xffffffffu, lo[a]);
    const unsigned v = __reduce_max_sync(0xffffffffu, hi[a]);
    if (l == 0) { smx[a][w] = u; smx[3 + a][w] = v; }
  }
  __syncthreads();
  if (w < 6) {
    const unsigned u = __reduce_max_sync(0xffffffffu, l < nw ? smx[w][l] : 0u);
    if (l == 0) atomicMax(mm + w, u);
  }
}
__device__ __forceinline__ void add_bounds(float4 p, float r, unsigned* lo, unsigned* hi) {
  const float c[3] = {p.x, p.y, p.z};
  for (int a = 0; a < 3; a++) {
    const unsigned u = bound_code((int)floorf(__fdiv_rn(c[a], r)));
    lo[a] = max(lo[a], ~u);
    hi[a] = max(hi[a], u);
  }
}

// The last block to come here sizes the search grid from the bounds in hdr->mm
// (grid_from_bounds) and notes whether it fits max_cells; the kernels behind
// read it from device memory.  True on its thread 0.
__device__ __forceinline__ bool size_grid(StaticHeader* hdr, float r, int64_t max_cells) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&hdr->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x != 0) return false;
  unsigned mm[6];
  for (int k = 0; k < 6; k++) mm[k] = atomicMax(hdr->mm + k, 0u);
  int64_t ncell = 0;
  bool fits = !(atomicOr(&hdr->status, 0) & WF_STATUS_GRID);
  int b[6];
  bounds_from_codes(mm, b);
  for (int a = 0; a < 3 && fits; a++) {
    const int64_t span = (int64_t)b[3 + a] - (int64_t)b[a];
    fits = span >= 0 && span + 5 <= max_cells;
  }
  if (fits) {
    GridDev g;
    grid_from_bounds(b, r, &g);
    ncell = 1;
    for (int a = 0; a < 3 && fits; a++) {
      fits = g.dim[a] > 0 && g.dim[a] <= max_cells;
      ncell *= g.dim[a];
      fits = fits && ncell <= max_cells;
    }
    hdr->grid = g;
  }
  hdr->ncell = fits ? (int)ncell : 0;
  return true;
}

// The float positions the search reads (x_h snapshot or the current ones) and
// their cell bounds, in one pass; with host not null also the grid, and the
// bounds and the number of cells go to that page-locked copy.
__global__ void __launch_bounds__(256) k_prep_bounds(int64_t n, const Fields F, int use_current,
                                                     float4* __restrict__ pf, float r,
                                                     StaticHeader* hdr, int64_t max_cells,
                                                     StaticHeader* host) {
  unsigned lo[3] = {0u, 0u, 0u}, hi[3] = {0u, 0u, 0u};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float4 p;
    if (use_current) {
      const double4 x = F.xm[i];
      p = make_float4(__double2float_rn(x.x), __double2float_rn(x.y), __double2float_rn(x.z), 0.f);
    } else {
      p = F.xh[i];
    }
    pf[i] = p;
    add_bounds(p, r, lo, hi);
  }
  reduce_bounds(lo, hi, hdr->mm);
  if (!host || !size_grid(hdr, r, max_cells)) return;
  for (int k = 0; k < 6; k++) host->mm[k] = __ldcg(hdr->mm + k);
  host->ncell = hdr->ncell;
}

// The same for a caller's double3 array (wf_find_neighbors_static), which also
// zeroes the cell counters; the last block to finish sizes the search grid
// (grid_from_bounds) and notes whether it fits: the kernels behind it read it
// from device memory, so the host waits once, at the end (with the cell sort
// and the lists by warps: 19,488 particles 192 -> 70 us a call, of which the
// kernels take 47).
__global__ void __launch_bounds__(256) k_static_prep(int64_t n, const double* __restrict__ x,
                                                     float4* __restrict__ pf, float r,
                                                     StaticHeader* __restrict__ hdr,
                                                     uint32_t* __restrict__ count,
                                                     int64_t max_cells) {
  unsigned lo[3] = {0u, 0u, 0u}, hi[3] = {0u, 0u, 0u};
  bool bad = false;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (int64_t i = i0; i < n; i += step) {
    const double x0 = x[3 * i], x1 = x[3 * i + 1], x2 = x[3 * i + 2];
    bad |= !isfinite(x0) || !isfinite(x1) || !isfinite(x2);
    const float4 p =
        make_float4(__double2float_rn(x0), __double2float_rn(x1), __double2float_rn(x2), 0.0f);
    pf[i] = p;
    add_bounds(p, r, lo, hi);
  }
  for (int64_t k = i0; k < max_cells; k += step) count[k] = 0u;
  if (bad) atomicOr(&hdr->status, WF_STATUS_GRID);
  reduce_bounds(lo, hi, hdr->mm);
  size_grid(hdr, r, max_cells);
}

// Each particle's cell and its rank of arrival there (the order inside a cell
// is settled by k_cell_sort).  The grid comes from the host (g) or, with its
// number of cells, from device memory (hdr).
__global__ void k_cell_count(int64_t n, const float4* __restrict__ pf, GridDev g,
                             const StaticHeader* __restrict__ hdr, uint32_t* __restrict__ cellid,
                             uint32_t* __restrict__ rank, uint32_t* __restrict__ count,
                             int* status) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (hdr) {
    if (hdr->ncell == 0) return;
    g = hdr->grid;
  }
  float4 p = pf[i];
  int cx = cell_coord(p.x, g.gmin[0], g.gdelta[0]);
  int cy = cell_coord(p.y, g.gmin[1], g.gdelta[1]);
  int cz = cell_coord(p.z, g.gmin[2], g.gdelta[2]);
  if (cx < 0 || cy < 0 || cz < 0 || cx >= g.dim[0] || cy >= g.dim[1] || cz >= g.dim[2]) {
    atomicOr(status, WF_STATUS_GRID);
    cx = min(max(cx, 0), g.dim[0] - 1);
    cy = min(max(cy, 0), g.dim[1] - 1);
    cz = min(max(cz, 0), g.dim[2] - 1);
  }
  uint32_t c = ((uint32_t)cz * g.dim[1] + cy) * g.dim[0] + cx;
  cellid[i] = c;
  rank[i] = atomicAdd(count + c, 1u);
}

// The block-local half of an exclusive scan over the cell counts (1,024 per
// block, in place); the last block to finish scans the blocks' totals, so a
// cell's offset is its local one plus bsum[cell / 1024] (k_cell_scatter adds
// them).  bsum: blocks + 1 words, the last one a ticket that starts and ends
// at zero.
__global__ void __launch_bounds__(256) k_cell_scan(uint32_t* __restrict__ data, int64_t cells,
                                                   const StaticHeader* __restrict__ hdr,
                                                   uint32_t* __restrict__ bsum,
                                                   uint32_t* __restrict__ ticket) {
  __shared__ uint32_t warp_tot[8];
  __shared__ bool last;
  if (hdr) cells = hdr->ncell;
  const int64_t blocks = (cells + 1023) / 1024;
  if (blockIdx.x >= blocks) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // exclusive prefix of t over the block; *total on every thread
  const auto scan = [&](uint32_t t, uint32_t* total) {
    uint32_t incl = t;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    __syncthreads();
    if (lane == 31) warp_tot[w] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int k = 0; k < 8; k++) {
      if (k < w) before += warp_tot[k];
      all += warp_tot[k];
    }
    *total = all;
    return before + incl - t;
  };
  const int64_t base = (int64_t)blockIdx.x * 1024 + threadIdx.x * 4;
  uint32_t v[4], total;
  for (int k = 0; k < 4; k++) v[k] = base + k < cells ? data[base + k] : 0u;
  uint32_t run = scan(v[0] + v[1] + v[2] + v[3], &total);
  for (int k = 0; k < 4; k++) {
    if (base + k < cells) data[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0) {
    bsum[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(ticket, 1u) == (uint32_t)blocks - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint32_t carry = 0;
  for (int64_t b0 = 0; b0 < blocks; b0 += 256) {
    const int64_t b = b0 + threadIdx.x;
    const uint32_t t = b < blocks ? *(volatile uint32_t*)(bsum + b) : 0u;
    const uint32_t e = scan(t, &total);
    if (b < blocks) bsum[b] = carry + e;
    carry += total;
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// exclusive scan, 1024 elements per block (256 threads x 4)
__global__ void k_scan_block(uint32_t* data, int64_t n, uint32_t* block_sums) {
  __shared__ uint32_t warp_tot[8];
  int64_t base = (int64_t)blockIdx.x * 1024 + threadIdx.x * 4;
  uint32_t v[4];
  for (int k = 0; k < 4; k++) v[k] = (base + k < n) ? data[base + k] : 0u;
  uint32_t t = v[0] + v[1] + v[2] + v[3];
  uint32_t incl = t;
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    uint32_t x = lane < 8 ? warp_tot[lane] : 0u;
    uint32_t xi = x;
    for (int o = 1; o < 8; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += y;
    }
    if (lane < 8) warp_tot[lane] = xi - x;
    if (lane == 7 && block_sums) block_sums[blockIdx.x] = xi;
  }
  __syncthreads();
  uint32_t run = warp_tot[w] + incl - t;
  for (int k = 0; k < 4; k++) {
    if (base + k < n) data[base + k] = run;
    run += v[k];
  }
}

__global__ void k_scan_add(uint32_t* data, int64_t n, const uint32_t* block_sums) {
  int64_t base = (int64_t)blockIdx.x * 1024 + threadIdx.x * 4;
  uint32_t add = block_sums[blockIdx.x];
  for (int k = 0; k < 4; k++)
    if (base + k < n) data[base + k] += add;
}

// Particles to their cells' ranges, and the cells' final offsets (start[ncell] = n).
// orig: original ids (null: the index itself).
__global__ void k_cell_scatter(int64_t n, int64_t cells, const StaticHeader* __restrict__ hdr,
                               const uint32_t* __restrict__ cellid,
                               const uint32_t* __restrict__ rank,
                               const uint32_t* __restrict__ local,
                               const uint32_t* __restrict__ bsum, uint32_t* __restrict__ start,
                               const int32_t* __restrict__ orig, int32_t* __restrict__ s_src,
                               int32_t* __restrict__ s_orig) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (hdr) cells = hdr->ncell;
  if (cells == 0) return;
  if (i < n) {
    const uint32_t c = cellid[i];
    const uint32_t pos = local[c] + bsum[c >> 10] + rank[i];
    s_src[pos] = (int32_t)i;
    s_orig[pos] = orig ? orig[i] : (int32_t)i;
  }
  for (int64_t c = i; c < cells; c += (int64_t)gridDim.x * blockDim.x)
    start[c] = local[c] + bsum[c >> 10];
  if (i == 0) start[cells] = (uint32_t)n;
}

// Orders each cell's slots by original id, one warp per cell: original ids
// are distinct, so an element's place is the number of smaller ids in its
// cell (32 broadcast compares for a cell of at most 32; the cells hold ~14).
// Every lane reads before any writes.  A larger cell is insertion-sorted by
// one lane.  With pf2 not null the search positions follow into the order.
// kStatic (wf_find_neighbors_static, s_src is s_orig; clouds of any density):
// a larger cell's ranks are counted by all lanes into tmp, and its particles
// behind the first 32 are listed in groups of 32, pairs of cell and first
// index, hdr->groups of them.
template <bool kStatic>
__global__ void k_cell_sort(int64_t cells, StaticHeader* hdr,
                            const uint32_t* __restrict__ start, int32_t* s_src, int32_t* s_orig,
                            const float4* __restrict__ pf, float4* __restrict__ pf2, int32_t* tmp,
                            uint32_t* groups) {
  const int lane = threadIdx.x & 31;
  if (hdr) cells = hdr->ncell;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < cells; c += warps) {
    const uint32_t b = start[c], e = start[c + 1];
    const uint32_t m = e - b;
    if (m == 0u) continue;
    if (m <= 32u) {
      const bool v = (uint32_t)lane < m;
      const int32_t o = v ? s_orig[b + lane] : 0;
      const int32_t sv = v ? s_src[b + lane] : 0;
      uint32_t rank = 0;
      for (uint32_t t = 0; t < m; t++) rank += __shfl_sync(0xffffffffu, o, (int)t) < o;
      __syncwarp();
      if (v) {
        s_orig[b + rank] = o;
        s_src[b + rank] = sv;
        if (pf2) pf2[b + rank] = pf[sv];
      }
      continue;
    }
    if constexpr (kStatic) {
      for (uint32_t k = b + lane; k < e; k += 32) {
        const int32_t o = s_src[k];
        uint32_t rank = 0;
#pragma unroll 8
        for (uint32_t t = b; t < e; t++) rank += s_src[t] < o;
        tmp[b + rank] = o;
      }
      __syncwarp();
      for (uint32_t k = b + lane; k < e; k += 32) s_src[k] = tmp[k];
      const uint32_t more = (m - 1u) / 32u;
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&hdr->groups, more);
      at = __shfl_sync(0xffffffffu, at, 0);
      for (uint32_t k = lane; k < more; k += 32) {
        groups[2 * (at + k)] = (uint32_t)c;
        groups[2 * (at + k) + 1] = b + 32u * (k + 1u);
      }
    } else if (lane == 0) {
      for (uint32_t k = b + 1; k < e; k++) {
        const int32_t ko = s_orig[k], ks = s_src[k];
        uint32_t q = k;
        while (q > b && s_orig[q - 1] > ko) {
          s_orig[q] = s_orig[q - 1];
          s_src[q] = s_src[q - 1];
          q--;
        }
        s_orig[q] = ko;
        s_src[q] = ks;
      }
    }
    __syncwarp();
    if (pf2)
      for (uint32_t k = b + lane; k < e; k += 32) pf2[k] = pf[s_src[k]];
  }
}

template <class T>
__device__ __forceinline__ void g1(T* dst, const T* src, int64_t k, int64_t s) {
  if (dst) dst[k] = src[s];
}
__device__ __forceinline__ void g6(double* dst, const double* src, int64_t k, int64_t s) {
  if (!dst) return;
  const double2* a = reinterpret_cast<const double2*>(src + 6 * s);
  double2* b = reinterpret_cast<double2*>(dst + 6 * k);
  b[0] = a[0]; b[1] = a[1]; b[2] = a[2];
}
__device__ __forceinline__ void g6f(float* dst, const float* src, int64_t k, int64_t s) {
  if (!dst) return;
  const float2* a = reinterpret_cast<const float2*>(src + 6 * s);
  float2* b = reinterpret_cast<float2*>(dst + 6 * k);
  b[0] = a[0]; b[1] = a[1]; b[2] = a[2];
}

// gather every per-slot array into the new order; inv[orig] = new slot
__global__ void k_reorder(int64_t n, const int32_t* __restrict__ s_src, const Fields A, Fields B,
                          const float4* __restrict__ pf, float4* __restrict__ pf2,
                          int32_t* __restrict__ inv) {
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  int64_t s = s_src[k];
  g1(B.xm, A.xm, k, s); g1(B.vd, A.vd, k, s); g1(B.u, A.u, k, s); g1(B.a, A.a, k, s);
  g6(B.sig6, A.sig6, k, s); g6(B.ss6, A.ss6, k, s); g6(B.eps6, A.eps6, k, s);
  g6(B.sr6, A.sr6, k, s); g6(B.rr6, A.rr6, k, s);
  g1(B.p, A.p, k, s); g1(B.seq, A.seq, k, s); g1(B.eps_p, A.eps_p, k, s); g1(B.sy, A.sy, k, s);
  g1(B.eff, A.eff, k, s); g1(B.dep, A.dep, k, s); g1(B.drho, A.drho, k, s);
  g1(B.eint, A.eint, k, s);
  g1(B.T, A.T, k, s); g1(B.Ta, A.Ta, k, s); g1(B.Tb, A.Tb, k, s); g1(B.dTdt, A.dTdt, k, s);
  g1(B.kT, A.kT, k, s); g1(B.cpT, A.cpT, k, s);
  g1(B.id, A.id, k, s); g1(B.bct, A.bct, k, s); g1(B.nw, A.nw, k, s); g1(B.xh, A.xh, k, s);
  g1(B.pv, A.pv, k, s); g1(B.tl32, A.tl32, k, s);
  g1(B.m32, A.m32, k, s); g6f(B.ss32, A.ss32, k, s);
  g1(B.th32, A.th32, k, s); g1(B.pwn, A.pwn, k, s);
  g1(B.nrm, A.nrm, k, s); g1(B.cf, A.cf, k, s); g1(B.qf, A.qf, k, s);
  g1(B.eps_rb, A.eps_rb, k, s);
  int32_t o = A.perm[s];
  B.perm[k] = o;
  inv[o] = (int32_t)k;
  pf2[k] = pf[s];
}

// Neighbour lists, one warp per cell.  The particles of a cell share its
// candidate set: the nine rows of three x-adjacent cells around it, each one
// contiguous range of sorted slots, visited z outer, y, x inner
// (cuNSearchKernels.cu:170-234).  The warp stages in shared memory, in that
// order, the candidates that lie within r of the box around its particles
// (any other one fails the distance test for all of them: the box distance
// is at most the distance to each particle, and a 1e-4 relative margin
// covers the FP32 rounding of both).  Then, for each chunk of 32 staged
// candidates and each particle, the lanes test their candidate against that
// particle with the float rule and the accepted ones are appended in
// candidate order (ballot, prefix popcount).  Lists, counts and the 70-entry
// cap are those of a per-particle scan, entry for entry; the staging halves
// the distance tests (a CPU model of the jittered lattice keeps 161 of 332
// candidates per cell) and the warp shares one candidate range, where
// particles scanned by separate lanes diverge at cell boundaries.  786k
// particles: 0.295 ms per rebuild against 0.385 for the per-particle scan
// (0.348 with 64-bit entry indices in the append loop).
// slot_of == nullptr: the state is in sorted order (sorted index = slot);
// else slot_of[k] is the storage slot of the k-th sorted particle.
constexpr int kNbWarps = 4;      // warps (cells in flight) per block
// List entry index (nb_at) in the index type I: 32-bit when the lists hold
// fewer than 2^31 entries (fewer than ~29M particles), else 64-bit.
// kRows: the caller's row-major lists instead (wf_find_neighbors_static).
template <class I, bool kRows>
__device__ __forceinline__ I nb_at_i(I npad, I i, int k) {
  if constexpr (kRows) return i * (I)WF_NB + (I)k;
  return ((I)(k >> 3) * npad + i) * (I)WF_NB_BLK + (I)(k & 7);
}
constexpr int kNbStage = 192;    // staged candidates per warp and round

// Tests the staged candidates against the group's particles (part[j]: position
// and, in w, the storage slot of particle j, whose count lane j holds) and appends the accepted ones to their lists.  Per chunk of 32
// candidates and per particle j, one ballot gives the accepting lanes; each
// writes its candidate at j's count before the chunk plus the accepting lanes
// below it, so the entries keep candidate order.  The counts advance once per
// chunk (lane j keeps particle j's mask of the chunk), which leaves no chain
// between the particles' iterations.
template <class I, bool kRows>
__device__ __forceinline__ void nb_append_round(int nstaged, const float4* __restrict__ sp,
                                                const int32_t* __restrict__ sid, int gn,
                                                const float4* __restrict__ part, float r2,
                                                int64_t npad, int32_t* __restrict__ nb,
                                                int& count) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  for (int ch = 0; ch < nstaged; ch += 32) {
    const int t = ch + lane;
    const bool v = t < nstaged;
    const float4 q = v ? sp[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int32_t qid = v ? sid[t] : 0;
    unsigned mine = 0u;
#pragma unroll 4
    for (int j = 0; j < gn; j++) {
      const float4 pj = part[j];   // same address on every lane: one broadcast read
      const int32_t ij = __float_as_int(pj.w);
      const int base = __shfl_sync(0xffffffffu, count, j);
      const float dx = __fsub_rn(q.x, pj.x), dy = __fsub_rn(q.y, pj.y), dz = __fsub_rn(q.z, pj.z);
      const float sq =
          __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
      const bool acc = v && sq < r2 && sq > 0.0f;
      const unsigned m = __ballot_sync(0xffffffffu, acc);
      const int k = base + __popc(m & lt);
      if (acc && k < WF_NB) nb[nb_at_i<I, kRows>((I)npad, (I)ij, k)] = qid;
      mine = lane == j ? m : mine;
    }
    count += __popc(mine);
  }
}

// Row r = 3 (dz + 1) + (dy + 1) of the candidates of cell c: slots [rb, rb + rn)
// on lane r < 9
__device__ __forceinline__ void nb_rows(const GridDev& g, const uint32_t* __restrict__ start,
                                        int64_t c, uint32_t& rb, uint32_t& rn) {
  const int lane = threadIdx.x & 31;
  // cell coordinates in 32-bit arithmetic (the grid holds at most 2e9 cells;
  // a 64-bit division is a long software sequence in this issue-bound kernel)
  const uint32_t cu = (uint32_t)c, dx = (uint32_t)g.dim[0], dy = (uint32_t)g.dim[1];
  const uint32_t cyz = cu / dx;
  const int cx = (int)(cu - cyz * dx);
  const int cy = (int)(cyz % dy);
  const int cz = (int)(cyz / dy);
  rb = rn = 0;
  if (lane < 9) {
    const int fz = cz + lane / 3 - 1, fy = cy + lane % 3 - 1;
    if (fz >= 0 && fz < g.dim[2] && fy >= 0 && fy < g.dim[1]) {
      const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.dim[0] - 1);
      const uint32_t rowc = ((uint32_t)fz * g.dim[1] + fy) * g.dim[0];
      rb = start[rowc + x0];
      rn = start[rowc + x1 + 1] - rb;
    }
  }
}

// The lists of a cell's particles g0 .. g0 + gn - 1 (gn <= 32) from its rows.
// kRows: the scan ends when every list of the group is full.
template <class I, bool kRows>
__device__ __forceinline__ void nb_group(uint32_t g0, int gn, uint32_t rb, uint32_t rn, float r2,
                                         int64_t npad, const float4* __restrict__ pf,
                                         const int32_t* __restrict__ slot_of,
                                         int32_t* __restrict__ nb, int32_t* __restrict__ cnt,
                                         int* status, float4* sp, int32_t* sid, float4* part) {
  const int lane = threadIdx.x & 31;
  const float thr = r2 * 1.0001f;
  // this group's particles (lane j < gn holds particle g0 + j) and their box
  float px = 0.f, py = 0.f, pz = 0.f;
  int32_t myslot = 0;
  float lo[3], hi[3];
  if (lane < gn) {
    const float4 p = pf[g0 + lane];
    px = p.x; py = p.y; pz = p.z;
    myslot = slot_of ? slot_of[g0 + lane] : (int32_t)(g0 + lane);
    part[lane] = make_float4(px, py, pz, __int_as_float(myslot));
  }
  {
    const float4 p0 = pf[g0];
    lo[0] = hi[0] = lane < gn ? px : p0.x;
    lo[1] = hi[1] = lane < gn ? py : p0.y;
    lo[2] = hi[2] = lane < gn ? pz : p0.z;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < 3; a++) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
  int count = 0;
  int nstaged = 0;
  for (int r = 0; r < 9; r++) {
    const uint32_t b = __shfl_sync(0xffffffffu, rb, r);
    const uint32_t nr = __shfl_sync(0xffffffffu, rn, r);
    for (uint32_t t0 = 0; t0 < nr; t0 += 32) {
      if (nstaged > kNbStage - 32) {          // staging full: test what is staged
        __syncwarp();
        nb_append_round<I, kRows>(nstaged, sp, sid, gn, part, r2, npad, nb, count);
        __syncwarp();
        nstaged = 0;
        if (kRows && __all_sync(0xffffffffu, lane >= gn || count >= WF_NB)) {
          rn = 0;                               // nothing of the rows behind either
          break;
        }
      }
      const bool v = t0 + lane < nr;
      const uint32_t s = b + t0 + lane;
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      int32_t id = (int32_t)s;
      bool keep = false;
      if (v) {
        q = pf[s];
        if (slot_of) id = slot_of[s];
        const float ex = fmaxf(0.f, fmaxf(lo[0] - q.x, q.x - hi[0]));
        const float ey = fmaxf(0.f, fmaxf(lo[1] - q.y, q.y - hi[1]));
        const float ez = fmaxf(0.f, fmaxf(lo[2] - q.z, q.z - hi[2]));
        keep = ex * ex + ey * ey + ez * ez < thr;
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int at = nstaged + __popc(m & ((1u << lane) - 1u));
        sp[at] = q;
        sid[at] = id;
      }
      nstaged += __popc(m);
    }
  }
  __syncwarp();
  nb_append_round<I, kRows>(nstaged, sp, sid, gn, part, r2, npad, nb, count);
  __syncwarp();
  if (lane < gn) {
    if (count >= WF_NB) atomicOr(status, WF_STATUS_NB_CAP);
    const int cn = min(count, WF_NB);
    cnt[myslot] = cn;
    // pad the last block with the particle's own slot (see nb_at)
    if constexpr (!kRows)
    for (int k = cn; k < ((cn + WF_NB_BLK - 1) & ~(WF_NB_BLK - 1)); k++)
      nb[nb_at(npad, myslot, k)] = myslot;
  }
}

// kRows: a cell's particles behind its first 32 are groups of the list that
// k_cell_sort left, so that the warps share dense cells, and a group's scan ends
// when its lists are full.  A call with 25,000 particles, 200 / 500 / 1,500 a
// cell: 0.22 / 0.36 / 0.86 ms; with a whole cell per warp, its scan to the end
// and its sort by one lane 2.9 / 10.2 / 53; with a thread per particle that
// leaves at 70 entries and a thread per cell for the sort 1.7 / 4.5 / 20.6.
// Up to 14 a cell there are no such groups (73 us).
// (kRows: eight blocks an SM, so 64 registers: 19,488 particles 23.0 us; with
// the 48 that the compiler takes of itself 25.7.)
template <class I, bool kRows>
__global__ void __launch_bounds__(32 * kNbWarps, kRows ? 8 : 0) k_nblist(int64_t ncell, int64_t npad,
                                                          const float4* __restrict__ pf, GridDev g,
                                                          const StaticHeader* __restrict__ hdr,
                                                          const uint32_t* __restrict__ start,
                                                          const int32_t* __restrict__ slot_of,
                                                          const uint32_t* __restrict__ groups,
                                                          int32_t* __restrict__ nb,
                                                          int32_t* __restrict__ cnt, int* status) {
  __shared__ float4 s_pos[kNbWarps][kNbStage];
  __shared__ int32_t s_id[kNbWarps][kNbStage];
  __shared__ float4 s_part[kNbWarps][32];
  const int w = threadIdx.x >> 5;
  if (hdr) {                                   // the grid is in device memory
    ncell = hdr->ncell;
    g = hdr->grid;
  }
  using K = std::conditional_t<kRows, uint32_t, int64_t>;
  const K cells = (K)ncell, total = cells + (K)(kRows ? hdr->groups : 0u);
  for (K k = (K)blockIdx.x * kNbWarps + w; k < total;
       k += (K)gridDim.x * kNbWarps) {         // whole warps together
    K c = k;
    uint32_t ps;
    if (kRows && k >= cells) {
      c = groups[2 * (k - cells)];
      ps = groups[2 * (k - cells) + 1];
    } else {
      ps = start[c];
    }
    const uint32_t end = start[c + 1], pe = kRows ? min(end, ps + 32u) : end;
    if (ps >= pe) continue;
    uint32_t rb, rn;
    nb_rows(g, start, c, rb, rn);
    for (uint32_t g0 = ps; g0 < pe; g0 += 32)
      nb_group<I, kRows>(g0, (int)min(32u, pe - g0), rb, rn, g.r2, npad, pf, slot_of, nb, cnt, status,
                         s_pos[w], s_id[w], s_part[w]);
  }
}

__global__ void k_snapshot(int64_t n, Fields F) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 x = F.xm[i];
  F.xh[i] = make_float4(__double2float_rn(x.x), __double2float_rn(x.y), __double2float_rn(x.z), 0.f);
}

inline int nblocks(int64_t n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

int device_exclusive_scan(uint32_t* data, int64_t n, uint32_t* tmp, cudaStream_t s) {
  int64_t nb = (n + 1023) / 1024;
  if (nb <= 1) {
    k_scan_block<<<1, 256, 0, s>>>(data, n, nullptr);
    return 1;
  }
  k_scan_block<<<(int)nb, 256, 0, s>>>(data, n, tmp);
  const int inner = device_exclusive_scan(tmp, nb, tmp + nb, s);
  k_scan_add<<<(int)nb, 256, 0, s>>>(data, n, tmp);
  return inner + 2;
}

int64_t scan_tmp_words(int64_t n) {
  int64_t w = 0;
  while (n > 1024) {
    n = (n + 1023) / 1024;
    w += n;
  }
  return w + 1;
}

int64_t cell_scan_words(int64_t cells) { return (cells + 1023) / 1024 + 1; }

void launch_prep_bounds(int64_t n, const Fields& F, int use_current, float4* pf, float r,
                        StaticHeader* hdr, int64_t max_cells, StaticHeader* host,
                        cudaStream_t s) {
  cudaMemsetAsync(hdr, 0, sizeof(StaticHeader), s);
  k_prep_bounds<<<std::min(nblocks(n, 256), 1024), 256, 0, s>>>(n, F, use_current, pf, r, hdr,
                                                                max_cells, host);
}
void launch_static_prep(int64_t n, const double* x, float4* pf, float r, StaticHeader* hdr,
                        uint32_t* count, int64_t max_cells, cudaStream_t s) {
  cudaMemsetAsync(hdr, 0, sizeof(StaticHeader), s);
  k_static_prep<<<std::min(nblocks(n, 256), 304), 256, 0, s>>>(n, x, pf, r, hdr, count, max_cells);
}
void launch_cell_sort(int64_t n, const float4* pf, const GridDev& g, StaticHeader* hdr,
                      const int32_t* orig, const CellWork& W, int32_t* s_src, int32_t* s_orig,
                      float4* pf2, int* status, cudaStream_t s) {
  // with the grid in device memory the launches are sized for the most cells
  const int64_t cells = hdr ? W.max_cells : (int64_t)g.dim[0] * g.dim[1] * g.dim[2];
  k_cell_count<<<nblocks(n, 256), 256, 0, s>>>(n, pf, g, hdr, W.cellid, W.rank, W.count, status);
  k_cell_scan<<<nblocks(cells, 1024), 256, 0, s>>>(W.count, cells, hdr, W.bsum, W.ticket);
  k_cell_scatter<<<nblocks(n, 256), 256, 0, s>>>(n, cells, hdr, W.cellid, W.rank, W.count, W.bsum,
                                                 W.start, orig, s_src, s_orig);
  const int blocks = nblocks(cells * 32, 256);
  const int grid = hdr ? std::min(blocks, 1216) : blocks;
  if (orig)
    k_cell_sort<false><<<grid, 256, 0, s>>>(cells, hdr, W.start, s_src, s_orig, pf, pf2, nullptr,
                                            nullptr);
  else   // the cell numbers and counts have done their work
    k_cell_sort<true><<<grid, 256, 0, s>>>(cells, hdr, W.start, s_src, s_orig, pf, pf2,
                                           reinterpret_cast<int32_t*>(W.cellid), W.count);
}
void launch_reorder(int64_t n, const int32_t* s_src, const Fields& A, const Fields& B,
                    const float4* pf, float4* pf2, int32_t* inv, cudaStream_t s) {
  k_reorder<<<nblocks(n, 256), 256, 0, s>>>(n, s_src, A, B, pf, pf2, inv);
}
void launch_nblist(int64_t ncell, int64_t npad, const float4* pf, const GridDev& g,
                   const StaticHeader* hdr, const uint32_t* start, const int32_t* slot_of,
                   int32_t* nb, int32_t* cnt, int* status, cudaStream_t s) {
  if ((int64_t)WF_NB_ALLOC * npad < ((int64_t)1 << 31))
    k_nblist<uint32_t, false><<<nblocks(ncell, kNbWarps), 32 * kNbWarps, 0, s>>>(
        ncell, npad, pf, g, hdr, start, slot_of, nullptr, nb, cnt, status);
  else
    k_nblist<int64_t, false><<<nblocks(ncell, kNbWarps), 32 * kNbWarps, 0, s>>>(
        ncell, npad, pf, g, hdr, start, slot_of, nullptr, nb, cnt, status);
}
void launch_static_lists(const float4* pf, const StaticHeader* hdr, const uint32_t* start,
                         const int32_t* order, const uint32_t* groups, int32_t* lists,
                         int32_t* counts, int* status, cudaStream_t s) {
  k_nblist<uint32_t, true><<<2432, 32 * kNbWarps, 0, s>>>(0, 0, pf, GridDev{}, hdr, start, order,
                                                          groups, lists, counts, status);
}
void launch_snapshot(int64_t n, const Fields& F, cudaStream_t s) {
  k_snapshot<<<nblocks(n, 256), 256, 0, s>>>(n, F);
}
