// wf_nsearch.cuh — neighbour-search launchers (wf_nsearch.cu).
#pragma once
#include <climits>
#include "wf_common.cuh"

struct GridDev {
  float gmin[3], gdelta[3], r2;
  int dim[3];
};

// The search grid and what it is sized from, in device memory: the head of the
// allocation-free search's scratch, and a domain's own for the rebuilds that do
// not wait for the host.
struct StaticHeader {
  unsigned mm[6];       // cell bounds (codes)
  int status;           // WF_STATUS_* bits
  unsigned ticket, scan_ticket;
  int ncell;            // cells of the grid; 0: it does not fit, nothing is searched
  unsigned groups;      // static search: groups of particles behind a cell's first 32
  GridDev grid;
};

// cell bounds min x, y, z, max x, y, z from the codes of launch_prep_bounds
__host__ __device__ inline void bounds_from_codes(const unsigned* mm, int* b) {
  for (int a = 0; a < 3; a++) {
    b[a] = (int)(~mm[a] ^ 0x80000000u);
    b[3 + a] = (int)(mm[3 + a] ^ 0x80000000u);
  }
}
// grid set-up, computeCellInformation (cuNSearchDeviceData.cu:80-123); the
// float operations round alike on the host and on the device
__host__ __device__ inline void grid_from_bounds(const int mm[6], float r, GridDev* g) {
#ifdef __CUDA_ARCH__
#define WF_FMUL(a, b) __fmul_rn(a, b)
#define WF_FSUB(a, b) __fsub_rn(a, b)
#define WF_FDIV(a, b) __fdiv_rn(a, b)
#else
#define WF_FMUL(a, b) ((a) * (b))
#define WF_FSUB(a, b) ((a) - (b))
#define WF_FDIV(a, b) ((a) / (b))
#endif
  for (int a = 0; a < 3; a++) {
    const float Min = WF_FMUL((float)mm[a], r), Max = WF_FMUL((float)mm[3 + a], r);
    const float gridSize = WF_FSUB(Max, Min);
    g->dim[a] = (int)((unsigned)ceilf(WF_FDIV(gridSize, r)) + 4u);
    g->gmin[a] = WF_FSUB(Min, WF_FMUL(r, 2.0f));
    const float gs2 = WF_FMUL((float)(unsigned)g->dim[a], r);
    g->gdelta[a] = WF_FDIV((float)(unsigned)g->dim[a], gs2);
  }
  g->r2 = WF_FMUL(r, r);
#undef WF_FMUL
#undef WF_FSUB
#undef WF_FDIV
}

// Work arrays of the cell sort.
struct CellWork {
  uint32_t* cellid;    // [n]; static search: a sort's scratch behind that
  uint32_t* rank;      // [n]
  uint32_t* count;     // [cells], zero on entry; static search: [2 n / 32] the groups at the end
  uint32_t* bsum;      // [cells / 1024 + 1]
  uint32_t* ticket;    // one word, zero on entry and on return
  uint32_t* start;     // [cells + 1] out: the cells' ranges in sorted order
  int64_t max_cells;   // for a grid in device memory
};
// returns the number of kernels launched
int device_exclusive_scan(uint32_t* data, int64_t n, uint32_t* tmp, cudaStream_t s);
int64_t scan_tmp_words(int64_t n);
int64_t cell_scan_words(int64_t cells);
// float positions (x_h or the current ones) into pf, their cell bounds' codes into hdr->mm; with
// host (page-locked) not null also the grid into hdr, if it fits max_cells, and codes and cells
// into *host
void launch_prep_bounds(int64_t n, const Fields& F, int use_current, float4* pf, float r,
                        StaticHeader* hdr, int64_t max_cells, StaticHeader* host, cudaStream_t s);
void launch_static_prep(int64_t n, const double* x, float4* pf, float r, StaticHeader* hdr,
                        uint32_t* count, int64_t max_cells, cudaStream_t s);
// Counting sort by cell, original ids ascending inside a cell (orig null: the
// index): s_src, s_orig in sorted order, W.start, and with pf2 not null the
// positions in sorted order.  The grid is g, or hdr's when hdr is not null.
void launch_cell_sort(int64_t n, const float4* pf, const GridDev& g, StaticHeader* hdr,
                      const int32_t* orig, const CellWork& W, int32_t* s_src, int32_t* s_orig,
                      float4* pf2, int* status, cudaStream_t s);
void launch_reorder(int64_t n, const int32_t* s_src, const Fields& A, const Fields& B,
                    const float4* pf, float4* pf2, int32_t* inv, cudaStream_t s);
// ncell: cells of the grid g, or about as many when the grid is hdr's
void launch_nblist(int64_t ncell, int64_t npad, const float4* pf, const GridDev& g,
                   const StaticHeader* hdr, const uint32_t* start, const int32_t* slot_of,
                   int32_t* nb, int32_t* cnt, int* status, cudaStream_t s);
// row-major lists and counts by the caller's index (order[k]: index of the k-th sorted particle;
// groups: W.count as launch_cell_sort left it)
void launch_static_lists(const float4* pf, const StaticHeader* hdr, const uint32_t* start,
                         const int32_t* order, const uint32_t* groups, int32_t* lists,
                         int32_t* counts, int* status, cudaStream_t s);
void launch_snapshot(int64_t n, const Fields& F, cudaStream_t s);
