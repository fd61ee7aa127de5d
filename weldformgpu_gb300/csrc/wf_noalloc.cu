// wf_noalloc.cu — neighbour search that allocates no device memory.
//
// wf_find_neighbors_static() gives the same lists as wf_find_neighbors()
// followed by wf_get_neighbors() (cuNSearch's float32 rule, candidates in the
// z, y, x cell order, ascending particle index inside a cell, at most 70 per
// particle), for callers that cannot call cudaMalloc: hosts whose framework
// owns every device allocation through its own pool or allocator, hosts that
// run under a fixed device-memory budget reserved up front, and code that must
// not allocate while other work runs on the device.  The caller passes device
// buffers for the positions and the output lists; the temporaries of the
// search (cell ids, cell counts and offsets, sorted indices and positions, the
// grid bounds, the scan's block sums) live in one file-scope device array,
// `g_static_scratch`, of fixed size.  Loading the library reserves it on every
// GPU the process uses, until the process exits.
//
// Sharing rules, stated in the header too: every call uses the same array and
// leaves its contents behind; each call clears what must start at zero (the
// grid bounds, the status word, the per-cell counters).  Two calls whose GPU
// work overlaps on one device (two streams, or two host threads at once) race
// on the array and give wrong lists; callers serialise them.
#include <climits>
#include <cstdio>
#include <mutex>

#include "wf_common.cuh"
#include "wf_nsearch.cuh"

namespace {

constexpr int64_t kMaxParticles = WF_STATIC_MAX_PARTICLES;
constexpr int64_t kMaxCells = WF_STATIC_MAX_CELLS;
constexpr int64_t kScanWords = 1024;   // block sums of the scan over kMaxCells entries

constexpr int64_t align256(int64_t b) { return (b + 255) / 256 * 256; }
// byte offsets inside the scratch array
constexpr int64_t kOffHeader = 0;                                     // StaticHeader
constexpr int64_t kOffPos = kOffHeader + 256;                         // float4[n] positions
constexpr int64_t kOffSorted = kOffPos + align256(16 * kMaxParticles);   // float4[n] cell order
constexpr int64_t kOffCellId = kOffSorted + align256(16 * kMaxParticles);  // uint32[n]
constexpr int64_t kOffOrder = kOffCellId + align256(4 * kMaxParticles);    // int32[n] index
constexpr int64_t kOffStart = kOffOrder + align256(4 * kMaxParticles);     // uint32[cells + 1]
constexpr int64_t kOffCount = kOffStart + align256(4 * (kMaxCells + 1));   // uint32[cells]
constexpr int64_t kOffScan = kOffCount + align256(4 * kMaxCells);          // uint32[kScanWords]
constexpr int64_t kScratchBytes = kOffScan + align256(4 * kScanWords);
static_assert(kScratchBytes == WF_STATIC_SCRATCH_BYTES, "header and layout disagree");
static_assert(sizeof(StaticHeader) <= 256 && kMaxCells / 1024 + 1 <= kScanWords &&
                  2 * (kMaxParticles / 32) <= kMaxCells,
              "scratch layout");

}  // namespace

// The device scratch.  In host code `g_static_scratch` names a host-side
// stand-in for the symbol, not a device address; the device address comes from
// cudaGetSymbolAddress, once per device.
static __device__ __align__(256) unsigned char g_static_scratch[kScratchBytes];

namespace {

void set_message(char* err, int64_t err_len, const char* msg) {
  if (err && err_len > 0) snprintf(err, (size_t)err_len, "%s", msg);
}

int fail(char* err, int64_t err_len, int code, const char* fmt, long long a = 0,
         long long b = 0) {
  char buf[256];
  snprintf(buf, sizeof buf, fmt, a, b);
  set_message(err, err_len, buf);
  return code;
}

int cuda_fail(char* err, int64_t err_len, cudaError_t e, const char* what) {
  char buf[256];
  snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
  set_message(err, err_len, buf);
  return WF_ERR_CUDA;
}

// Device address of the scratch array on the current device.  The first call
// on each device looks it up with cudaGetSymbolAddress and caches it.
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
unsigned char* g_scratch_ptr[kMaxDevices] = {};

cudaError_t scratch_on_current_device(unsigned char** out, int* dev_out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  *dev_out = dev;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess) return e;
    g_scratch_ptr[dev] = static_cast<unsigned char*>(p);
  }
  *out = g_scratch_ptr[dev];
  return cudaSuccess;
}

// a pointer the kernels may dereference: device, managed or mapped host memory
bool device_accessible(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) return true;
  return a.type == cudaMemoryTypeHost && a.devicePointer != nullptr;
}

}  // namespace

extern "C" int wf_find_neighbors_static(const double* x, int64_t n, double h, int32_t* counts,
                                        int32_t* lists, void* stream, char* err,
                                        int64_t err_len) {
  set_message(err, err_len, "");
  if (n < 0) return fail(err, err_len, WF_ERR_ARG, "particle count %lld is negative", n);
  if (n > kMaxParticles)
    return fail(err, err_len, WF_ERR_ARG,
                "particle count %lld exceeds the static scratch limit of %lld particles "
                "(WF_STATIC_MAX_PARTICLES)",
                n, kMaxParticles);
  if (!(h > 0.0) || !(h < 1.0e30))
    return fail(err, err_len, WF_ERR_ARG, "smoothing length must be positive and finite");
  if (n == 0) return WF_OK;
  if (!x || !counts || !lists)
    return fail(err, err_len, WF_ERR_ARG, "null positions, counts or lists pointer");
  if (!device_accessible(x) || !device_accessible(counts) || !device_accessible(lists))
    return fail(err, err_len, WF_ERR_ARG,
                "positions, counts and lists must be device-accessible memory");

  unsigned char* base = nullptr;
  int dev = -1;
  cudaError_t e = scratch_on_current_device(&base, &dev);
  if (e != cudaSuccess) return cuda_fail(err, err_len, e, "scratch address (cudaGetSymbolAddress)");

  cudaStream_t s = static_cast<cudaStream_t>(stream);
  StaticHeader* hdr = reinterpret_cast<StaticHeader*>(base + kOffHeader);
  float4* pf = reinterpret_cast<float4*>(base + kOffPos);
  float4* sorted = reinterpret_cast<float4*>(base + kOffSorted);
  int32_t* order = reinterpret_cast<int32_t*>(base + kOffOrder);
  CellWork W;
  W.cellid = reinterpret_cast<uint32_t*>(base + kOffCellId);
  W.rank = reinterpret_cast<uint32_t*>(sorted);      // until the sorted positions go there
  W.count = reinterpret_cast<uint32_t*>(base + kOffCount);
  W.bsum = reinterpret_cast<uint32_t*>(base + kOffScan);
  W.ticket = &hdr->scan_ticket;
  W.start = reinterpret_cast<uint32_t*>(base + kOffStart);
  W.max_cells = kMaxCells;

  // Bounds and grid (cuNSearch kComputeMinMax, computeCellInformation), the
  // counting sort by cell and the lists, all sized on the device; a grid that
  // does not fit leaves ncell = 0 and the kernels behind it do nothing.  One
  // wait, for the header.
  const float r = (float)(2.0 * h);
  launch_static_prep(n, x, pf, r, hdr, W.count, kMaxCells, s);
  launch_cell_sort(n, pf, GridDev{}, hdr, nullptr, W, order, order, sorted, &hdr->status, s);
  launch_static_lists(sorted, hdr, W.start, order, W.count, lists, counts, &hdr->status, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(err, err_len, e, "neighbour search launch");
  StaticHeader head;
  e = cudaMemcpyAsync(&head, hdr, sizeof head, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(err, err_len, e, "neighbour search");
  const int status = head.status;
  if (head.ncell == 0) {
    if (status & WF_STATUS_GRID)
      return fail(err, err_len, WF_ERR_ARG, "a position is not finite");
    int mm[6];
    bounds_from_codes(head.mm, mm);
    for (int a = 0; a < 3; a++) {
      const int64_t span = (int64_t)mm[3 + a] - (int64_t)mm[a];
      if (span < 0 || span + 5 > kMaxCells)
        return fail(err, err_len, WF_ERR_ARG,
                    "positions span %lld search radii (2h) along an axis; the static scratch "
                    "holds %lld cells (WF_STATIC_MAX_CELLS)",
                    span, kMaxCells);
    }
    for (int a = 0; a < 3; a++)
      if (head.grid.dim[a] <= 0 || head.grid.dim[a] > kMaxCells)
        return fail(err, err_len, WF_ERR_ARG,
                    "search grid needs %lld cells along an axis; the static scratch holds "
                    "%lld cells (WF_STATIC_MAX_CELLS)",
                    (long long)head.grid.dim[a], kMaxCells);
    return fail(err, err_len, WF_ERR_ARG,
                "search grid needs more than %lld cells (positions span too many radii "
                "2h); the static scratch holds %lld cells (WF_STATIC_MAX_CELLS)",
                kMaxCells, kMaxCells);
  }
  if (status & WF_STATUS_GRID)
    return fail(err, err_len, WF_ERR_NUMERIC,
                "a position is not finite or lies outside the search grid");
  return WF_OK;
}
