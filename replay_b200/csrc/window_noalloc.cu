// Allocation-free window CSR build (rp_window_csr_noalloc).
//
// The same device builder as rp_window_csr (interval-index candidate scan,
// hit cap, row fill, per-row sort and duplicate merge, compaction), with
// every scratch buffer carved out of one file-scope device array instead of
// cudaMalloc'd workspaces, and the result left in caller-owned device
// buffers.  It exists for callers that must not allocate or free device
// memory on this path: cudaFree waits for the whole device, so a process that
// keeps other streams busy (or hands all device memory to its own pool) cannot
// afford it per window.
//
// Limits: at most kNoAllocMaxNodes nodes in the graph and kNoAllocMaxCandidates
// candidate contacts in one window (contacts whose stored start falls inside
// the window's scan range); larger requests fail with RP_ERR_RANGE.  The
// scratch array is shared by all calls on a device, so calls must not
// overlap: issue them from one thread on one stream at a time.  Every call
// looks up the array's address (cudaGetSymbolAddress; the first call in a
// context may load this module) and synchronizes the stream before it returns,
// so a call cannot be made while the stream is being captured.  The window is
// planned in the stream, in front of its build: planned and waited for first, a
// call took 20 us longer (107 us against 86 for a window of 53 contacts).  The caller's current device is
// restored on return.
#include "rp_internal.h"

namespace rp {
namespace {

constexpr int32_t kNoAllocMaxNodes = 65536;
constexpr int64_t kNoAllocMaxCandidates = 131072;
constexpr int32_t kNoAllocMaxTiles = 64;

constexpr size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Byte offsets of the scratch regions.
constexpr size_t kHitsOff = 0;
constexpr size_t kEntOff = kHitsOff + align256(sizeof(Hit) * kNoAllocMaxCandidates);
constexpr size_t kErankOff = kEntOff + align256(sizeof(int2) * 2 * kNoAllocMaxCandidates);
constexpr size_t kTmpEOff = kErankOff + align256(sizeof(int32_t) * 2 * kNoAllocMaxCandidates);
constexpr size_t kTmpROff = kTmpEOff + align256(sizeof(int2) * 2 * kNoAllocMaxCandidates);
constexpr size_t kRowPtrOff = kTmpROff + align256(sizeof(int32_t) * 2 * kNoAllocMaxCandidates);
constexpr size_t kNodeBytes = align256(sizeof(int32_t) * (kNoAllocMaxNodes + 1));
constexpr size_t kDegOff = kRowPtrOff + kNodeBytes;
constexpr size_t kLongOff = kDegOff + kNodeBytes;
constexpr size_t kOutPtrOff = kLongOff + kNodeBytes;
constexpr size_t kTilesOff = kOutPtrOff + kNodeBytes;
constexpr size_t kCtrOff = kTilesOff + align256(sizeof(int32_t) * kNoAllocMaxTiles);
constexpr size_t kTotalOff = kCtrOff + sizeof(unsigned long long) * 4;  // read with the counters
constexpr size_t kWinOff = kCtrOff + align256(sizeof(unsigned long long) * 5);
constexpr size_t kRangeOff = kWinOff + align256(sizeof(WinDesc));
constexpr size_t kScratchBytes = kRangeOff + align256(sizeof(CandRange) * kClasses);  // ~9 MB

static __device__ __align__(256) unsigned char g_window_scratch[kScratchBytes];

// Address of the scratch array in the current device's context.  Looked up
// on every call (no allocation, and cheap): a cached address would go stale
// if the primary context were reset and the module reloaded elsewhere.
rp_status scratch_address(unsigned char **out) {
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_window_scratch);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(window scratch)");
  *out = static_cast<unsigned char *>(p);
  return RP_OK;
}

// Makes `device` current for the scope and restores the caller's device.
struct DeviceScope {
  int prev = -1;
  cudaError_t err = cudaSuccess;
  explicit DeviceScope(int device) {
    err = cudaGetDevice(&prev);
    if (err == cudaSuccess && prev != device) err = cudaSetDevice(device);
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

rp_status window_csr_noalloc(const Graph &g, int64_t ws, int64_t we, float scale, int weight_kind,
                             int ncls_cap, int32_t *d_row_ptr, int32_t *d_entries,
                             int64_t capacity, int64_t *nnz, int64_t *n_hits, cudaStream_t st) {
  if (!d_row_ptr || !nnz || !n_hits || capacity < 0 || (capacity > 0 && !d_entries) || we <= ws ||
      (weight_kind != kWeightF32 && weight_kind != kWeightI32)) {
    set_error("invalid window CSR request");
    return RP_ERR_ARG;
  }
  if (weight_kind == kWeightI32 && we - ws > INT32_MAX) {
    set_error("integer weights need a window of at most 2^31-1 s");
    return RP_ERR_RANGE;
  }
  if (g.n_nodes > kNoAllocMaxNodes) {
    set_error("graph has %d nodes; the allocation-free window build takes at most %d", g.n_nodes,
              kNoAllocMaxNodes);
    return RP_ERR_RANGE;
  }
  DeviceScope scope(g.device);
  if (scope.err != cudaSuccess) return cuda_fail(scope.err, "cudaSetDevice");
  unsigned char *base = nullptr;
  RP_TRY(scratch_address(&base));

  const int64_t cap = ncls_cap ? (g.nlists > 0 ? g.nlists : 1) : INT64_MAX;
  const int32_t n = g.n_nodes;
  if (window_scan_tiles(n) > kNoAllocMaxTiles) {
    set_error("internal: scan tiles exceed the scratch layout");
    return RP_ERR_RANGE;
  }

  // sized for the most candidates that a window of this graph can have
  const int64_t most = g.n_contacts < kNoAllocMaxCandidates ? g.n_contacts : kNoAllocMaxCandidates;
  WindowWorkspace w;
  w.n_nodes = n;
  w.cap_hits = most < 1 ? 1 : most;
  w.cap_entries = 2 * w.cap_hits;
  w.n_tiles = window_scan_tiles(n);
  w.hits.borrow(base + kHitsOff, sizeof(Hit) * w.cap_hits);
  w.entries.borrow(base + kEntOff, sizeof(int2) * w.cap_entries);
  w.erank.borrow(base + kErankOff, sizeof(int32_t) * w.cap_entries);
  w.tmp_e.borrow(base + kTmpEOff, sizeof(int2) * w.cap_entries);
  w.tmp_r.borrow(base + kTmpROff, sizeof(int32_t) * w.cap_entries);
  w.row_ptr.borrow(base + kRowPtrOff, sizeof(int32_t) * ((size_t)n + 1));
  w.deg.borrow(base + kDegOff, sizeof(int32_t) * ((size_t)n + 1));
  w.long_rows.borrow(base + kLongOff, sizeof(int32_t) * ((size_t)n + 1));
  w.tiles.borrow(base + kTilesOff, sizeof(int32_t) * (size_t)w.n_tiles);
  w.counters.borrow(base + kCtrOff, sizeof(unsigned long long) * 4);
  w.win.borrow(base + kWinOff, sizeof(WinDesc));
  w.ranges.borrow(base + kRangeOff, sizeof(CandRange) * kClasses);
  int32_t *out_ptr = reinterpret_cast<int32_t *>(base + kOutPtrOff);

  // The builder zeroes its hit counters and expects zero degrees (a call that
  // failed on the way may have left others here).
  RP_TRY_CUDA(cudaMemsetAsync(w.deg.ptr, 0, w.deg.bytes, st));
  enqueue_plan_window(g, ws, we, scale, cap, kNoAllocMaxCandidates, w.win.as<WinDesc>(),
                      w.ranges.as<CandRange>(), reinterpret_cast<int64_t *>(base + kTotalOff), st);
  WindowGroup grp;
  grp.count = 1;
  grp.truncate = g.n_contacts > cap;  // the window's descriptor decides
  grp.candidates = grp.max_candidates = most;
  enqueue_window_build(g, w, grp, cap, weight_kind, true, st);
  // compacted pairs go to tmp_e (free once the rows are sorted); nothing is
  // written for the caller before the numbers are known
  enqueue_window_compact(w, grp, out_ptr, w.tmp_e.as<int2>(), nullptr, st);
  RP_TRY_CUDA(cudaGetLastError());
  unsigned long long ctr[5] = {0, 0, 0, 0, 0};  // the counters and the number of candidates
  int32_t total = 0;
  RP_TRY_CUDA(cudaMemcpyAsync(ctr, w.counters.ptr, sizeof(ctr), cudaMemcpyDeviceToHost, st));
  RP_TRY_CUDA(cudaMemcpyAsync(&total, out_ptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  RP_TRY_CUDA(cudaStreamSynchronize(st));
  if ((int64_t)ctr[4] > kNoAllocMaxCandidates) {
    set_error("window [%lld, %lld) scans %lld candidate contacts; the allocation-free window "
              "build takes at most %lld", (long long)ws, (long long)we, (long long)ctr[4],
              (long long)kNoAllocMaxCandidates);
    return RP_ERR_RANGE;
  }
  *nnz = total;
  *n_hits = (int64_t)ctr[3] < cap ? (int64_t)ctr[3] : cap;
  RP_TRY_CUDA(cudaMemcpyAsync(d_row_ptr, out_ptr, sizeof(int32_t) * ((size_t)n + 1),
                              cudaMemcpyDeviceToDevice, st));
  if (total > 0 && total <= capacity)
    RP_TRY_CUDA(cudaMemcpyAsync(d_entries, w.tmp_e.ptr, sizeof(int2) * (size_t)total,
                                cudaMemcpyDeviceToDevice, st));
  RP_TRY_CUDA(cudaStreamSynchronize(st));
  if (total > capacity) {
    set_error("CSR has %d entries, capacity %lld", total, (long long)capacity);
    return RP_ERR_RANGE;
  }
  return RP_OK;
}

}  // namespace
}  // namespace rp

extern "C" RP_API rp_status rp_window_csr_noalloc(rp_graph *g, int64_t ws, int64_t we,
                                                  float scale, int32_t weight_kind,
                                                  int32_t ncls_cap, int32_t *d_row_ptr,
                                                  int32_t *d_entries, int64_t capacity,
                                                  int64_t *nnz, int64_t *n_hits, void *stream) {
  if (!g) {
    rp::set_error("null graph");
    return RP_ERR_ARG;
  }
  return rp::window_csr_noalloc(g->g, ws, we, scale, weight_kind, ncls_cap, d_row_ptr, d_entries,
                                capacity, nnz, n_hits, static_cast<cudaStream_t>(stream));
}
