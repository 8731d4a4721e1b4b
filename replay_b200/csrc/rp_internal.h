// Internal types shared by the host driver and the kernel translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <utility>
#include <cstdlib>
#include <vector>

#include "../../include/replay.h"

namespace rp {

struct FlowThresholds {
  unsigned long long te, ti, tr;
  int te_all, ti_all, tr_all;
  int lead;                      // every threshold's first 8, 4 or 0 bits are 0
  uint32_t me[8], mi[8], mr[8];  // their top 8 bits as masks, most significant first
};

// ---- errors ---------------------------------------------------------------
void set_error(const char *fmt, ...);
rp_status cuda_fail(cudaError_t e, const char *what);
#define RP_TRY_CUDA(call)                                  \
  do {                                                     \
    cudaError_t _e = (call);                               \
    if (_e != cudaSuccess) return ::rp::cuda_fail(_e, #call); \
  } while (0)
#define RP_TRY(call)                 \
  do {                               \
    rp_status _s = (call);           \
    if (_s != RP_OK) return _s;      \
  } while (0)

// ---- device buffer ----------------------------------------------------------
// Device blocks released while no device work can touch them are kept for
// reuse instead of going back through cudaFree, whose device-wide wait and
// unmapping dominate closing a simulation or a graph and whose matching
// cudaMalloc calls dominate creating the next one.  An owner parks its
// buffers (ParkGuard) after synchronizing the device; DevBuf::alloc takes
// the smallest kept block of the current device that fits (at most twice
// the request); a failing cudaMalloc returns that device's kept blocks and
// retries.  At most kCacheBytes stay kept per device (the oldest go first; a
// larger block is freed); rp_release_cached_memory returns them all.
constexpr size_t kCacheBytes = size_t(8) << 30;
void *cache_take(int device, size_t n, size_t *cap);
void cache_put(int device, void *p, size_t cap);
void cache_trim(int device);  // -1: every device
extern thread_local int g_park;  // > 0: releases on this thread keep their blocks

// Declared before the buffers it covers (so it is destroyed after them) and
// armed once the device work that used them has completed: from then on the
// buffers released on this thread are kept instead of freed.
struct ParkGuard {
  bool armed = false;
  ParkGuard() = default;
  ParkGuard(const ParkGuard &) = delete;
  ParkGuard &operator=(const ParkGuard &) = delete;
  void arm() {
    if (!armed) {
      armed = true;
      ++g_park;
    }
  }
  // Waits for all work on `device` (the wait cudaFree would have made: work
  // a caller enqueued on its own streams may still read the buffers), then
  // arms; the caller's current device is left as it was.
  void arm_after_sync(int device) {
    int cur = 0;
    const bool have_cur = cudaGetDevice(&cur) == cudaSuccess;
    if (cudaSetDevice(device) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess) arm();
    if (have_cur) cudaSetDevice(cur);
    (void)cudaGetLastError();
  }
  ~ParkGuard() {
    if (armed) --g_park;
  }
};

struct DevBuf {
  void *ptr = nullptr;
  size_t bytes = 0;
  size_t cap = 0;     // bytes of the block behind ptr (>= bytes)
  int dev = 0;        // device of the block
  bool owned = true;  // false: a view of memory this buffer must not free
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  ~DevBuf() { release(); }
  rp_status alloc(size_t n) {
    release();
    if (n == 0) n = 16;
    int d = 0;
    cudaGetDevice(&d);
    size_t c = 0;
    if (void *p = cache_take(d, n, &c)) {
      ptr = p;
      bytes = n;
      cap = c;
      dev = d;
      return RP_OK;
    }
    cudaError_t e = cudaMalloc(&ptr, n);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      cache_trim(d);
      e = cudaMalloc(&ptr, n);
    }
    if (e != cudaSuccess) {
      ptr = nullptr;
      (void)cudaGetLastError();
      set_error("cudaMalloc of %zu bytes failed: %s", n, cudaGetErrorString(e));
      return RP_ERR_NOMEM;
    }
    bytes = n;
    cap = n;
    dev = d;
    return RP_OK;
  }
  void release() {
    if (ptr && owned) {
      if (g_park > 0)
        cache_put(dev, ptr, cap);
      else
        cudaFree(ptr);
    }
    ptr = nullptr;
    bytes = 0;
    cap = 0;
    owned = true;
  }
  // Exchanges the blocks of two buffers (pointer, sizes, device, ownership:
  // a block's size must travel with it, or it would be kept under the wrong
  // size).
  void swap(DevBuf &o) {
    std::swap(ptr, o.ptr);
    std::swap(bytes, o.bytes);
    std::swap(cap, o.cap);
    std::swap(dev, o.dev);
    std::swap(owned, o.owned);
  }
  // Points at memory owned elsewhere (no allocation; release() won't free it).
  void borrow(void *p, size_t n) {
    release();
    ptr = p;
    bytes = n;
    owned = false;
  }
  template <typename T>
  T *as() const {
    return static_cast<T *>(ptr);
  }
};

// ---- large copies between pageable host memory and the device (transfer.cpp) ----
struct HostPart {
  void *dev;
  const void *host;
  size_t bytes;
};
rp_status upload(int device, const HostPart *parts, int n);
rp_status download(int device, void *host, const void *dev, size_t n);
void touch_pages(void *host, size_t n);
void release_slots();

// ---- interval index -----------------------------------------------------------
// Contacts live in "stored coordinates" (the reference interval database's
// orientation rule, see graph.cpp) and are partitioned into duration classes:
// class 0 holds durations <= 1 s (including empty and inverted intervals),
// class c >= 1 holds durations in (2^(c-1), 2^c].  Inside a class contacts
// are ordered by start, so the candidates of a query [qs, qe) in class c are
// the contiguous run with start in (qs - 2^c, qe): two binary searches.
constexpr int kClasses = 64;

struct CandRange {
  int64_t lo;     // first candidate, index into the class-ordered arrays
  int64_t count;  // candidates in this class
  int64_t prefix; // candidates in earlier ranges of the same window
};

struct WinDesc {
  int64_t ws, we;        // window [ws, we)
  int64_t qs, qe;        // query actually run (mirrored when ws < 0)
  int64_t n_candidates;  // sum of range counts
  float scale;           // 1 / steps in the window (reference weight scale)
  int32_t range_off;     // first CandRange of this window
  int32_t n_ranges;
  int32_t may_truncate;  // candidates exceed the hit cap
  int64_t hit_off;       // first hit of this window in its group's list
};

// Consecutive windows built by one chain of launches.  In the workspace the
// window in slot k holds its hits from hit_off, its pairs and ranks from
// 2 * hit_off, and its per-node arrays from k * n (row pointers: k * (n + 1)).
struct WindowGroup {
  int32_t first = 0, count = 0;
  int32_t truncate = 0;  // some window's candidates exceed the hit cap
  int64_t candidates = 0, max_candidates = 0;
};

struct Graph {
  int device = 0;
  int32_t n_nodes = 0, n_index = 0;
  int64_t n_contacts = 0, nlists = 0, n_malformed = 0;
  int64_t t_min = 0, t_max = 0;
  int32_t n_classes_used = 0;
  std::vector<int64_t> class_off;  // kClasses + 1 offsets
  DevBuf cs, ce;                   // int64 stored start / end, class order
  DevBuf cu, cv;                   // int32 endpoints (u <= v)
  DevBuf crank;                    // int32 position in (start asc, end desc) order
};

// Contacts read from a text file: malloc'd arrays of n entries in file
// order (u <= v, compressed indices), owned by this object until release().
struct ParsedContacts {
  int32_t n_nodes = 0, n_index = 0;
  int64_t n_malformed = 0, n = 0;
  int64_t *start = nullptr, *end = nullptr;
  int32_t *u = nullptr, *v = nullptr;
  ParsedContacts() = default;
  ParsedContacts(const ParsedContacts &) = delete;
  ParsedContacts &operator=(const ParsedContacts &) = delete;
  ~ParsedContacts() { release_all(); }
  void release_all() {
    free(start), free(end), free(u), free(v);
    start = end = nullptr;
    u = v = nullptr;
  }
  void release() { start = end = nullptr, u = v = nullptr; }  // ownership passed on
};
rp_status parse_contact_file(const char *path, ParsedContacts &out);
// Builds the device interval index of n contacts given in host memory;
// ingest.cu.  `raw`: the endpoints come as the caller gave them; they are
// ordered (u <= v), checked and counted (g.n_index) on the device, and *bad is
// the first contact with an endpoint outside [0, n_nodes), or -1.
rp_status graph_build_device(Graph &g, const int64_t *start, const int64_t *end,
                             const int32_t *u, const int32_t *v, int64_t n, int32_t n_nodes,
                             bool raw, int64_t *bad);

// Plans the queries of the windows [ws[k], ws[k] + length): candidate ranges
// appended to `ranges`, one WinDesc each to `wins`.  The binary searches run
// on the device (ingest.cu).
rp_status plan_windows(const Graph &g, const std::vector<int64_t> &ws, int64_t length,
                       const std::vector<float> &scale, int64_t cap,
                       std::vector<CandRange> &ranges, std::vector<WinDesc> &wins);
// One window, planned in the stream: its descriptor, its ranges (kClasses
// entries) and the number of its candidates stay on the device; with more than
// `limit` of them the descriptor is of an empty window.
void enqueue_plan_window(const Graph &g, int64_t ws, int64_t we, float scale, int64_t cap,
                         int64_t limit, WinDesc *win, CandRange *ranges, int64_t *total,
                         cudaStream_t st);

// ---- window builder ----------------------------------------------------------
struct Hit {
  int32_t rank;  // position in (start asc, end desc) order
  int32_t u;     // < 0: counts toward the hit cap but carries no weight
  int32_t v;
  int32_t w;     // int32 seconds or float bits
};

// Rows with many pairs, listed while a window's row pointers are written:
// rows of more than kHeavyPairs pairs from the front of the list, of more than
// kHugePairs pairs from its end; counts[0] and counts[2] of them.  A sparse
// window lists entries of its RowList.
constexpr int32_t kHeavyPairs = 48, kHugePairs = 256;
struct HeavyRows {
  const int32_t *rows, *end;
  const unsigned long long *counts;
};
// The rows of a sparse window that have pairs, in any order (WindowWorkspace
// with sparse set), or null: every row by its row pointers.
struct RowList {
  const int32_t *rows;       // counts[1] of them
  const int2 *span;          // {first pair, pairs}
  const unsigned long long *counts;
  int64_t bound;             // at most so many rows
};

struct WindowWorkspace {
  int32_t n_nodes = 0;
  // Windows with pairs in few rows: only those rows are counted, placed and
  // listed, so that a window costs its contacts and not its nodes.
  bool sparse = false;
  int64_t cap_hits = 0, cap_entries = 0;
  int32_t n_tiles = 0;
  // a group of windows, slot after slot (WindowGroup); G slots
  DevBuf hits;      // Hit[cap_hits]
  DevBuf entries;   // int2 {col, weight}[cap_entries]
  DevBuf erank;     // int32[cap_entries], sorted rows only (as the next two)
  DevBuf tmp_e;     // int2[cap_entries]  radix ping-pong for hub rows
  DevBuf tmp_r;     // int32[cap_entries]
  DevBuf row_ptr;   // int32[G][n+1]
  DevBuf deg;       // int32[G][n] degrees, counted down to zero while pairs are placed
  DevBuf tiles;     // int32[G][n_tiles]
  DevBuf hpos;      // int2[cap_hits], sparse: a hit's positions in its two rows
  DevBuf rows;      // int32[cap_entries], sparse: rows with pairs
  DevBuf span;      // int2[cap_entries], sparse: their first pairs and pairs
  DevBuf placed;    // u64[G], sparse: pairs placed so far
  DevBuf counters;  // u64[G][4]: heavy rows, long rows (sparse: listed rows), huge rows,
                    // predicate hits
  DevBuf long_rows; // int32[G][n]: heavy rows (unsorted rows) or rows to sort in a block
  DevBuf win;       // WinDesc[n_windows]
  DevBuf ranges;    // CandRange[...]
  int64_t bytes() const {
    int64_t b = 0;
    for (const DevBuf *d : {&hits, &entries, &erank, &tmp_e, &tmp_r, &row_ptr, &deg, &tiles, &hpos,
                            &rows, &span, &placed, &counters, &long_rows, &win, &ranges})
      b += (int64_t)d->bytes;
    return b;
  }
};

// Room for any group of at most `slots` windows and `cap_hits` candidates.
rp_status window_workspace_alloc(WindowWorkspace &w, int32_t n_nodes, int32_t slots,
                                 int64_t cap_hits, bool sort_rows, bool sparse,
                                 const std::vector<WinDesc> &wins,
                                 const std::vector<CandRange> &ranges);
// Splits the windows into groups (`single`: one window each) and places each
// window's hits in its group's list.
void plan_window_groups(std::vector<WinDesc> &wins, int32_t n_nodes, bool single, bool sparse,
                        std::vector<WindowGroup> &groups);
// Whether windows of at most max_candidates contacts on n_nodes rows are built
// sparse: fewer than one row in four has pairs then.
inline bool sparse_windows(int64_t max_candidates, int32_t n_nodes) {
  return 8 * max_candidates < n_nodes;
}

// ---- mean-field replay (meanfield.cu) ----
struct MfRates {
  float beta, p_ei, p_ir, p_rs;
  int32_t has_exposed, ir_to_s;
};
int32_t mf_warps(int32_t n);  // rows of the per-warp partial sums
// after_kernel: the previous work on the stream is another mf_step or
// mf_adjoint (which this one may overlap up to its first dependent load).
void mf_step(const int32_t *rp, const int2 *ent, int32_t n, float scale, const MfRates *r,
             const float *sus, const float *x, float *xo, float *q_out, float *e_out,
             float *inc_part, bool after_kernel, cudaStream_t st);
void mf_incidence(const float *part, int32_t nwarp, int32_t T, float *inc, cudaStream_t st);
// early: x, q and e come from before the previous kernel.
void mf_adjoint(int32_t n, const int32_t *rp_c, const int2 *ent_c, const float *z_in,
                const float *a_in, const float *x, const float *q, const float *e,
                const float *ginc, int32_t tl, float scale, const MfRates *r, const float *sus,
                float *a_out, float *z_out, float *gsus, double *gpart, bool early,
                bool after_kernel, cudaStream_t st);
// A whole forward, or adjoint, by one thread block cluster: up to
// kMfClusterNodes nodes, at least one step, every state kept (states holds
// x_0 .. x_T, q and e a plane per step).
constexpr int32_t kMfClusterNodes = 4096;
struct MfStep {
  const int32_t *row_ptr;
  const int2 *entries;
  float scale;
};
void mf_forward_cluster(const MfStep *steps, int32_t n_steps, int32_t n, const MfRates *r,
                        const float *sus, float *states, float *q, float *e, float *inc_part,
                        cudaStream_t st);
void mf_reverse_cluster(const MfStep *steps, int32_t n_steps, int32_t n, const MfRates *r,
                        const float *sus, const float *a_in, const float *states, const float *q,
                        const float *e, const float *ginc, float *gx0, float *gsus, double *gpart,
                        cudaStream_t st);
void mf_finish(const double *gpart, int32_t nwarp, double *out, cudaStream_t st);

// ---- node-state text (text.cu) ----
int64_t text_line_bound(int32_t n_nodes);  // bytes of one line at most
int64_t text_segments(int32_t n_nodes);    // segments of one replica's lines
void enqueue_states_text(const uint8_t *cls, int32_t n, int32_t r0, int32_t r1, int64_t ts,
                         int64_t *seglen, int64_t *segoff, char *out,
                         cudaStream_t st);

// Scan tiles the window builder uses for n_nodes rows.
int32_t window_scan_tiles(int32_t n_nodes);

enum WeightKind { kWeightF32 = 0, kWeightI32 = 1 };

// Enqueues the CSR build of a group of windows into ws.row_ptr / ws.entries;
// returns the kernels launched.  sort_rows: order each row by (col, rank) and
// merge duplicates in place (merged-away entries keep their column with
// weight 0).
int enqueue_window_build(const Graph &g, WindowWorkspace &ws, const WindowGroup &grp, int64_t cap,
                         int weight_kind, bool sort_rows, cudaStream_t st);
// Compacts the sorted, merged CSRs of the group in ws: row pointers to
// row_ptr_out (n + 1 per window), pairs (merged-away entries dropped) to
// entries_out + entries_off[window] (device offsets; null: one window, at
// entries_out; without entries_out only the row pointers are made).  With
// `heavy` the rows with many pairs are listed from heavy_off[window] up to the
// next window's, their counts (4 words a window, zeroed by the caller) in
// heavy_counts.
void enqueue_window_compact(WindowWorkspace &ws, const WindowGroup &grp, int32_t *row_ptr_out,
                            int2 *entries_out, const int64_t *entries_off, cudaStream_t st,
                            int32_t *heavy = nullptr, const int64_t *heavy_off = nullptr,
                            unsigned long long *heavy_counts = nullptr);

// ---- kernels of the step loop -------------------------------------------------
struct StepConsts {
  uint32_t key0, key1;
  uint32_t rk[20];    // Philox round keys of (key0, key1)
  FlowThresholds th;  // p_ei, p_ir, p_rs as 64-bit fixed point
  float step_size;
  float neg_log_base;  // -logf(1 - infect_prob), countdown mode
  int32_t upper, medium, lower, E, I, R;  // countdown ranges / durations
  float p_ei, p_ir, p_rs;
  int32_t has_exposed, ir_to_s;
  float beta;
  const float *beta_r;  // device, may be null
  const float *beta_word;  // device, with beta_r: max |beta_r| of each 32-replica word
  const float *sus;     // device, may be null
  uint32_t roff;        // replica offset of the stream layout (multiple of 32)
};

// Plain path (column-major N x M state, per-replica SpMV + elementwise).
void plain_init(int transition, void *state, int32_t n, int32_t m,
                float p0, int32_t k_exact, const StepConsts &c,
                cudaStream_t st);
void plain_spmv(int transition, const int32_t *row_ptr, const int2 *entries,
                const void *state, void *exposure, int32_t n, int32_t m,
                const StepConsts &c, cudaStream_t st);
void plain_transition(int transition, void *state, const void *exposure,
                      int32_t n, int32_t m, uint32_t step, float scale,
                      int32_t *counts_row, const StepConsts &c,
                      cudaStream_t st);
void plain_count(int transition, const void *state, int32_t n, int32_t m,
                 int32_t *counts_row, const StepConsts &c, cudaStream_t st);
void plain_classify(int transition, const void *state, int32_t n, int32_t m,
                    uint8_t *out, const StepConsts &c, cudaStream_t st);

// Batched path (bit-packed replica words).
struct PackedTask {
  int32_t row_begin, row_end;  // rows of one network
  int32_t slice;               // 32 four-word columns (128 words) per slice
  int32_t count_base;          // index of replica 0 of this network in counts
};
struct PackedLayout {
  int32_t n_nodes;
  int32_t words;      // words per node row, padded to a multiple of 4
  int32_t vwords;     // words holding replicas: ceil(m / 32)
  int32_t q4;         // four-word columns per row (words / 4)
  int32_t m;          // replicas per network
  uint32_t last_mask; // valid bits of word vwords - 1
  int32_t lb;         // bitmap bits per row: 1 << lb, the power of 2 >= min(q4, 32)
  int32_t n_slices;   // slices of 32 four-word columns
  int64_t bit_words;  // words of one item bitmap (packed.cu)
  int32_t n_tasks;
};
rp_status packed_prepare();  // kernel attributes, once per device
// `bits`: the four item bitmaps (act, inf, sus, evb), or null (countdown mode).
// Returns the kernels launched.
int packed_init(const PackedLayout &L, uint32_t *sa, uint32_t *sb,
                uint32_t *mask, uint32_t *bits, float p0, int32_t k_exact,
                const int32_t *net_first_row, const int32_t *net_rows,
                int32_t n_nets, const StepConsts &c, cudaStream_t st);
// One step: exposure + infection draws (k_infect), then transitions, counts
// and the next infectious mask (k_flow).
void packed_infect(const PackedLayout &L, const int32_t *row_ptr, const int2 *entries,
                   const RowList &list, const HeavyRows &heavy, const uint32_t *mask, const uint32_t *sa,
                   const uint32_t *sb, uint32_t *evs, uint32_t *bits, uint32_t step, float scale,
                   const StepConsts &c, cudaStream_t st);
// net_first: first row of each of several networks (their counts follow one
// another in ev_row and rs_row).
void packed_flow(const PackedLayout &L, uint32_t *mask, uint32_t *sa, uint32_t *sb, uint32_t *evs,
                 uint32_t *bits, unsigned long long *ev_row, unsigned long long *rs_row,
                 const int32_t *net_first, int32_t n_nets, uint32_t step, const StepConsts &c,
                 cudaStream_t st);
// Batched countdown mode (countdown.cu) as changes of state at fixed ages: a
// source is a set of replicas (a bit plane and its item bitmap) that enters
// one summary class from another in this step.
struct CdSource {
  uint32_t *plane, *bits;
  int32_t clear;           // the set is not needed after this change
  int32_t from, to;        // summary classes (0 S, 1 E, 2 I, 3 R)
  int32_t infectious;      // from this change on
  int32_t busy;            // 0: susceptible from this change on
};
constexpr int kCdSources = 8;
struct CdSources {
  CdSource s[kCdSources];
  int32_t n;
};
void cd_bits(const PackedLayout &L, const uint32_t *plane, uint32_t *bits, cudaStream_t st);
void cd_infect(const PackedLayout &L, const int32_t *row_ptr, const int2 *entries,
               const uint32_t *mask, const uint32_t *busy, uint32_t *evs, const uint32_t *infb,
               const uint32_t *susb, uint32_t *evb, uint32_t step, const StepConsts &c,
               cudaStream_t st);
// ca, cb: class planes (packed_classify's), or null.
void cd_flow(const PackedLayout &L, const CdSources &src, uint32_t *busy, uint32_t *mask,
             uint32_t *ca, uint32_t *cb, uint32_t *infb, uint32_t *susb,
             unsigned long long *ev_row, const int32_t *net_first, int32_t n_nets,
             cudaStream_t st);
// The same rule with per-replica codes into the host's countdown table (next |
// class << 16 | infectious << 18), 1 or 2 bytes each: for replays whose sets
// of replicas per age would not fit.
rp_status cd_prepare();
void cd_init(const PackedLayout &L, const PackedTask *tasks, const uint32_t *infected,
             void *codes, int code_bytes, uint32_t *mask, const uint32_t *tab,
             uint32_t init_code, unsigned long long *init_counts, cudaStream_t st);
void cd_step(const PackedLayout &L, const PackedTask *tasks, const int32_t *row_ptr,
             const int2 *entries, const uint32_t *mask_in, uint32_t *mask_out, void *codes,
             int code_bytes, const uint32_t *tab, int32_t n_codes, uint32_t infect_code,
             unsigned long long *ev_row, uint32_t step, const StepConsts &c, cudaStream_t st);
void cd_finalize(const unsigned long long *init, const unsigned long long *ev, int32_t steps,
                 int32_t per_row, const int32_t *net_size, int32_t m, int32_t *counts,
                 cudaStream_t st);
void cd_classify(const PackedLayout &L, const void *codes, int code_bytes, const uint32_t *tab,
                 uint8_t *out, cudaStream_t st);
void packed_count(const PackedLayout &L, const PackedTask *tasks,
                  const uint32_t *sa, const uint32_t *sb,
                  unsigned long long *counts_row, cudaStream_t st);
void packed_finalize_events(const unsigned long long *init,
                            const unsigned long long *ev,
                            const unsigned long long *rs, int32_t steps,
                            int32_t per_row, const int32_t *net_size,
                            int32_t m, int32_t has_exposed, int32_t ir_to_s,
                            int32_t *counts, cudaStream_t st);
void packed_classify(const PackedLayout &L, const uint32_t *sa,
                     const uint32_t *sb, uint8_t *out, cudaStream_t st);
void packed_exposure(const int32_t *row_ptr, const int2 *entries, int32_t n,
                     const uint32_t *masks, int32_t words, int32_t m,
                     int64_t *exposure, cudaStream_t st);
void plain_spmv_f32_raw(const int32_t *row_ptr, const int32_t *col,
                        const float *val, int32_t n, const float *b, float *c,
                        int32_t m, cudaStream_t st);

}  // namespace rp

// rp_sim_create_batch with another bound on the bytes of the countdown rule's
// sets (0: the code table), so that a test can take the code table, the form of
// replays too large for the sets, at sizes that an oracle can follow.
extern "C" RP_API rp_status rp_sim_create_bounded(const rp_graph *g, const rp_params *p,
                                                  const int32_t *net_first, int32_t n_networks,
                                                  int64_t set_bytes, rp_sim **out);

struct rp_graph {
  rp::ParkGuard park;  // destroyed after g: its blocks are kept for reuse
  rp::Graph g;
  double prep_ms = 0.0, build_ms = 0.0;  // creation phases (rp_graph_info)
  ~rp_graph() { park.arm_after_sync(g.device); }
};
