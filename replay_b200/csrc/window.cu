// Per-window symmetric CSR builder on the device.
//
// Replaces the reference's per-step host path: find_intervals over the NCLS
// (tool/ncls/ncls/src/intervaldb.c:426-485, called with nbuf = nlists from
// tool/gpu_cpu_temporal_sim.cu:973-991) and build_csr_from_intervals
// (tool/gpu_cpu_temporal_sim.cu:238-350: overlap weights, symmetric
// emission, qsort by (row, col), FP32 duplicate merge, counting sort).
//
// Kernels, in launch order for one group of consecutive windows (grid y):
//   k_hits      candidates of the duration-class index -> hit list (+degrees)
//   k_trunc     only when the reference's hit cap can bind: keep the cap
//               smallest ranks (radix select), then count degrees
//   k_scan_*    degrees -> row_ptr (exclusive scan)
//   k_fill      hits -> row segments {col, weight} + rank
//   k_rowsort_* rows ordered by (col, rank), duplicates merged in rank order
#include <algorithm>
#include <cstdio>

#include "rp_device.cuh"
#include "rp_internal.h"

namespace rp {
namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanTile = 4 * kScanThreads;
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ int block_excl_scan(int v, int *warp_tot,
                                               int &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(kFull, w, o);
      if (lane >= o) w += y;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  const int off = warp ? warp_tot[warp - 1] : 0;
  total = warp_tot[(blockDim.x >> 5) - 1];
  __syncthreads();
  return off + x - v;
}

__device__ __forceinline__ int block_sum(int v, int *warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = __reduce_add_sync(kFull, v);
  if (lane == 0) warp_tot[warp] = v;
  __syncthreads();
  int t = 0;
  if (warp == 0) {
    t = (lane < (int)(blockDim.x >> 5)) ? warp_tot[lane] : 0;
    t = __reduce_add_sync(kFull, t);
    if (lane == 0) warp_tot[0] = t;
  }
  __syncthreads();
  t = warp_tot[0];
  __syncthreads();
  return t;
}

// ---------------------------------------------------------------------------
// Every kernel below builds a group of consecutive windows: blockIdx.y is the
// window's slot in the group, and the per-window arrays of the workspace lie
// slot after slot (WindowGroup in rp_internal.h).
//
// k_hits writes candidate t's hit at slot t of the window's list (u = -2
// where the candidate does not overlap the window): the class ranges hold few
// candidates that miss, and a dense list would take one atomic per warp on
// one address (180,000 candidates of a replica-sweep window: 5,600 of them).
__global__ void __launch_bounds__(256)
    k_hits(const WinDesc *__restrict__ wins, const CandRange *__restrict__ ranges,
           const int64_t *__restrict__ cs, const int64_t *__restrict__ ce,
           const int32_t *__restrict__ cu, const int32_t *__restrict__ cv,
           const int32_t *__restrict__ crank, Hit *__restrict__ hits_all,
           unsigned long long *__restrict__ counters, int32_t *__restrict__ deg_all, int32_t n,
           int weight_f32, int2 *__restrict__ hpos_all, int32_t *__restrict__ rows_all) {
  __shared__ CandRange sr[kClasses];
  __shared__ WinDesc sw;
  __shared__ int s_pred;
  if (threadIdx.x == 0) {
    sw = wins[blockIdx.y];
    s_pred = 0;
  }
  __syncthreads();
  if ((int)threadIdx.x < sw.n_ranges) sr[threadIdx.x] = ranges[sw.range_off + threadIdx.x];
  __syncthreads();
  const int nr = sw.n_ranges;
  const int64_t total = sw.n_candidates;
  const int count_deg = !sw.may_truncate;
  const int query_neg = sw.ws < 0;
  Hit *hits = hits_all + sw.hit_off;
  int32_t *deg = deg_all + (int64_t)blockIdx.y * n;
  int npred = 0;
  const int lane = threadIdx.x & 31;
  // warp-uniform trip count (the list of a sparse window is appended per warp)
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; base < total;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = base + lane;
    bool new_u = false, new_v = false;
    Hit h;
    h.rank = -1;
    h.u = -2;
    h.v = h.w = 0;
    if (t < total) {
      int k = 0;
      for (int step = 32; step > 0; step >>= 1)
        if (k + step < nr && sr[k + step].prefix <= t) k += step;
      const int64_t idx = sr[k].lo + (t - sr[k].prefix);
      const int64_t s = cs[idx], e = ce[idx];
      if (s < sw.qe && sw.qs < e) {
        ++npred;
        // Coordinates handed to the CSR builder: mirrored back when the
        // stored orientation differs from the query's.
        int64_t hs = s, he = e;
        if ((s < 0) != query_neg) {
          hs = -e;
          he = -(int64_t)(int32_t)s;
        }
        const int64_t os = hs > sw.ws ? hs : sw.ws;
        const int64_t oe = he < sw.we ? he : sw.we;
        const int64_t ov = oe - os;
        h.rank = crank[idx];
        h.v = cv[idx];
        h.u = -1;  // in the window without overlap: counts toward the hit cap only
        if (ov > 0) {
          h.u = cu[idx];
          h.w = weight_f32 ? __float_as_int(__fmul_rn(__ll2float_rn(ov), sw.scale)) : (int32_t)ov;
          if (rows_all) {  // sparse window: the first pair of a row lists it
            const int pu = atomicAdd(&deg[h.u], 1), pv = atomicAdd(&deg[h.v], 1);
            hpos_all[sw.hit_off + t] = make_int2(pu, pv);
            new_u = pu == 0;
            new_v = pv == 0;
          } else if (count_deg) {
            atomicAdd(&deg[h.u], 1);
            atomicAdd(&deg[h.v], 1);
          }
        }
      }
      hits[t] = h;
    }
    if (rows_all) {
      const unsigned mu = __ballot_sync(kFull, new_u), mv = __ballot_sync(kFull, new_v);
      if (mu | mv) {
        unsigned long long at = 0;
        if (lane == 0)
          at = atomicAdd(&counters[4 * blockIdx.y + 1],
                         (unsigned long long)(__popc(mu) + __popc(mv)));
        int32_t *rows = rows_all + 2 * sw.hit_off + __shfl_sync(kFull, at, 0);
        const unsigned below = (1u << lane) - 1u;
        if (new_u) rows[__popc(mu & below)] = h.u;
        if (new_v) rows[__popc(mu) + __popc(mv & below)] = h.v;
      }
    }
  }
  npred = __reduce_add_sync(kFull, npred);
  if ((threadIdx.x & 31) == 0 && npred) atomicAdd(&s_pred, npred);
  __syncthreads();
  if (threadIdx.x == 0 && s_pred)
    atomicAdd(&counters[4 * blockIdx.y + 3], (unsigned long long)s_pred);
}

// The reference query stops after max(nlists,1) hits taken in sorted order
// (the NCLS depth-first order), i.e. it keeps the cap smallest ranks.
// Candidates outside the window rank last (-1 is the largest unsigned rank)
// and carry no weight, so they never displace a hit.
__global__ void __launch_bounds__(1024)
    k_trunc(const WinDesc *__restrict__ wins, Hit *__restrict__ hits_all, int64_t cap,
            int32_t *__restrict__ deg_all, int32_t nodes) {
  __shared__ unsigned hist[256];
  __shared__ unsigned s_prefix, s_k;
  if (!wins[blockIdx.y].may_truncate) return;
  Hit *hits = hits_all + wins[blockIdx.y].hit_off;
  int32_t *deg = deg_all + (int64_t)blockIdx.y * nodes;
  const int64_t n = wins[blockIdx.y].n_candidates;
  uint32_t thr = 0xFFFFFFFFu;
  if (n > cap) {
    if (threadIdx.x == 0) {
      s_prefix = 0;
      s_k = (unsigned)cap;  // 1-based rank of the last kept hit
    }
    __syncthreads();
    for (int d = 3; d >= 0; --d) {
      for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0;
      __syncthreads();
      const unsigned pre = s_prefix;
      const unsigned hi_mask = (d == 3) ? 0u : (0xFFFFFFFFu << (8 * (d + 1)));
      for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const unsigned r = (unsigned)hits[i].rank;
        if ((r & hi_mask) == (pre & hi_mask)) atomicAdd(&hist[(r >> (8 * d)) & 255u], 1u);
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned k = s_k, acc = 0;
        int b = 0;
        for (; b < 256; ++b) {
          if (acc + hist[b] >= k) break;
          acc += hist[b];
        }
        s_k = k - acc;
        s_prefix = pre | ((unsigned)b << (8 * d));
      }
      __syncthreads();
    }
    thr = s_prefix;
  }
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    Hit h = hits[i];
    if ((uint32_t)h.rank > thr) {
      hits[i].u = -2;
      continue;
    }
    if (h.u >= 0) {
      atomicAdd(&deg[h.u], 1);
      atomicAdd(&deg[h.v], 1);
    }
  }
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_tiles(const int32_t *__restrict__ in_all, int32_t n, int32_t *__restrict__ tiles) {
  __shared__ int wt[32];
  const int32_t *in = in_all + (int64_t)blockIdx.y * n;
  const int64_t base = (int64_t)blockIdx.x * kScanTile + 4 * threadIdx.x;
  int s = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (base + j < n) s += in[base + j];
  s = block_sum(s, wt);
  if (threadIdx.x == 0) tiles[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
}

// Row pointers from the degrees (one block per tile and window; a window of
// one tile needs no tile sums).
__global__ void __launch_bounds__(kScanThreads)
    k_scan_apply(int32_t *__restrict__ in_all, int32_t n,
                 const int32_t *__restrict__ tiles, int32_t *__restrict__ out_all,
                 int zero_in, int32_t *__restrict__ heavy_all,
                 const int64_t *__restrict__ heavy_off, unsigned long long *__restrict__ heavy_counts) {
  __shared__ int wt[32];
  int32_t *in = in_all + (int64_t)blockIdx.y * n;
  int32_t *out = out_all + (int64_t)blockIdx.y * (n + 1);
  int off = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += blockDim.x)
    off += tiles[(int64_t)blockIdx.y * gridDim.x + b];
  off = block_sum(off, wt);
  const int64_t base = (int64_t)blockIdx.x * kScanTile + 4 * threadIdx.x;
  int v[4], s = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = (base + j < n) ? in[base + j] : 0;
    s += v[j];
  }
  int total;
  int ex = block_excl_scan(s, wt, total) + off;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (base + j < n) {
      out[base + j] = ex;
      if (zero_in) in[base + j] = 0;
      if (heavy_all && v[j] > kHeavyPairs) {  // the step kernel's list of long rows
        // the window's list: at heavy_off (n_windows + 1 offsets), or n rows a slot
        const int64_t lo = heavy_off ? heavy_off[blockIdx.y] : (int64_t)blockIdx.y * n;
        const int64_t hi = heavy_off ? heavy_off[blockIdx.y + 1] : lo + n;
        unsigned long long *cnt = heavy_counts + 4 * blockIdx.y;
        const bool huge = v[j] > kHugePairs;
        const int64_t at = (int64_t)atomicAdd(&cnt[huge ? 2 : 0], 1ull);
        heavy_all[huge ? hi - 1 - at : lo + at] = (int32_t)(base + j);
      }
    }
    ex += v[j];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = off + total;
}

// Sparse window: places the listed rows' pairs in list order (one reduction per
// block), lists the long rows, and leaves every degree zero again.
__global__ void __launch_bounds__(256)
    k_place_rows(const WinDesc *__restrict__ wins, int32_t *__restrict__ deg_all,
                 const int32_t *__restrict__ rows_all, int2 *__restrict__ span_all,
                 int32_t *__restrict__ row_ptr_all, unsigned long long *__restrict__ placed,
                 unsigned long long *__restrict__ counters, int32_t *__restrict__ heavy_all,
                 int32_t n) {
  __shared__ int wt[32];
  __shared__ unsigned long long s_base;
  const int64_t hoff = 2 * wins[blockIdx.y].hit_off;
  const int32_t *rows = rows_all + hoff;
  int2 *span = span_all + hoff;
  int32_t *deg = deg_all + (int64_t)blockIdx.y * n;
  int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (n + 1);
  unsigned long long *cnt = counters + 4 * blockIdx.y;
  const int64_t m = (int64_t)cnt[1];
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < m;
       base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = base + threadIdx.x;
    int32_t row = 0;
    int d = 0;
    if (j < m) {
      row = rows[j];
      // one exchange: a load and a store of the sector that the atomics of
      // k_hits left took 118 us for 7 windows of 146,000 rows, this 30
      d = atomicExch(&deg[row], 0);
    }
    int total;
    const int off = block_excl_scan(d, wt, total);
    if (threadIdx.x == 0) s_base = atomicAdd(&placed[blockIdx.y], (unsigned long long)total);
    __syncthreads();
    if (j < m) {
      const int32_t beg = (int32_t)s_base + off;
      row_ptr[row] = beg;
      span[j] = make_int2(beg, d);
      if (d > kHeavyPairs) {
        int32_t *list = heavy_all + (int64_t)blockIdx.y * n;
        const bool huge = d > kHugePairs;
        const int64_t at = (int64_t)atomicAdd(&cnt[huge ? 2 : 0], 1ull);
        list[huge ? n - 1 - at : at] = (int32_t)j;  // by list entry: the row's end is there
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256)
    k_fill_sparse(const WinDesc *__restrict__ wins, const Hit *__restrict__ hits_all,
                  const int2 *__restrict__ hpos_all, const int32_t *__restrict__ row_ptr_all,
                  int2 *__restrict__ entries_all, int32_t nodes) {
  const int64_t n = wins[blockIdx.y].n_candidates, hoff = wins[blockIdx.y].hit_off;
  const int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (nodes + 1);
  int2 *entries = entries_all + 2 * hoff;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Hit h = hits_all[hoff + i];
    if (h.u < 0) continue;
    const int2 p = hpos_all[hoff + i];
    entries[row_ptr[h.u] + p.x] = make_int2(h.v, h.w);
    entries[row_ptr[h.v] + p.y] = make_int2(h.u, h.w);
  }
}

__global__ void __launch_bounds__(256)
    k_fill(const WinDesc *__restrict__ wins, const Hit *__restrict__ hits_all,
           const int32_t *__restrict__ row_ptr_all, int32_t *__restrict__ cursor_all,
           int2 *__restrict__ entries_all, int32_t *__restrict__ erank_all, int32_t nodes,
           int keep_rank) {
  const int64_t n = wins[blockIdx.y].n_candidates, hoff = wins[blockIdx.y].hit_off;
  const Hit *hits = hits_all + hoff;
  const int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (nodes + 1);
  int32_t *cursor = cursor_all + (int64_t)blockIdx.y * nodes;
  int2 *entries = entries_all + 2 * hoff;
  int32_t *erank = erank_all + 2 * hoff;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Hit h = hits[i];
    if (h.u < 0) continue;
    // the degrees count down to the zeros that the next window starts from
    const int32_t pu = row_ptr[h.u] + atomicSub(&cursor[h.u], 1) - 1;
    entries[pu] = make_int2(h.v, h.w);
    const int32_t pv = row_ptr[h.v] + atomicSub(&cursor[h.v], 1) - 1;
    entries[pv] = make_int2(h.u, h.w);
    if (keep_rank) {
      erank[pu] = h.rank;
      erank[pv] = h.rank;
    }
  }
}

// ---- row sort + merge -----------------------------------------------------------
// The leader of a peer group is its lowest lane.
__device__ __forceinline__ bool before_leader(unsigned peers, unsigned lane) {
  return (unsigned)(__ffs(peers) - 1) == lane;
}

__device__ __forceinline__ uint64_t make_key(int32_t col, int32_t rank) {
  return ((uint64_t)(uint32_t)col << 32) | (uint32_t)rank;
}

__device__ __forceinline__ int32_t merge_add(int32_t acc, int32_t w, int f32) {
  return f32 ? __float_as_int(__fadd_rn(__int_as_float(acc), __int_as_float(w)))
             : acc + w;
}

constexpr int kWarpCap = 512;       // rows up to this length sort in a warp
constexpr int kRowsortWarps = 4;

// Merges runs of equal columns in a sorted segment held in shared memory:
// the first entry of a run receives the sequential sum, the rest weight 0.
__device__ void merge_runs_smem(const uint64_t *key, int32_t *val, int L, int f32,
                                int tid, int nthreads) {
  for (int i = tid; i < L; i += nthreads) {
    const uint32_t c = (uint32_t)(key[i] >> 32);
    const bool head = (i == 0) || ((uint32_t)(key[i - 1] >> 32) != c);
    if (!head) continue;
    int32_t acc = val[i];
    int j = i + 1;
    for (; j < L && (uint32_t)(key[j] >> 32) == c; ++j) acc = merge_add(acc, val[j], f32);
    val[i] = acc;
    for (int q = i + 1; q < j; ++q) val[q] = 0;
  }
}

__global__ void __launch_bounds__(32 * kRowsortWarps)
    k_rowsort_warp(const WinDesc *__restrict__ wins, int32_t n,
                   const int32_t *__restrict__ row_ptr_all, int2 *__restrict__ entries_all,
                   int32_t *__restrict__ erank_all, unsigned long long *__restrict__ counters,
                   int32_t *__restrict__ long_rows, int f32) {
  const int64_t hoff = wins[blockIdx.y].hit_off;
  const int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (n + 1);
  int2 *entries = entries_all + 2 * hoff;
  int32_t *erank = erank_all + 2 * hoff;
  counters += 4 * blockIdx.y;
  long_rows += (int64_t)blockIdx.y * n;
  __shared__ uint64_t skey[kRowsortWarps][kWarpCap];
  __shared__ int32_t sval[kRowsortWarps][kWarpCap];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = gw; row < n; row += nw) {
    const int32_t beg = row_ptr[row], L = row_ptr[row + 1] - beg;
    if (L <= 1) continue;
    if (L > kWarpCap) {
      if (lane == 0) {
        unsigned long long p = atomicAdd(&counters[1], 1ull);
        long_rows[p] = (int32_t)row;
      }
      continue;
    }
    if (L <= 32) {
      uint64_t k = ~0ull;
      int32_t w = 0;
      if (lane < L) {
        const int2 en = entries[beg + lane];
        k = make_key(en.x, erank[beg + lane]);
        w = en.y;
      }
      // bitonic sort of 32 keys across the warp, ascending
#pragma unroll
      for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          const uint64_t ok = __shfl_xor_sync(kFull, k, stride);
          const int32_t ow = __shfl_xor_sync(kFull, w, stride);
          const bool up = ((lane & size) == 0);
          const bool lower = ((lane & stride) == 0);
          const bool take = (lower == up) ? (ok < k) : (ok > k);
          if (take) {
            k = ok;
            w = ow;
          }
        }
      }
      const uint32_t c = (uint32_t)(k >> 32);
      const uint32_t cprev = __shfl_up_sync(kFull, c, 1);
      const bool head = lane < L && (lane == 0 || cprev != c);
      int32_t acc = w;
      bool active = head;
      for (int d = 1; d < 32; ++d) {
        const int32_t ow = __shfl_down_sync(kFull, w, d);
        const uint32_t oc = __shfl_down_sync(kFull, c, d);
        if (active) {
          if (lane + d < L && oc == c)
            acc = merge_add(acc, ow, f32);
          else
            active = false;
        }
        if (!__any_sync(kFull, active)) break;
      }
      if (lane < L) {
        entries[beg + lane] = make_int2((int32_t)c, head ? acc : 0);
        erank[beg + lane] = (int32_t)(uint32_t)k;
      }
      continue;
    }
    // 32 < L <= kWarpCap: bitonic sort in this warp's shared-memory slot
    int P = 64;
    while (P < L) P <<= 1;
    uint64_t *key = skey[wib];
    int32_t *val = sval[wib];
    for (int i = lane; i < P; i += 32) {
      if (i < L) {
        const int2 en = entries[beg + i];
        key[i] = make_key(en.x, erank[beg + i]);
        val[i] = en.y;
      } else {
        key[i] = ~0ull;
        val[i] = 0;
      }
    }
    __syncwarp();
    for (int size = 2; size <= P; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = lane; i < P; i += 32) {
          const int j = i ^ stride;
          if (j > i) {
            const bool up = ((i & size) == 0);
            const uint64_t a = key[i], b = key[j];
            if ((a > b) == up) {
              key[i] = b;
              key[j] = a;
              const int32_t t = val[i];
              val[i] = val[j];
              val[j] = t;
            }
          }
        }
        __syncwarp();
      }
    }
    merge_runs_smem(key, val, L, f32, lane, 32);
    __syncwarp();
    for (int i = lane; i < L; i += 32) {
      entries[beg + i] = make_int2((int32_t)(key[i] >> 32), val[i]);
      erank[beg + i] = (int32_t)(uint32_t)key[i];
    }
    __syncwarp();
  }
}

// Rows longer than a warp slot: one CTA per row, stable LSD radix sort on
// (rank, then col) between the row segment and a scratch segment, then the
// sequential merge.  Only reached by hub rows of FP32-weight windows.
__global__ void __launch_bounds__(256)
    k_rowsort_long(const WinDesc *__restrict__ wins, int32_t n,
                   const int32_t *__restrict__ row_ptr_all, int2 *__restrict__ entries_all,
                   int32_t *__restrict__ erank_all, int2 *__restrict__ tmp_e,
                   int32_t *__restrict__ tmp_r,
                   const unsigned long long *__restrict__ counters,
                   const int32_t *__restrict__ long_rows, int rank_bits,
                   int col_bits, int f32) {
  const int64_t hoff = wins[blockIdx.y].hit_off;
  const int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (n + 1);
  int2 *entries = entries_all + 2 * hoff;
  int32_t *erank = erank_all + 2 * hoff;
  tmp_e += 2 * hoff;
  tmp_r += 2 * hoff;
  counters += 4 * blockIdx.y;
  long_rows += (int64_t)blockIdx.y * n;
  __shared__ unsigned hist[256];
  __shared__ unsigned offs[256];
  const int64_t nl = (int64_t)counters[1];
  for (int64_t li = blockIdx.x; li < nl; li += gridDim.x) {
    const int32_t row = long_rows[li];
    const int32_t beg = row_ptr[row], L = row_ptr[row + 1] - beg;
    int2 *ea = entries + beg, *eb = tmp_e + beg;
    int32_t *ra = erank + beg, *rb = tmp_r + beg;
    int npass = 0;
    for (int field = 0; field < 2; ++field) {
      const int bits = field == 0 ? rank_bits : col_bits;
      for (int sh = 0; sh < bits; sh += 8) {
        for (int b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < L; i += blockDim.x) {
          const uint32_t key = field == 0 ? (uint32_t)ra[i] : (uint32_t)ea[i].x;
          atomicAdd(&hist[(key >> sh) & 255u], 1u);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          unsigned acc = 0;
          for (int b = 0; b < 256; ++b) {
            offs[b] = acc;
            acc += hist[b];
          }
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // stable scatter by one warp, in order
          const unsigned lane = threadIdx.x;
          for (int base = 0; base < L; base += 32) {
            const int i = base + lane;
            const bool ok = i < L;
            uint32_t dig = 0;
            if (ok) {
              const uint32_t key = field == 0 ? (uint32_t)ra[i] : (uint32_t)ea[i].x;
              dig = (key >> sh) & 255u;
            }
            const unsigned act = __ballot_sync(kFull, ok);
            const unsigned peers = __match_any_sync(kFull, ok ? dig : 0xFFFFu) & act;
            if (ok) {
              const unsigned before = __popc(peers & ((1u << lane) - 1u));
              const unsigned pos = offs[dig] + before;
              eb[pos] = ea[i];
              rb[pos] = ra[i];
            }
            __syncwarp();
            if (ok && before_leader(peers, lane)) offs[dig] += __popc(peers);
            __syncwarp();
          }
        }
        __syncthreads();
        int2 *te = ea; ea = eb; eb = te;
        int32_t *tr = ra; ra = rb; rb = tr;
        ++npass;
      }
    }
    if (npass & 1) {  // result lives in the scratch segment: copy back
      for (int i = threadIdx.x; i < L; i += blockDim.x) {
        entries[beg + i] = ea[i];
        erank[beg + i] = ra[i];
      }
      __syncthreads();
    }
    // sequential merge of equal-column runs
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
      const int32_t c = entries[beg + i].x;
      const bool head = (i == 0) || entries[beg + i - 1].x != c;
      if (!head) continue;
      int32_t acc = entries[beg + i].y;
      int j = i + 1;
      for (; j < L && entries[beg + j].x == c; ++j) acc = merge_add(acc, entries[beg + j].y, f32);
      entries[beg + i].y = acc;
      for (int q = i + 1; q < j; ++q) entries[beg + q].y = 0;
    }
    __syncthreads();
  }
}

__global__ void k_count_kept(const WinDesc *__restrict__ wins, int32_t n,
                             const int32_t *__restrict__ row_ptr_all,
                             const int2 *__restrict__ entries_all, int32_t *__restrict__ len_all) {
  const int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (n + 1);
  const int2 *entries = entries_all + 2 * wins[blockIdx.y].hit_off;
  int32_t *len = len_all + (int64_t)blockIdx.y * n;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    int c = 0;
    for (int32_t k = row_ptr[r]; k < row_ptr[r + 1]; ++k) c += entries[k].y != 0;
    len[r] = c;
  }
}

// out_off: where each window's pairs go (null: one window, at out).
__global__ void k_compact(const WinDesc *__restrict__ wins, int32_t n,
                          const int32_t *__restrict__ row_ptr_all,
                          const int2 *__restrict__ entries_all,
                          const int32_t *__restrict__ out_ptr_all,
                          const int64_t *__restrict__ out_off, int2 *__restrict__ out) {
  const int32_t *row_ptr = row_ptr_all + (int64_t)blockIdx.y * (n + 1);
  const int32_t *out_ptr = out_ptr_all + (int64_t)blockIdx.y * (n + 1);
  const int2 *entries = entries_all + 2 * wins[blockIdx.y].hit_off;
  if (out_off) out += out_off[blockIdx.y];
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    int32_t o = out_ptr[r];
    for (int32_t k = row_ptr[r]; k < row_ptr[r + 1]; ++k) {
      const int2 en = entries[k];
      if (en.y != 0) out[o++] = en;
    }
  }
}

int grid_for(int64_t work, int threads, int cap) {
  int64_t b = (work + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (int)b;
}

int bits_for(int64_t maxval) {
  int b = 0;
  while (b < 63 && (int64_t(1) << b) <= maxval) ++b;
  return b < 1 ? 1 : b;
}

}  // namespace

int32_t window_scan_tiles(int32_t n_nodes) {
  const int32_t t = (int32_t)((n_nodes + kScanTile - 1) / kScanTile);
  return t < 1 ? 1 : t;
}

rp_status window_workspace_alloc(WindowWorkspace &w, int32_t n_nodes, int32_t slots,
                                 int64_t cap_hits, bool sort_rows, bool sparse,
                                 const std::vector<WinDesc> &wins,
                                 const std::vector<CandRange> &ranges) {
  w.n_nodes = n_nodes;
  w.sparse = sparse;
  w.cap_hits = cap_hits < 1 ? 1 : cap_hits;
  w.cap_entries = 2 * w.cap_hits;
  w.n_tiles = window_scan_tiles(n_nodes);
  const size_t n = (size_t)n_nodes, g = (size_t)(slots < 1 ? 1 : slots);
  RP_TRY(w.hits.alloc(sizeof(Hit) * w.cap_hits));
  RP_TRY(w.entries.alloc(sizeof(int2) * w.cap_entries));
  if (sort_rows) {
    RP_TRY(w.erank.alloc(sizeof(int32_t) * w.cap_entries));
    RP_TRY(w.tmp_e.alloc(sizeof(int2) * w.cap_entries));
    RP_TRY(w.tmp_r.alloc(sizeof(int32_t) * w.cap_entries));
  }
  RP_TRY(w.long_rows.alloc(sizeof(int32_t) * g * n));
  RP_TRY(w.row_ptr.alloc(sizeof(int32_t) * g * (n + 1)));
  RP_TRY(w.deg.alloc(sizeof(int32_t) * g * n));
  RP_TRY(w.tiles.alloc(sizeof(int32_t) * g * (size_t)w.n_tiles));
  RP_TRY(w.counters.alloc(sizeof(unsigned long long) * 4 * g));
  RP_TRY_CUDA(cudaMemset(w.deg.ptr, 0, w.deg.bytes));  // every build leaves them zero
  if (sparse) {
    RP_TRY(w.hpos.alloc(sizeof(int2) * w.cap_hits));
    RP_TRY(w.rows.alloc(sizeof(int32_t) * w.cap_entries));
    RP_TRY(w.span.alloc(sizeof(int2) * w.cap_entries));
    RP_TRY(w.placed.alloc(sizeof(unsigned long long) * g));
  }
  RP_TRY(w.win.alloc(sizeof(WinDesc) * (wins.empty() ? 1 : wins.size())));
  RP_TRY(w.ranges.alloc(sizeof(CandRange) * (ranges.empty() ? 1 : ranges.size())));
  if (!wins.empty())
    RP_TRY_CUDA(cudaMemcpy(w.win.ptr, wins.data(), sizeof(WinDesc) * wins.size(),
                           cudaMemcpyHostToDevice));
  if (!ranges.empty())
    RP_TRY_CUDA(cudaMemcpy(w.ranges.ptr, ranges.data(),
                           sizeof(CandRange) * ranges.size(), cudaMemcpyHostToDevice));
  return RP_OK;
}

// Consecutive windows whose candidates and per-node arrays fit the budget
// form a group (at most kGroupMax windows).  A window of a small network is a
// chain of six launches of a few microseconds each, most of it launch
// latency: 22 us for N = 1,000, twice what the two step kernels of the window
// take.  A group pays that chain once.  The budget keeps a group's pairs in
// L2 between its build and its last step; the first group is smaller, since
// no step can overlap its build.  Sparse windows touch few of their per-node
// arrays, so their budget is a matter of memory: at 2.6M nodes and 75,000
// contacts a window built alone took 31 us, in groups of eight 7 us.
constexpr int64_t kGroupBytes = 32ll << 20, kFirstGroupBytes = 4ll << 20;
constexpr int64_t kSparseGroupBytes = 256ll << 20;
constexpr int32_t kGroupMax = 256;

void plan_window_groups(std::vector<WinDesc> &wins, int32_t n_nodes, bool single, bool sparse,
                        std::vector<WindowGroup> &groups) {
  groups.clear();
  const int64_t node_bytes = 12ll * n_nodes;  // degrees, row pointers, long rows
  for (int32_t w = 0; w < (int32_t)wins.size();) {
    const int64_t budget = groups.empty() ? kFirstGroupBytes
                                          : (sparse ? kSparseGroupBytes : kGroupBytes);
    WindowGroup g;
    g.first = w;
    do {
      wins[w].hit_off = g.candidates;
      g.candidates += wins[w].n_candidates;
      if (wins[w].n_candidates > g.max_candidates) g.max_candidates = wins[w].n_candidates;
      g.truncate |= wins[w].may_truncate;
      ++g.count;
      ++w;
    } while (!single && w < (int32_t)wins.size() && g.count < kGroupMax &&
             48 * (g.candidates + wins[w].n_candidates) + node_bytes * (g.count + 1) <= budget);
    groups.push_back(g);
  }
}

int enqueue_window_build(const Graph &g, WindowWorkspace &ws, const WindowGroup &grp, int64_t cap,
                         int weight_kind, bool sort_rows, cudaStream_t st) {
  const int32_t n = ws.n_nodes;
  const unsigned G = (unsigned)grp.count;
  int launches = 0;
  unsigned long long *ctr = ws.counters.as<unsigned long long>();
  const WinDesc *wins = ws.win.as<WinDesc>() + grp.first;
  cudaMemsetAsync(ctr, 0, sizeof(unsigned long long) * 4 * G, st);
  if (ws.sparse) cudaMemsetAsync(ws.placed.ptr, 0, sizeof(unsigned long long) * G, st);
  const int f32 = weight_kind == kWeightF32;
  const int blocks = std::max(1, 148 * 16 / (int)G);  // per window
  k_hits<<<dim3(grid_for(grp.max_candidates, 256, blocks), G), 256, 0, st>>>(
      wins, ws.ranges.as<CandRange>(), g.cs.as<int64_t>(), g.ce.as<int64_t>(),
      g.cu.as<int32_t>(), g.cv.as<int32_t>(), g.crank.as<int32_t>(), ws.hits.as<Hit>(), ctr,
      ws.deg.as<int32_t>(), n, f32, ws.sparse ? ws.hpos.as<int2>() : nullptr,
      ws.sparse ? ws.rows.as<int32_t>() : nullptr);
  ++launches;
  if (ws.sparse) {
    // every row pass below would touch n rows: 45 us a window at 2.6M nodes and
    // 75,000 contacts, 15 us this way
    k_place_rows<<<dim3(grid_for(2 * grp.max_candidates, 256, blocks), G), 256, 0, st>>>(
        wins, ws.deg.as<int32_t>(), ws.rows.as<int32_t>(), ws.span.as<int2>(),
        ws.row_ptr.as<int32_t>(), ws.placed.as<unsigned long long>(), ctr,
        ws.long_rows.as<int32_t>(), n);
    k_fill_sparse<<<dim3(grid_for(grp.max_candidates, 256, blocks), G), 256, 0, st>>>(
        wins, ws.hits.as<Hit>(), ws.hpos.as<int2>(), ws.row_ptr.as<int32_t>(),
        ws.entries.as<int2>(), n);
    return launches + 2;
  }
  if (grp.truncate) {
    k_trunc<<<dim3(1, G), 1024, 0, st>>>(wins, ws.hits.as<Hit>(), cap, ws.deg.as<int32_t>(), n);
    ++launches;
  }
  if (ws.n_tiles > 1) {
    k_scan_tiles<<<dim3(ws.n_tiles, G), kScanThreads, 0, st>>>(ws.deg.as<int32_t>(), n,
                                                               ws.tiles.as<int32_t>());
    ++launches;
  }
  k_scan_apply<<<dim3(ws.n_tiles, G), kScanThreads, 0, st>>>(
      ws.deg.as<int32_t>(), n, ws.tiles.as<int32_t>(), ws.row_ptr.as<int32_t>(), 0,
      sort_rows ? nullptr : ws.long_rows.as<int32_t>(), nullptr, ctr);
  k_fill<<<dim3(grid_for(grp.max_candidates, 256, blocks), G), 256, 0, st>>>(
      wins, ws.hits.as<Hit>(), ws.row_ptr.as<int32_t>(), ws.deg.as<int32_t>(),
      ws.entries.as<int2>(), ws.erank.as<int32_t>(), n, sort_rows);
  launches += 2;
  if (sort_rows) {
    k_rowsort_warp<<<dim3(grid_for(n, kRowsortWarps, blocks), G), 32 * kRowsortWarps, 0, st>>>(
        wins, n, ws.row_ptr.as<int32_t>(), ws.entries.as<int2>(), ws.erank.as<int32_t>(), ctr,
        ws.long_rows.as<int32_t>(), f32);
    k_rowsort_long<<<dim3(std::max(1, 148 / (int)G), G), 256, 0, st>>>(
        wins, n, ws.row_ptr.as<int32_t>(), ws.entries.as<int2>(), ws.erank.as<int32_t>(),
        ws.tmp_e.as<int2>(), ws.tmp_r.as<int32_t>(), ctr, ws.long_rows.as<int32_t>(),
        bits_for(g.n_contacts), bits_for(n), f32);
    launches += 2;
  }
  return launches;
}

void enqueue_window_compact(WindowWorkspace &ws, const WindowGroup &grp, int32_t *row_ptr_out,
                            int2 *entries_out, const int64_t *entries_off, cudaStream_t st,
                            int32_t *heavy, const int64_t *heavy_off,
                            unsigned long long *heavy_counts) {
  const int32_t n = ws.n_nodes;
  const unsigned G = (unsigned)grp.count;
  const WinDesc *wins = ws.win.as<WinDesc>() + grp.first;
  int32_t *len = ws.deg.as<int32_t>();
  const dim3 grid(grid_for(n, 256, std::max(1, 148 * 8 / (int)G)), G);
  k_count_kept<<<grid, 256, 0, st>>>(wins, n, ws.row_ptr.as<int32_t>(), ws.entries.as<int2>(), len);
  if (ws.n_tiles > 1)
    k_scan_tiles<<<dim3(ws.n_tiles, G), kScanThreads, 0, st>>>(len, n, ws.tiles.as<int32_t>());
  k_scan_apply<<<dim3(ws.n_tiles, G), kScanThreads, 0, st>>>(
      len, n, ws.tiles.as<int32_t>(), row_ptr_out, 1, heavy, heavy_off, heavy_counts);
  if (entries_out)
    k_compact<<<grid, 256, 0, st>>>(wins, n, ws.row_ptr.as<int32_t>(), ws.entries.as<int2>(),
                                    row_ptr_out, entries_off, entries_out);
}

}  // namespace rp
