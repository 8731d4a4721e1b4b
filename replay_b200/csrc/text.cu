// Node-state CSV text formatted on the device.
//
// The reference writes one line per (replica, node) and recorded step,
// "time,simulation_id,node_id,state\n" with state in {susceptible,
// incubating, infectious, resistant}, replicas outer and nodes inner
// (write_simulation_state, tool/gpu_cpu_temporal_sim.cu:505-568).  Here a
// chunk of replica rows [r0, r1) of one step is formatted by segments of
// kTextThreads lines, a block each:
//   k_text_rows   byte length of each segment;
//   k_text_scan   exclusive scan of the lengths (one block);
//   k_text_write  a line per thread, formatted in shared memory, from where
//                 the block stores its segment in whole 16-byte pieces.
// The device's part is bound by its stores of single characters: a thread
// that wrote its lines to global memory character by character, with the 64-bit
// divisions of every number, took 36 us for 64 x 1,000 lines (1.8 MB), this
// form 6.5 us.  The rest of a step's time is the copy to the host and the
// caller's callback.
#include "rp_internal.h"

namespace rp {
namespace {

constexpr int kTextThreads = 256;

__device__ __constant__ char kNames[4][12] = {"susceptible", "incubating", "infectious",
                                              "resistant"};
__device__ __constant__ int kNameLen[4] = {11, 10, 10, 9};

__device__ __forceinline__ int digits_u64(unsigned long long x) {
  int d = 1;
  while (x >= 10ull) {
    x /= 10ull;
    ++d;
  }
  return d;
}

__device__ __forceinline__ int len_i64(long long x) {
  return x < 0 ? 1 + digits_u64(0ull - (unsigned long long)x) : digits_u64((unsigned long long)x);
}

// Writes x in decimal at p; returns the end.
__device__ __forceinline__ char *put_i64(char *p, long long x) {
  unsigned long long u = (unsigned long long)x;
  if (x < 0) {
    *p++ = '-';
    u = 0ull - u;
  }
  char tmp[20];
  int n = 0;
  do {
    tmp[n++] = (char)('0' + (int)(u % 10ull));
    u /= 10ull;
  } while (u);
  while (n) *p++ = tmp[--n];
  return p;
}

template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T *sh, T &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < (int)(blockDim.x >> 5) ? sh[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += y;
    }
    sh[lane] = w;
  }
  __syncthreads();
  const T off = warp ? sh[warp - 1] : T(0);
  total = sh[(blockDim.x >> 5) - 1];
  __syncthreads();
  return off + x - v;
}

__device__ __forceinline__ int digits_u32(uint32_t x) {
  return 1 + (x >= 10u) + (x >= 100u) + (x >= 1000u) + (x >= 10000u) + (x >= 100000u) +
         (x >= 1000000u) + (x >= 10000000u) + (x >= 100000000u) + (x >= 1000000000u);
}

// Byte length of each segment of the chunk.
__global__ void __launch_bounds__(kTextThreads)
    k_text_rows(const uint8_t *__restrict__ cls, int32_t n, int32_t segs, int32_t r0, long long ts,
                long long *__restrict__ seglen) {
  __shared__ int sh[32];
  const int32_t r = r0 + blockIdx.x / segs;
  const int32_t i = (blockIdx.x % segs) * kTextThreads + threadIdx.x;
  int len = 0;
  if (i < n)
    len = len_i64(ts) + digits_u32((uint32_t)r) + 4 + digits_u32((uint32_t)i) +
          kNameLen[cls[(int64_t)r * n + i] & 3];
  int total;
  block_excl_scan(len, sh, total);
  if (threadIdx.x == 0) seglen[blockIdx.x] = total;
}

// Exclusive scan of the chunk's segment lengths (one block); total at [rows].
__global__ void __launch_bounds__(1024)
    k_text_scan(const long long *__restrict__ rowlen, int32_t rows, long long *__restrict__ rowoff) {
  __shared__ long long sh[32];
  const int32_t per = (rows + blockDim.x - 1) / blockDim.x;
  const int32_t b = threadIdx.x * per, e = min(rows, b + per);
  long long s = 0;
  for (int32_t k = b; k < e; ++k) s += rowlen[k];
  long long total;
  long long run = block_excl_scan(s, sh, total);
  for (int32_t k = b; k < e; ++k) {
    rowoff[k] = run;
    run += rowlen[k];
  }
  if (threadIdx.x == 0) rowoff[rows] = total;
}

constexpr int kLineBound = 57;    // 20 + 11 + 11 + 11 characters and 4 separators
constexpr int kPrefixBound = 33;  // "time,simulation_id,"

__global__ void __launch_bounds__(kTextThreads)
    k_text_write(const uint8_t *__restrict__ cls, int32_t n, int32_t segs, int32_t r0, long long ts,
                 const long long *__restrict__ segoff, char *__restrict__ out) {
  __shared__ int sh[32];
  __shared__ char s_prefix[kPrefixBound];
  __shared__ int s_plen;
  __shared__ __align__(16) char s_text[kTextThreads * kLineBound + 16];
  const int32_t r = r0 + blockIdx.x / segs;
  const int32_t i = (blockIdx.x % segs) * kTextThreads + threadIdx.x;
  if (threadIdx.x == 0) {
    char *p = put_i64(s_prefix, ts);
    *p++ = ',';
    p = put_i64(p, r);
    *p++ = ',';
    s_plen = (int)(p - s_prefix);
  }
  __syncthreads();
  const int plen = s_plen;
  int nd = 0, c = 0, len = 0;
  if (i < n) {
    c = cls[(int64_t)r * n + i] & 3;
    nd = digits_u32((uint32_t)i);
    len = plen + nd + 2 + kNameLen[c];
  }
  int total;
  const int off = block_excl_scan(len, sh, total);
  // the segment lies in shared memory as it will in out, relative to 16 bytes
  char *dst = out + segoff[blockIdx.x];
  const int lead = (int)(reinterpret_cast<uintptr_t>(dst) & 15u);
  if (i < n) {
    char *p = s_text + lead + off;
    for (int k = 0; k < plen; ++k) p[k] = s_prefix[k];
    p += plen;
    uint32_t x = (uint32_t)i;
    for (int k = nd - 1; k >= 0; --k) {
      p[k] = (char)('0' + x % 10u);
      x /= 10u;
    }
    p += nd;
    *p++ = ',';
    for (int k = 0; k < kNameLen[c]; ++k) *p++ = kNames[c][k];
    *p = '\n';
  }
  __syncthreads();
  // whole 16-byte pieces; the first and the last may be shared with a neighbour
  const int end = lead + total;
  char *base = dst - lead;
  for (int k = threadIdx.x; 16 * k < end; k += kTextThreads) {
    if (16 * k >= lead && 16 * k + 16 <= end)
      *reinterpret_cast<uint4 *>(base + 16 * k) = *reinterpret_cast<const uint4 *>(s_text + 16 * k);
    else
      for (int j = max(16 * k, lead); j < min(16 * k + 16, end); ++j) base[j] = s_text[j];
  }
}

}  // namespace

int64_t text_line_bound(int32_t n_nodes) {
  (void)n_nodes;
  return kLineBound;
}

int64_t text_segments(int32_t n_nodes) { return (n_nodes + kTextThreads - 1) / kTextThreads; }

void enqueue_states_text(const uint8_t *cls, int32_t n, int32_t r0, int32_t r1, int64_t ts,
                         int64_t *seglen, int64_t *segoff, char *out, cudaStream_t st) {
  const int32_t segs = (int32_t)text_segments(n), blocks = (r1 - r0) * segs;
  if (blocks <= 0) return;
  k_text_rows<<<blocks, kTextThreads, 0, st>>>(cls, n, segs, r0, (long long)ts,
                                               reinterpret_cast<long long *>(seglen));
  k_text_scan<<<1, 1024, 0, st>>>(reinterpret_cast<const long long *>(seglen), blocks,
                                  reinterpret_cast<long long *>(segoff));
  k_text_write<<<blocks, kTextThreads, 0, st>>>(cls, n, segs, r0, (long long)ts,
                                                reinterpret_cast<const long long *>(segoff), out);
}

}  // namespace rp
