// Large copies between pageable host memory and the device.
//
// The runtime stages a pageable copy through one thread: 480 MB of contacts
// take 44 ms up and 252 MB of counts into fresh pages 54 ms down, where the
// link takes 9 and 5.  Here several host threads each move 2 MB chunks through
// a pinned buffer of their own, and the pages of a result are touched while the
// device still computes it.  The pinned buffers are kept for the next copy (at
// most kSlotsMax of them, shared by all threads of the process, returned by
// rp_release_cached_memory); a copy that finds none free takes the plain path,
// as do copies below kPlainBytes and pinned host memory.
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "rp_internal.h"

namespace rp {
namespace {

constexpr size_t kChunk = size_t(2) << 20;
constexpr size_t kPlainBytes = size_t(4) << 20;
constexpr int kSlotsMax = 32, kThreadsMax = 16;

std::mutex g_slots_mu;
std::vector<void *> g_slots;  // free pinned buffers of kChunk bytes
int g_slots_live = 0;         // free or in use

std::vector<void *> take_slots(int want) {
  std::vector<void *> got;
  got.reserve((size_t)want);
  std::lock_guard<std::mutex> lk(g_slots_mu);
  while ((int)got.size() < want) {
    if (!g_slots.empty()) {
      got.push_back(g_slots.back());
      g_slots.pop_back();
      continue;
    }
    void *p = nullptr;
    if (g_slots_live >= kSlotsMax || cudaHostAlloc(&p, kChunk, cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      break;
    }
    ++g_slots_live;
    got.push_back(p);
  }
  return got;
}

void give_slots(const std::vector<void *> &s) {
  std::lock_guard<std::mutex> lk(g_slots_mu);
  g_slots.insert(g_slots.end(), s.begin(), s.end());
}

bool pinned(const void *p) {
  cudaPointerAttributes a{};
  const bool ok = cudaPointerGetAttributes(&a, p) == cudaSuccess;
  (void)cudaGetLastError();
  return ok && a.type != cudaMemoryTypeUnregistered;
}

int threads_for(size_t bytes) {
  const size_t hw = std::max(1u, std::thread::hardware_concurrency());
  return (int)std::min<size_t>({hw, (size_t)kThreadsMax, bytes / (2 * kChunk) + 1});
}

// Runs work(0) .. work(n - 1), one thread each (this thread takes the first,
// and any that no thread could be created for).
template <typename F>
void run_threads(int n, F work) {
  std::vector<std::thread> pool;
  int made = 1;
  try {
    pool.reserve((size_t)n);
    for (; made < n; ++made) pool.emplace_back(work, made);
  } catch (...) {
  }
  work(0);
  for (int k = made; k < n; ++k) work(k);
  for (std::thread &t : pool) t.join();
}

struct Chunk {
  char *dev, *host;
  size_t bytes;
};

rp_status staged(int device, const std::vector<Chunk> &chunks, size_t total, bool up) {
  const std::vector<void *> slots = take_slots(threads_for(total));
  if (slots.empty()) {
    for (const Chunk &c : chunks)
      RP_TRY_CUDA(up ? cudaMemcpy(c.dev, c.host, c.bytes, cudaMemcpyHostToDevice)
                     : cudaMemcpy(c.host, c.dev, c.bytes, cudaMemcpyDeviceToHost));
    return RP_OK;
  }
  std::atomic<size_t> next{0};
  std::atomic<int> err{cudaSuccess};
  run_threads((int)slots.size(), [&](int k) {
    void *slot = slots[(size_t)k];
    cudaStream_t st = nullptr;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    for (size_t i; e == cudaSuccess && err.load() == cudaSuccess && (i = next++) < chunks.size();) {
      const Chunk &c = chunks[i];
      if (up) {
        memcpy(slot, c.host, c.bytes);
        e = cudaMemcpyAsync(c.dev, slot, c.bytes, cudaMemcpyHostToDevice, st);
      } else {
        e = cudaMemcpyAsync(slot, c.dev, c.bytes, cudaMemcpyDeviceToHost, st);
      }
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e == cudaSuccess && !up) memcpy(c.host, slot, c.bytes);
    }
    if (st) cudaStreamDestroy(st);
    if (e != cudaSuccess) err.store((int)e);
  });
  give_slots(slots);
  if (err.load() != cudaSuccess)
    return cuda_fail((cudaError_t)err.load(), up ? "staged upload" : "staged download");
  return RP_OK;
}

}  // namespace

// Copies the parts to the device; returns when the copies are done.  The
// destinations must be idle.
rp_status upload(int device, const HostPart *parts, int n) {
  std::vector<Chunk> chunks;
  size_t total = 0;
  for (int k = 0; k < n; ++k) {
    char *dev = static_cast<char *>(parts[k].dev), *host = const_cast<char *>(static_cast<const char *>(parts[k].host));
    if (parts[k].bytes < kPlainBytes || pinned(host)) {
      RP_TRY_CUDA(cudaMemcpy(dev, host, parts[k].bytes, cudaMemcpyHostToDevice));
      continue;
    }
    for (size_t o = 0; o < parts[k].bytes; o += kChunk)
      chunks.push_back(Chunk{dev + o, host + o, std::min(kChunk, parts[k].bytes - o)});
    total += parts[k].bytes;
  }
  return chunks.empty() ? RP_OK : staged(device, chunks, total, true);
}

// Copies n bytes of finished device results to the host.
rp_status download(int device, void *host, const void *dev, size_t n) {
  if (n < kPlainBytes || pinned(host)) {
    RP_TRY_CUDA(cudaMemcpy(host, dev, n, cudaMemcpyDeviceToHost));
    return RP_OK;
  }
  std::vector<Chunk> chunks;
  char *d = const_cast<char *>(static_cast<const char *>(dev)), *h = static_cast<char *>(host);
  for (size_t o = 0; o < n; o += kChunk) chunks.push_back(Chunk{d + o, h + o, std::min(kChunk, n - o)});
  return staged(device, chunks, n, false);
}

// Brings the pages of a result buffer in, without changing its contents
// (call while the device computes the result).
void touch_pages(void *host, size_t n) {
  if (n < kPlainBytes || pinned(host)) return;
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  const int nt = threads_for(n);
  char *p = static_cast<char *>(host);
  run_threads(nt, [&](int k) {
    const size_t lo = n * (size_t)k / (size_t)nt, hi = n * ((size_t)k + 1) / (size_t)nt;
    for (size_t o = lo; o < hi; o += page) {
      volatile char *q = p + o;
      *q = *q;
    }
  });
}

void release_slots() {
  std::lock_guard<std::mutex> lk(g_slots_mu);
  for (void *p : g_slots) cudaFreeHost(p);
  g_slots_live -= (int)g_slots.size();
  g_slots.clear();
}

}  // namespace rp
