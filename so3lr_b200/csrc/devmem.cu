// Cached device and pinned host blocks for evaluation contexts.
//
// A context of a thousand atoms holds some ninety arrays; cudaMalloc and cudaFree cost 100-200 us each (cudaFree waits for the
// device, cudaMallocHost pins pages), which made creating and destroying the context of one small batch cost 5-8 ms around 1 ms of
// kernels.  A context takes one block for all its arrays (engine.cu:Pool::plan), and blocks that it gives back are kept and handed to
// the next context of about the same size: creating one of 22 to 1,281 atoms takes 30 us, releasing it 4 us (24,000 atoms, whose
// block is above kMaxBlock: 2.9 and 2.6 ms); six batches of 32 molecules, a context each, 48.6 -> 7.7 ms.
//
// The cache is bounded (kMaxCached bytes per device, blocks above kMaxBlock are never kept), shared by all threads under one
// lock, emptied when an allocation fails, and emptied per device when a model is destroyed.  dev_free keeps the guarantee of cudaFree:
// the device is idle with respect to the block before anybody else can receive it (a context that frees many blocks waits once:
// DevFreeBatch).  Blocks are not cleared.
#include <map>
#include <mutex>
#include <unordered_map>

#include "kernels.h"

namespace so3lr {

namespace {

constexpr size_t kMaxCached = (size_t)256 << 20;
constexpr size_t kMaxBlock = (size_t)96 << 20;
constexpr size_t kMaxCachedHost = (size_t)32 << 20;

struct Cache {
  std::mutex lock;
  std::unordered_map<void*, std::pair<size_t, int>> live;      // block -> (bytes, device; -1 = pinned host)
  std::multimap<std::pair<int, size_t>, void*> idle;           // (device, bytes) -> block
  std::map<int, size_t> idle_bytes;
};
Cache& cache() {
  static Cache* c = new Cache();      // never destroyed: contexts may be released during the process's exit
  return *c;
}
thread_local int tl_batch = 0;
thread_local long long tl_fail_in = 0;      // tests: the allocation of this thread that finds no memory, 0 = none
thread_local bool tl_fail_on = false;       //   ... and all after it

// sizes in steps of an eighth of their power of two (512 bytes at least), so that similar requests share blocks
size_t round_size(size_t b) {
  if (b < 512) return 512;
  size_t p = 512;
  while (p * 2 <= b) p *= 2;
  const size_t step = p / 8 < 512 ? 512 : p / 8;
  return (b + step - 1) / step * step;
}
void* take_idle(Cache& c, int dev, size_t bytes) {
  auto it = c.idle.lower_bound({dev, bytes});
  if (it == c.idle.end() || it->first.first != dev || it->first.second > bytes + bytes / 2) return nullptr;
  void* p = it->second;
  c.idle_bytes[dev] -= it->first.second;
  c.live[p] = {it->first.second, dev};
  c.idle.erase(it);
  return p;
}
void flush_locked(Cache& c, int dev) {
  for (auto it = c.idle.begin(); it != c.idle.end();) {
    if (it->first.first == dev) {
      if (dev < 0) cudaFreeHost(it->second); else cudaFree(it->second);
      it = c.idle.erase(it);
    } else {
      ++it;
    }
  }
  c.idle_bytes[dev] = 0;
}
bool keep_locked(Cache& c, void* p, size_t most_total, size_t most_block) {
  auto it = c.live.find(p);
  if (it == c.live.end()) return false;
  const std::pair<size_t, int> b = it->second;
  c.live.erase(it);
  if (b.first > most_block || c.idle_bytes[b.second] + b.first > most_total) return false;
  c.idle.insert({{b.second, b.first}, p});
  c.idle_bytes[b.second] += b.first;
  return true;
}

}  // namespace

cudaError_t dev_alloc_bytes(void** p, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  *p = nullptr;
  if (tl_fail_in > 0 && (tl_fail_in == 1 || --tl_fail_in == 0)) {
    if (!tl_fail_on) tl_fail_in = 0;
    return cudaErrorMemoryAllocation;
  }
  bytes = round_size(bytes);
  Cache& c = cache();
  std::lock_guard<std::mutex> g(c.lock);
  if ((*p = take_idle(c, dev, bytes))) return cudaSuccess;
  e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    flush_locked(c, dev);
    e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();      // the caller has the status; it may go on without the array
  }
  if (e != cudaSuccess) { *p = nullptr; return e; }
  c.live[*p] = {bytes, dev};
  return cudaSuccess;
}

void dev_free(void* p) {
  if (!p) return;
  if (!tl_batch) cudaDeviceSynchronize();
  Cache& c = cache();
  std::lock_guard<std::mutex> g(c.lock);
  if (!keep_locked(c, p, kMaxCached, kMaxBlock)) cudaFree(p);
}

cudaError_t host_alloc_bytes(void** p, size_t bytes) {
  bytes = round_size(bytes);
  Cache& c = cache();
  std::lock_guard<std::mutex> g(c.lock);
  if ((*p = take_idle(c, -1, bytes))) return cudaSuccess;
  const cudaError_t e = cudaHostAlloc(p, bytes, cudaHostAllocPortable);      // usable from whichever device takes it next
  if (e != cudaSuccess) { *p = nullptr; return e; }
  c.live[*p] = {bytes, -1};
  return cudaSuccess;
}

void host_free(void* p) {
  if (!p) return;
  if (!tl_batch) cudaDeviceSynchronize();      // a copy into or out of the block may be in flight
  Cache& c = cache();
  std::lock_guard<std::mutex> g(c.lock);
  if (!keep_locked(c, p, kMaxCachedHost, kMaxCachedHost)) cudaFreeHost(p);
}

DevFreeBatch::DevFreeBatch() {
  cudaDeviceSynchronize();
  ++tl_batch;
}
DevFreeBatch::~DevFreeBatch() { --tl_batch; }

long long devmem_fail(long long nth, bool on) {
  const long long left = tl_fail_in;
  tl_fail_in = nth; tl_fail_on = on;
  return left;
}

void devmem_flush(int device) {
  Cache& c = cache();
  std::lock_guard<std::mutex> g(c.lock);
  flush_locked(c, device);
  flush_locked(c, -1);
}

}  // namespace so3lr
