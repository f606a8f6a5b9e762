// Cache of freed device blocks behind DevBuf.
//
// The entry points size their scratch by the call (orbital count, memory left)
// and release it on return.  cudaMalloc and cudaFree took 1 to 8 ms each where
// they map or unmap memory (measured on a B200, 1 MB to 1 GB), which was 5 ms of
// an 18 ms gradient and half of a geometry step.  Freed blocks are kept here and
// handed out again:
//   * dev_free waits for the device first, as cudaFree does, so a block in the
//     cache has no work pending on any stream and any stream may reuse it;
//   * the cache is bounded (POOL_BYTES per device, oldest blocks returned to the
//     driver first; larger blocks are never kept), is emptied when an allocation
//     fails, and can be emptied by jk_release_cached;
//   * one mutex guards the lists, so engines may live on several threads; no call
//     that may wait for the device is made under it.
#include <cuda_runtime.h>

#include <iterator>
#include <list>
#include <mutex>
#include <unordered_map>

#include "engine.h"

namespace m2 {
namespace {

constexpr size_t POOL_BYTES = size_t(4) << 30;

struct Block {
  void* p;
  size_t bytes;
  int device;
};
struct Pool {
  std::mutex mu;
  std::mutex full;         // held while the cache is emptied for an allocation that failed
  std::list<Block> cache;  // oldest first
  std::unordered_map<void*, Block> in_use;
};
// never destroyed: engines may outlive the library's static objects at exit
Pool& pool() {
  static Pool* p = new Pool;
  return *p;
}

// Sizes are rounded to an eighth of their power of two (at least 512 bytes), so
// that nearly equal requests share blocks, but to no more than the 2 MB pages that
// cudaMalloc takes by itself: the callers that size their scratch by the free
// memory (0.94 of it for one array) get what they ask for.
size_t round_size(size_t n) {
  size_t step = 512;
  while (step * 16 < n && step < (size_t(2) << 20)) step *= 2;
  return (n + step - 1) / step * step;
}
size_t cached_bytes(int device) {
  size_t b = 0;
  for (const Block& k : pool().cache)
    if (k.device == device) b += k.bytes;
  return b;
}
// Takes the oldest cached blocks of the device out of the list until at most
// `keep` bytes stay; the caller returns them to the driver without the lock.
std::list<Block> take(int device, size_t keep) {
  std::list<Block>& cache = pool().cache;
  std::list<Block> out;
  size_t have = cached_bytes(device);
  for (auto it = cache.begin(); it != cache.end() && have > keep;) {
    const auto b = it++;
    if (b->device != device) continue;
    have -= b->bytes;
    out.splice(out.end(), cache, b);
  }
  return out;
}
void give_back(const std::list<Block>& blocks) {
  for (const Block& b : blocks) cudaFree(b.p);
}

}  // namespace

cudaError_t dev_alloc(void** p, size_t bytes) {
  int device = 0;
  cudaError_t st = cudaGetDevice(&device);
  if (st != cudaSuccess) return st;
  const size_t n = round_size(bytes);
  Pool& P = pool();
  std::unique_lock<std::mutex> lock(P.mu);
  for (auto it = P.cache.rbegin(); it != P.cache.rend(); ++it)
    if (it->device == device && it->bytes == n) {
      *p = it->p;
      P.in_use[it->p] = *it;
      P.cache.erase(std::next(it).base());
      return cudaSuccess;
    }
  lock.unlock();
  st = cudaMalloc(p, n);
  if (st == cudaErrorMemoryAllocation) {
    std::lock_guard<std::mutex> one(P.full);
    lock.lock();
    const std::list<Block> old = take(device, 0);
    lock.unlock();
    give_back(old);
    cudaGetLastError();  // or a later query finds the failure
    st = cudaMalloc(p, n);
  }
  if (st != cudaSuccess) {
    cudaGetLastError();
    return st;
  }
  lock.lock();
  P.in_use[*p] = Block{*p, n, device};
  return st;
}

void dev_free(void* p) {
  if (!p) return;
  Pool& P = pool();
  std::unique_lock<std::mutex> lock(P.mu);
  auto it = P.in_use.find(p);
  if (it == P.in_use.end()) {
    lock.unlock();
    cudaFree(p);
    return;
  }
  const Block b = it->second;
  P.in_use.erase(it);
  lock.unlock();  // other threads allocate while this one waits for the device
  int device = -1;
  const bool here = cudaGetDevice(&device) == cudaSuccess && device == b.device;
  if (!here || b.bytes > POOL_BYTES / 2 || cudaDeviceSynchronize() != cudaSuccess) {
    cudaFree(p);
    return;
  }
  lock.lock();
  const std::list<Block> old = take(device, POOL_BYTES - b.bytes);
  P.cache.push_back(b);
  lock.unlock();
  give_back(old);
}

cudaError_t dev_mem_info(size_t* free_bytes, size_t* total) {
  cudaError_t st = cudaMemGetInfo(free_bytes, total);
  int device = 0;
  if (st == cudaSuccess) st = cudaGetDevice(&device);
  if (st != cudaSuccess) return st;
  std::lock_guard<std::mutex> lock(pool().mu);
  *free_bytes += cached_bytes(device);
  return cudaSuccess;
}

}  // namespace m2

extern "C" int jk_release_cached(int device) {
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) return JK_ERR_CUDA;
  if (cur != device && cudaSetDevice(device) != cudaSuccess) return JK_ERR_ARG;
  std::list<m2::Block> old;
  {
    std::lock_guard<std::mutex> lock(m2::pool().mu);
    old = m2::take(device, 0);
  }
  m2::give_back(old);
  if (cur != device) cudaSetDevice(cur);
  return JK_OK;
}
