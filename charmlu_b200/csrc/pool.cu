// Resources that destroyed handles leave for the next ones (handle.h).
#include <mutex>

#include "handle.h"

namespace lub {
namespace {

constexpr unsigned kIdleDestroys = 32;  // a block unused for so many destroys is freed
constexpr size_t kMaxRes = 8;

struct Block {
  void* p;
  size_t bytes;
  unsigned tick;
};
struct DevPool {
  std::mutex mu;
  std::vector<Block> blocks;
  std::vector<HandleRes> res;
  size_t cached = 0, cap = 0;
  unsigned tick = 0;
};
DevPool& pool_of(int dev) {
  static DevPool* pools = new DevPool[64];  // never destroyed: no CUDA call after the runtime's own exit
  return pools[dev];
}

// a block that cannot be freed now (during a capture, say) stays
void drop(DevPool& d, size_t i) {
  if (cudaFree(d.blocks[i].p) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  d.cached -= d.blocks[i].bytes;
  d.blocks.erase(d.blocks.begin() + i);
}

// cudaMalloc, after giving the cached blocks back if there is no room (lock held)
int malloc_or_empty(DevPool& d, void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    for (size_t i = d.blocks.size(); i-- > 0;) drop(d, i);
    e = cudaMalloc(p, bytes);
  }
  if (e == cudaSuccess) return LU_OK;
  cudaGetLastError();
  *p = nullptr;
  return LU_ERR_NOMEM;
}

void destroy_res(const HandleRes& r) {
  if (r.sP) cudaStreamDestroy(r.sP);
  if (r.sG) cudaStreamDestroy(r.sG);
  for (cudaEvent_t e : r.ev)
    if (e) cudaEventDestroy(e);
  if (r.pinned) cudaFreeHost(r.pinned);
}

int current_device(int* dev) {
  if (cudaGetDevice(dev) != cudaSuccess) {
    cudaGetLastError();
    return LU_ERR_CUDA;
  }
  return *dev >= 0 && *dev < 64 ? LU_OK : LU_ERR_UNSUPPORTED;
}

}  // namespace

int pool_alloc(void** p, size_t bytes, size_t* got) {
  int dev = 0;
  LUB_TRY(current_device(&dev));
  const size_t unit = bytes >= (size_t(1) << 20) ? size_t(1) << 20 : 512;
  const size_t want = std::max<size_t>((bytes + unit - 1) / unit * unit, 512);
  DevPool& d = pool_of(dev);
  std::lock_guard<std::mutex> lk(d.mu);
  // the smallest cached block that is not more than a quarter too large
  size_t best = d.blocks.size();
  for (size_t i = 0; i < d.blocks.size(); i++)
    if (d.blocks[i].bytes >= want && d.blocks[i].bytes <= want + want / 4 &&
        (best == d.blocks.size() || d.blocks[i].bytes < d.blocks[best].bytes))
      best = i;
  if (best < d.blocks.size()) {
    *p = d.blocks[best].p;
    *got = d.blocks[best].bytes;
    d.cached -= *got;
    d.blocks.erase(d.blocks.begin() + best);
    return LU_OK;
  }
  *got = want;
  return malloc_or_empty(d, p, want);
}

int pool_malloc(void** p, size_t bytes) {
  int dev = 0;
  LUB_TRY(current_device(&dev));
  DevPool& d = pool_of(dev);
  std::lock_guard<std::mutex> lk(d.mu);
  return malloc_or_empty(d, p, bytes);
}

void pool_free(int device, void* p, size_t bytes, size_t limit) {
  if (device < 0 || device >= 64) {
    cudaFree(p);
    return;
  }
  DevPool& d = pool_of(device);
  std::lock_guard<std::mutex> lk(d.mu);
  if (!d.cap) {
    size_t fr = 0, total = 0;
    if (cudaMemGetInfo(&fr, &total) == cudaSuccess) d.cap = total / 64;
    else cudaGetLastError();
  }
  if (d.cached + bytes > std::min(limit, d.cap)) {
    cudaFree(p);
    return;
  }
  d.blocks.push_back({p, bytes, d.tick});
  d.cached += bytes;
}

int pool_release() {
  int dev = 0;
  LUB_TRY(current_device(&dev));
  DevPool& d = pool_of(dev);
  std::lock_guard<std::mutex> lk(d.mu);
  for (size_t i = d.blocks.size(); i-- > 0;) drop(d, i);
  for (const HandleRes& r : d.res) destroy_res(r);
  d.res.clear();
  return d.blocks.empty() ? LU_OK : LU_ERR_CUDA;
}

int pool_take_res(HandleRes* r) {
  int dev = 0;
  LUB_TRY(current_device(&dev));
  DevPool& d = pool_of(dev);
  std::lock_guard<std::mutex> lk(d.mu);
  if (!d.res.empty()) {
    *r = d.res.back();
    d.res.pop_back();
    return LU_OK;
  }
  int lo = 0, hi = 0;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  *r = HandleRes();
  bool ok = cudaStreamCreateWithPriority(&r->sP, cudaStreamNonBlocking, hi) == cudaSuccess &&
            cudaStreamCreateWithFlags(&r->sG, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMallocHost(&r->pinned, sizeof(ResidualAccum)) == cudaSuccess;
  for (cudaEvent_t& e : r->ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (ok) return LU_OK;
  cudaGetLastError();
  destroy_res(*r);
  *r = HandleRes();
  return LU_ERR_CUDA;
}

void pool_give_res(int device, const HandleRes& r, size_t limit) {
  if (device < 0 || device >= 64) {
    destroy_res(r);
    return;
  }
  DevPool& d = pool_of(device);
  std::lock_guard<std::mutex> lk(d.mu);
  // once per destroy: blocks that nothing has asked for since long go back
  d.tick++;
  for (size_t i = d.blocks.size(); i-- > 0;)
    if (d.tick - d.blocks[i].tick > kIdleDestroys || d.cached > limit) drop(d, i);
  if (limit > 0 && d.res.size() < kMaxRes) d.res.push_back(r);
  else destroy_res(r);
}

}  // namespace lub
