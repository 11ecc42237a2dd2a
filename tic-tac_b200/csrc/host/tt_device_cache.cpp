// Cache of large device blocks and pool of small ones behind DevBuf (see tt_device.h).
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "../cuda/tt_device.h"

namespace tt {
namespace {

// never destroyed: buffers with static storage duration release into the
// cache during exit
std::mutex& cache_mu() {
  static std::mutex* m = new std::mutex;
  return *m;
}
std::map<int, std::vector<std::pair<void*, size_t>>>& cache() {  // device -> (block, bytes)
  static auto* c = new std::map<int, std::vector<std::pair<void*, size_t>>>;
  return *c;
}

int current_device() {
  int d = 0;
  cudaGetDevice(&d);
  return d;
}

// one pool per device, never destroyed (as the cache); null: not available
cudaMemPool_t pool_of(int dev) {
  static std::mutex* mu = new std::mutex;
  static auto* pools = new std::map<int, cudaMemPool_t>;
  std::lock_guard<std::mutex> lk(*mu);
  const auto it = pools->find(dev);
  if (it != pools->end()) return it->second;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    pool = nullptr;
  } else {
    unsigned long long keep = kPoolKeepBytes;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  pools->emplace(dev, pool);
  return pool;
}

thread_local cudaStream_t g_scope = nullptr;

}  // namespace

StreamScope::StreamScope(cudaStream_t st) : prev_(g_scope), errors_(error_count()) { g_scope = st; }
StreamScope::~StreamScope() {
  if (g_scope && error_count() != errors_ && cudaStreamSynchronize(g_scope) != cudaSuccess) cudaGetLastError();
  g_scope = prev_;
}

cudaError_t device_pool_alloc(void** p, size_t bytes, bool* pooled) {
  *pooled = false;
  const cudaMemPool_t pool = g_scope ? pool_of(current_device()) : nullptr;
  if (!pool) return cudaMalloc(p, bytes);
  const cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, g_scope);
  *pooled = e == cudaSuccess;
  return e;
}

void device_pool_free(void* p) {
  if (g_scope && cudaFreeAsync(p, g_scope) == cudaSuccess) return;
  cudaGetLastError();
  cudaFree(p);
}

void device_pool_trim(size_t keep) {
  const cudaMemPool_t pool = pool_of(current_device());
  if (!pool) return;
  // frees queued on a stream count once the stream has reached them
  if (g_scope) cudaStreamSynchronize(g_scope);
  cudaMemPoolTrimTo(pool, keep);
}

size_t device_pool_idle_bytes() {
  const cudaMemPool_t pool = pool_of(current_device());
  unsigned long long reserved = 0, used = 0;
  if (!pool || cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
    return 0;
  return reserved > used ? reserved - used : 0;
}

void* device_cache_take(size_t bytes, size_t* capacity) {
  std::lock_guard<std::mutex> lk(cache_mu());
  auto& v = cache()[current_device()];
  int best = -1;
  for (int i = 0; i < (int)v.size(); i++) {
    const size_t c = v[i].second;
    if (c >= bytes && 2 * c <= 3 * bytes && (best < 0 || c < v[best].second)) best = i;
  }
  if (best < 0) return nullptr;
  void* p = v[best].first;
  *capacity = v[best].second;
  v.erase(v.begin() + best);
  return p;
}

void device_cache_give(void* p, size_t capacity) {
  // the block may still be in use by queued work: wait, as cudaFree would
  cudaDeviceSynchronize();
  std::lock_guard<std::mutex> lk(cache_mu());
  cache()[current_device()].emplace_back(p, capacity);
}

size_t device_cache_bytes() {
  std::lock_guard<std::mutex> lk(cache_mu());
  size_t s = 0;
  for (const auto& b : cache()[current_device()]) s += b.second;
  return s;
}

size_t device_cache_evict_one() {
  std::pair<void*, size_t> b{nullptr, 0};
  {
    std::lock_guard<std::mutex> lk(cache_mu());
    auto& v = cache()[current_device()];
    if (v.empty()) return 0;
    b = v.front();  // the block released longest ago
    v.erase(v.begin());
  }
  cudaFree(b.first);
  return b.second;
}

void device_cache_trim() {
  std::vector<std::pair<void*, size_t>> v;
  {
    std::lock_guard<std::mutex> lk(cache_mu());
    v.swap(cache()[current_device()]);
  }
  for (const auto& b : v) cudaFree(b.first);
}

}  // namespace tt
