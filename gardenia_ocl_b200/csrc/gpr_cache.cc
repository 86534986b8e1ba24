// Device allocations: the block cache behind dmalloc / dfree and its C-ABI entry points.
#include <mutex>
#include <unordered_map>
#include <vector>

#include "gpr_internal.cuh"

namespace gpr {

// Block cache of device allocations.  One-shot solver calls (the reference's
// PRSolver shape: copy in, build, solve, free) make dozens of allocations each, of
// a few bytes to gigabytes: mapping and unmapping the large ones makes cudaMalloc
// / cudaFree slow and erratic, and every cudaFree of a small one waits for the
// device.  Blocks are kept after dfree and handed out again: large ones (kCacheMin
// bytes and more) to requests that fit them within 1/8, at most kCacheCap bytes of
// them; small ones by size class (powers of two from kSmallMin), at most kSmallCap
// bytes.  A freed block may still be in use by a kernel, so it is handed out again
// only behind a device synchronisation: one when the first block freed since the
// last one is taken, for all of them.  Where that is refused, a new block is
// allocated.  An allocation that fails releases the
// cache and retries; gpr_release_cached() empties it.
// One-shot PageRank of 65,536 vertices on host arrays: 2.76 ms with the small blocks
// allocated and freed each time and a synchronisation per free, 1.20 ms this way.
namespace {

constexpr size_t kCacheMin = size_t(1) << 20;
constexpr size_t kCacheCap = size_t(24) << 30;
constexpr size_t kSmallMin = 512;
constexpr size_t kSmallCap = size_t(64) << 20;
constexpr int kSmallClasses = 11;  // 512 bytes .. 512 KiB

struct Block {
  void *p;
  size_t bytes;
  int device;
  unsigned long long freed;  // number of the free (g_frees) that returned it
};

std::mutex g_mu;
std::unordered_map<void *, Block> g_live;  // blocks handed out
std::vector<Block> g_free;                // cached large blocks, unused
std::vector<Block> g_small[kSmallClasses];  // cached small blocks, by class
size_t g_free_bytes = 0, g_small_bytes = 0;
unsigned long long g_frees = 0;
std::unordered_map<int, unsigned long long> g_synced;  // per device: frees it has waited for

int small_class(size_t bytes) {
  int c = 0;
  while ((kSmallMin << c) < bytes) ++c;
  return c;
}

void give_back(const Block &b) {
  int cur = -1;
  cudaGetDevice(&cur);
  if (cur != b.device) cudaSetDevice(b.device);
  cudaFree(b.p);
  if (cur >= 0 && cur != b.device) cudaSetDevice(cur);
}

// Waits for the device of a block that is handed out (others are left to cudaFree).
cudaError_t wait_for_owner(void *p) {
  int device = -1, cur = -1;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_live.find(p);
    if (it == g_live.end()) return cudaSuccess;
    device = it->second.device;
  }
  cudaGetDevice(&cur);
  if (cur != device) cudaSetDevice(device);
  const cudaError_t e = cudaDeviceSynchronize();
  if (cur >= 0 && cur != device) cudaSetDevice(cur);
  return e;
}

// Takes the cached blocks of a device (-1: of all) out of the cache.
std::vector<Block> drain_locked(int device) {
  std::vector<Block> out;
  auto drop = [&](std::vector<Block> &v, size_t &total) {
    for (size_t i = 0; i < v.size();) {
      if (device < 0 || v[i].device == device) {
        out.push_back(v[i]);
        total -= v[i].bytes;
        v[i] = v.back();
        v.pop_back();
      } else {
        ++i;
      }
    }
  };
  drop(g_free, g_free_bytes);
  for (auto &v : g_small) drop(v, g_small_bytes);
  return out;
}

// Cached block for a request on device `dev`, out of its list: the smallest large block
// that holds `bytes` within 1/8 (of equal ones the first in the list, whose free a wait
// rather covers), or the last small block of its class.
bool find_locked(size_t bytes, int dev, Block *out) {
  const bool large = bytes >= kCacheMin;
  std::vector<Block> &v = large ? g_free : g_small[small_class(bytes)];
  int best = -1;
  for (size_t i = 0; i < v.size(); ++i) {
    const Block &b = v[i];
    if (b.device != dev || (large && (b.bytes < bytes || b.bytes - bytes > bytes / 8))) continue;
    if (best < 0 || !large || b.bytes < v[best].bytes) best = (int)i;
  }
  if (best < 0) return false;
  *out = v[best];
  v[best] = v.back();
  v.pop_back();
  (large ? g_free_bytes : g_small_bytes) -= out->bytes;
  return true;
}

void put_locked(const Block &b) {
  if (b.bytes >= kCacheMin) {
    g_free.push_back(b);
    g_free_bytes += b.bytes;
  } else {
    g_small[small_class(b.bytes)].push_back(b);
    g_small_bytes += b.bytes;
  }
}

// A cached block for the current device `dev`, or null.  The wait for the device is
// made without the lock, so that other threads allocate and free meanwhile; it covers
// the blocks freed before it.  Where it is refused (another thread captures a stream)
// the block goes back.
void *take(size_t bytes, int dev) {
  std::unique_lock<std::mutex> lk(g_mu);
  Block b;
  if (!find_locked(bytes, dev, &b)) return nullptr;
  if (b.freed > g_synced[dev]) {
    const unsigned long long upto = g_frees;
    lk.unlock();
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) cudaGetLastError();
    lk.lock();
    if (e != cudaSuccess) {
      put_locked(b);
      return nullptr;
    }
    if (g_synced[dev] < upto) g_synced[dev] = upto;
  }
  g_live[b.p] = b;
  return b.p;
}

}  // namespace

int dmalloc(void **p, size_t bytes, const char *what) {
  *p = nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  if (bytes > (kSmallMin << (kSmallClasses - 1)) && bytes < kCacheMin) bytes = kCacheMin;
  if (bytes < kCacheMin) bytes = kSmallMin << small_class(bytes);
  *p = take(bytes, dev);
  if (*p) return GPR_OK;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    std::vector<Block> kept;
    {
      std::lock_guard<std::mutex> lk(g_mu);
      kept = drain_locked(dev);
    }
    for (const Block &b : kept) give_back(b);
    e = cudaMalloc(p, bytes);
  }
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    *p = nullptr;
    set_error("cudaMalloc(%zu bytes) for %s: out of device memory", bytes, what);
    return GPR_ENOMEM;
  }
  if (e != cudaSuccess) {
    *p = nullptr;
    set_error("cudaMalloc(%zu bytes) for %s: %s", bytes, what, cudaGetErrorString(e));
    return GPR_ECUDA;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  g_live[*p] = Block{*p, bytes, dev, 0};
  return GPR_OK;
}

namespace {
thread_local std::vector<void *> *t_deferred = nullptr;
}  // namespace

DeferFrees::DeferFrees() : prev_(t_deferred) { t_deferred = &list_; }

DeferFrees::~DeferFrees() {
  t_deferred = prev_;
  for (void *p : list_) dfree(p);
}

void dfree(void *p) {
  if (!p) return;
  if (t_deferred) {
    t_deferred->push_back(p);
    return;
  }
  std::unique_lock<std::mutex> lk(g_mu);
  auto it = g_live.find(p);
  if (it == g_live.end()) {
    lk.unlock();
    cudaFree(p);
    return;
  }
  Block b = it->second;
  g_live.erase(it);
  b.freed = ++g_frees;
  if (b.bytes < kCacheMin && g_small_bytes + b.bytes > kSmallCap) {
    lk.unlock();
    give_back(b);
    return;
  }
  put_locked(b);
  while (g_free_bytes > kCacheCap && !g_free.empty()) {
    size_t big = 0;
    for (size_t i = 1; i < g_free.size(); ++i)
      if (g_free[i].bytes > g_free[big].bytes) big = i;
    Block v = g_free[big];
    g_free[big] = g_free.back();
    g_free.pop_back();
    g_free_bytes -= v.bytes;
    lk.unlock();  // cudaFree waits for the device
    give_back(v);
    lk.lock();
  }
}

size_t cached_bytes() {
  std::lock_guard<std::mutex> lk(g_mu);
  return g_free_bytes + g_small_bytes;
}

}  // namespace gpr

extern "C" {

int gpr_free(void *d_ptr) {
  // As cudaFree, waits for the device of the block, so that the caller's work on it is
  // over, and frees it whatever that work's status.
  const cudaError_t e = gpr::wait_for_owner(d_ptr);
  gpr::dfree(d_ptr);
  GPR_CUDA(e);
  GPR_CUDA(cudaGetLastError());
  return GPR_OK;
}

int gpr_release_cached(long long *released_bytes) {
  std::vector<gpr::Block> kept;
  {
    std::lock_guard<std::mutex> lk(gpr::g_mu);
    if (released_bytes) *released_bytes = (long long)(gpr::g_free_bytes + gpr::g_small_bytes);
    kept = gpr::drain_locked(-1);
  }
  for (const gpr::Block &b : kept) gpr::give_back(b);
  GPR_CUDA(cudaGetLastError());
  return GPR_OK;
}

int gpr_cached_bytes(long long *bytes) {
  if (!bytes) {
    gpr::set_error("gpr_cached_bytes: NULL out");
    return GPR_EINVAL;
  }
  *bytes = (long long)gpr::cached_bytes();
  return GPR_OK;
}

int gpr_malloc(void **d_ptr, size_t bytes) {
  if (!d_ptr) {
    gpr::set_error("gpr_malloc: NULL out");
    return GPR_EINVAL;
  }
  return gpr::dmalloc(d_ptr, bytes ? bytes : 1, "gpr_malloc");
}

}  // extern "C"
