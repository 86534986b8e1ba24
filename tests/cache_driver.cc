// The block cache (gpr_cache.cc) over a CUDA runtime that only keeps books: blocks are
// numbers, and every call is recorded.
//
//   cache_driver <case>      prints "ok", or what differs
#include <cuda_runtime_api.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <chrono>
#include <condition_variable>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "gpr_internal.cuh"

namespace {
std::mutex mu;
std::condition_variable cv;
thread_local int device = 0;
std::vector<int> syncs;        // devices that were waited for, in order
std::set<void *> allocated;    // blocks the driver has handed out
cudaError_t sync_result = cudaSuccess;
void (*on_sync)() = nullptr;   // called from inside a wait, without locks of the runtime
uintptr_t next_block = 1 << 20;

int failed = 0;
void expect(bool what, const char *text) {
  if (what) return;
  printf("wrong: %s\n", text);
  failed = 1;
}
void *get(size_t bytes) {
  void *p = nullptr;
  expect(gpr::dmalloc(&p, bytes, "block") == GPR_OK, "allocation");
  return p;
}
}  // namespace

namespace gpr {
void set_error(const char *, ...) {}
}  // namespace gpr

extern "C" {
cudaError_t cudaGetDevice(int *d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  device = d;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t bytes) {
  std::lock_guard<std::mutex> lk(mu);
  *p = reinterpret_cast<void *>(next_block);
  next_block += (bytes + 511) / 512 * 512;
  allocated.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> lk(mu);
  expect(allocated.erase(p) == 1, "free of a block that is not allocated");
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  if (on_sync) on_sync();
  std::lock_guard<std::mutex> lk(mu);
  syncs.push_back(device);
  return sync_result;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
}

namespace {

// One wait covers every block freed before it; blocks stay with their device.
void waits() {
  void *a = get(1000), *b = get(1000), *big = get(3 << 20);
  gpr::dfree(a);
  gpr::dfree(b);
  gpr::dfree(big);
  expect(syncs.empty(), "a free waits for nothing");
  void *c = get(1000), *d = get(900), *e = get((3 << 20) - 4096);
  expect((c == a && d == b) || (c == b && d == a), "small blocks come back");
  expect(e == big, "a large block comes back");
  expect(syncs == std::vector<int>({0}), "one wait for all three");
  gpr::dfree(c);
  device = 1;
  void *f = get(1000);
  expect(f != c, "a block of another device");
  expect(syncs.size() == 1, "a new block waits for nothing");
  device = 0;
  expect(get(1000) == c && syncs.size() == 2, "a block freed since needs a wait of its own");
  void *x = get(2 << 20), *y = get(2 << 20), *z = get(3000);
  gpr::dfree(x);
  gpr::dfree(z);
  expect(get(3000) == z && syncs.size() == 3, "a wait");
  gpr::dfree(y);
  expect(get(2 << 20) == x && syncs.size() == 3, "of equal blocks one that needs no wait");
}

// A wait that is refused has waited for nothing.
void refused() {
  void *a = get(1000), *b = get(2 << 20);
  gpr::dfree(a);
  gpr::dfree(b);
  sync_result = cudaErrorStreamCaptureUnsupported;
  void *c = get(1000), *d = get(2 << 20);
  expect(c != a && d != b, "blocks that may be in use are not handed out");
  sync_result = cudaSuccess;
  const size_t before = syncs.size();
  void *e = get(1000), *f = get(2 << 20);
  expect(e == a && f == b, "they come back behind a wait that succeeds");
  expect(syncs.size() == before + 1, "one wait for both");
}

// While one thread waits for the GPU, others allocate and free.
bool in_wait = false, other_done = false;
void while_waiting() {
  std::unique_lock<std::mutex> lk(mu);
  in_wait = true;
  cv.notify_all();
  expect(cv.wait_for(lk, std::chrono::seconds(5), [] { return other_done; }),
         "another thread's allocation and free do not wait for the GPU");
}
void waiting_in_malloc() {
  void *a = get(1000), *b = get(2000);
  gpr::dfree(a);
  on_sync = while_waiting;
  std::thread other([&] {
    {
      std::unique_lock<std::mutex> lk(mu);
      cv.wait(lk, [] { return in_wait; });
      on_sync = nullptr;
    }
    gpr::dfree(get(5000));
    gpr::dfree(b);
    std::lock_guard<std::mutex> lk(mu);
    other_done = true;
    cv.notify_all();
  });
  expect(get(1000) == a, "the block behind the wait");
  other.join();
  // blocks freed during that wait are not covered by it
  const size_t before = syncs.size();
  get(2000);
  expect(syncs.size() == before + 1, "a block freed while another thread waited");
}

// gpr_free waits for the block's device, and frees whatever that wait reports.
void free_entry() {
  void *a = get(1000);
  device = 1;
  expect(gpr_free(a) == GPR_OK, "gpr_free");
  expect(syncs == std::vector<int>({0}) && device == 1, "waits for the block's device");
  device = 0;
  void *b = get(5000);
  sync_result = cudaErrorLaunchFailure;
  long long before = 0, after = 0;
  gpr_cached_bytes(&before);
  expect(gpr_free(b) == GPR_ECUDA, "gpr_free reports the error");
  gpr_cached_bytes(&after);
  expect(after == before + 8192, "and frees");
  sync_result = cudaSuccess;
  syncs.clear();
  expect(gpr_free(nullptr) == GPR_OK && syncs.empty(), "gpr_free(NULL)");
  long long released = 0;
  expect(gpr_release_cached(&released) == GPR_OK && released == after, "release");
  expect(allocated.empty(), "every block given back");
}

}  // namespace

int main(int argc, char **argv) {
  const std::string c = argc > 1 ? argv[1] : "";
  if (c == "waits") waits();
  else if (c == "refused") refused();
  else if (c == "threads") waiting_in_malloc();
  else if (c == "free") free_entry();
  else return 2;
  if (!failed) printf("ok\n");
  return 0;
}
