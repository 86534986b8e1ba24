// Loaded ahead of libgpr.so (RTLD_GLOBAL), takes the place of its device allocations:
// each goes to the library's own, unless a failure is asked for by the name that the
// caller gives the block, and the blocks handed out are counted.  Host only: nothing
// on the GPU fails.
#include <dlfcn.h>
#include <string.h>

#include <map>
#include <mutex>
#include <set>
#include <string>

namespace {
std::mutex mu;
std::set<void *> live;
std::map<std::string, size_t> asked;  // bytes of the last allocation of each name
std::string fail_what;
int fail_status = 0, fail_count = 0;
std::string call_what;
void (*call)() = nullptr;

void *real(const char *name) {
  static void *lib = nullptr;
  if (!lib) lib = dlopen("libgpr.so", RTLD_NOLOAD | RTLD_LAZY);
  return dlsym(lib, name);
}
}  // namespace

namespace gpr {
int dmalloc(void **p, size_t bytes, const char *what) {
  {
    std::lock_guard<std::mutex> lk(mu);
    asked[what] = bytes;
    if (fail_count > 0 && fail_what == what) {
      --fail_count;
      *p = nullptr;
      return fail_status;
    }
  }
  static auto f = reinterpret_cast<int (*)(void **, size_t, const char *)>(
      real("_ZN3gpr7dmallocEPPvmPKc"));
  const int rc = f(p, bytes, what);
  if (call && call_what == what) call();
  std::lock_guard<std::mutex> lk(mu);
  if (rc == 0) live.insert(*p);
  return rc;
}

void dfree(void *p) {
  {
    std::lock_guard<std::mutex> lk(mu);
    live.erase(p);
  }
  static auto f = reinterpret_cast<void (*)(void *)>(real("_ZN3gpr5dfreeEPv"));
  f(p);
}
}  // namespace gpr

extern "C" {
// The next `count` allocations named `what` return `status`.
void shim_fail(const char *what, int status, int count) {
  std::lock_guard<std::mutex> lk(mu);
  fail_what = what;
  fail_status = status;
  fail_count = count;
}
// `f` is called behind every allocation named `what`.
void shim_call(const char *what, void (*f)()) {
  call_what = what;
  call = f;
}
// Bytes of the last allocation named `what` (0: none).
long long shim_bytes(const char *what) {
  std::lock_guard<std::mutex> lk(mu);
  return (long long)asked[what];
}
int shim_pending() { return fail_count; }
int shim_live() { return (int)live.size(); }
}
