// PageRank entry point that allocates no memory.
//
// Some callers cannot let a library call cudaMalloc: a host framework that
// reserves the device heap for its own allocator up front, or a latency-
// critical caller that may not take the device-wide synchronisation that
// cudaMalloc / cudaFree can cause.  gpr_pagerank_noalloc serves them: it
// solves directly on the caller's device CSR, and the only memory it needs
// beyond the caller's inputs and outputs -- two contribution buffers, the
// per-CTA residual partials, the per-sweep residual history and a few status
// words -- lives in one file-scope device array, g_noalloc_scratch, of fixed
// size (kNoAllocBytes, about 8 MiB).  Every GPU that loads the library holds
// that array until the process exits.
//
// Host code only ever sees a host-side stand-in for the array's name, so the
// device address is looked up once per device with cudaGetSymbolAddress, with
// that device current, on the first call made on it; that first call should
// therefore come before any stream capture.  All calls share the array and it
// keeps the previous call's contents: the words that must start at zero are
// cleared at the start of every call, and calls that overlap on the GPU (on
// different streams, or from different host threads) race on it.
//
// The sweep sums each row in CSR order with the reference's float operations
// (src/pr/omp_base.cc:34-39), so its scores are identical to the reference's;
// the residual is reduced in FP64 per CTA and combined by the last CTA of each
// sweep.
#include <math.h>
#include <string.h>

#include <chrono>
#include <mutex>

#include "gpr_internal.cuh"
#include "gpr_guard.h"

namespace {

constexpr int kNoAllocMaxVertices = 1 << 20;  // largest m accepted
constexpr int kNoAllocMaxIter = 1000;         // largest max_iter accepted
constexpr int kNoAllocBlock = 256;
// Edges a CTA stages in shared memory at a time: 16 independent loads per
// thread.  Half of that measured slower: a long row pays for every tile's end.
constexpr int kNoAllocTile = 16 * kNoAllocBlock;
constexpr int kNoAllocMaxCtas = (kNoAllocMaxVertices + kNoAllocBlock - 1) / kNoAllocBlock;

// Byte layout of the scratch array (all offsets 256-byte aligned).
constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kOffContrib0 = 0;
constexpr size_t kOffContrib1 = align256(kOffContrib0 + sizeof(float) * (kNoAllocMaxVertices + 1));
constexpr size_t kOffCtaErr = align256(kOffContrib1 + sizeof(float) * (kNoAllocMaxVertices + 1));
constexpr size_t kOffHist = align256(kOffCtaErr + sizeof(double) * kNoAllocMaxCtas);
constexpr size_t kOffWords = align256(kOffHist + sizeof(double) * kNoAllocMaxIter);
constexpr size_t kNoAllocBytes = align256(kOffWords + sizeof(int) * 8);

// words[0] arrival count, [1] sweeps done, [2] done flag, [3] CSR error flags
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

struct NoAllocArgs {
  int m;
  const int *rowptr, *col, *outdeg;
  float *s;
  float *c0, *c1;
  double *cta_err, *hist;
  int *words;
  float base, damp;
  double tol;
  int max_iter;
};

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void k_na_validate(int m, long long nnz, const int *__restrict__ rowptr,
                              const int *__restrict__ col, const int *__restrict__ outdeg,
                              int *words) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i <= m; i += stride) {
    if (i == 0 && rowptr[0] != 0) atomicOr(words + 3, 1);
    if (i == m && (long long)rowptr[m] != nnz) atomicOr(words + 3, 2);
    if (i < m && (rowptr[i] > rowptr[i + 1] || outdeg[i] < 0)) atomicOr(words + 3, 4);
  }
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nnz; e += stride) {
    const int c = col[e];
    if (c < 0 || c >= m) atomicOr(words + 3, 8);
  }
}

__global__ void k_na_prologue(NoAllocArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.m) a.c0[i] = __fdiv_rn(a.s[i], __int2float_rn(a.outdeg[i]));
}

// acc + v[lo] + ... + v[hi - 1] in order.  The loads of a batch are issued before
// its additions, so a value costs an addition's latency and not a load's as well.
__device__ __forceinline__ float add_in_order(const float *v, int lo, int hi, float acc) {
  for (; lo < hi; lo += 16) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = lo + i < hi ? v[lo + i] : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (lo + i < hi) acc = __fadd_rn(acc, x[i]);
  }
  return acc;
}

// Values of a long row per lane and step of ordered_sum; odd, so that the
// lanes' strides fall on different shared-memory banks.
constexpr int kOrdV = 31;
// Rows with more values than this in a staged tile are added by their warp.
// A shorter row gains nothing from a warp: its first steps, with a new binade after
// every doubling of the sum, mostly add one by one.
constexpr int kOrdMin = 384;

// acc + v[lo] + v[lo + 1] + ... + v[hi - 1], each addition rounded to nearest
// even as __fadd_rn does in that order, by one warp (all lanes call it with
// the same arguments and get the sum).
//
// While the running sum stays within one binade it is A * u for an integer A in
// [2^23, 2^24), and adding x >= 0 rounds x / u to an integer by itself: only
// where x / u lies halfway between two integers does the result depend on A
// (on its parity).  So where no value is halfway and the sum stays in the
// binade, the roundings are independent, the integers can be added in any order,
// and their total is added to the sum's bits.  Each lane takes kOrdV
// consecutive values (x / u = y, an exact scaling by a power of two; y < 2^22, so
// that adding 1.5 * 2^23 rounds y to the nearest integer and leaves it in the
// low bits).  Lanes before the first one that meets a halfway value, a y out of
// range (a negative, infinite or NaN value among them) or the end of the binade
// are accepted; that lane's values are added one by one, and the next step
// starts behind them with the new binade.  A step that accepts few lanes adds
// a longer stretch one by one.
__device__ float ordered_sum(const float *v, int lo, int hi, float acc, int lane) {
  constexpr float kRound = 12582912.f;  // 1.5 * 2^23
  constexpr unsigned kRoundBits = 0x4B400000u, kTooBig = 0x4A800000u;  // 2^22
  while (lo < hi) {
    const unsigned bits = __float_as_uint(acc), eb = bits >> 23;
    int take = 0;  // lanes accepted
    if (eb >= 23u && eb < 255u) {  // positive, finite, and 2^s below is a normal float
      const float scale = __uint_as_float((277u - eb) << 23);
      const int b = lo + lane * kOrdV;
      unsigned sum = 0u, top = 0u;
      bool half = false;
#pragma unroll
      for (int q = 0; q < kOrdV; ++q) {
        const float y = b + q < hi ? __fmul_rn(v[b + q], scale) : 0.f;
        const float t = __fadd_rn(y, kRound);
        half |= fabsf(__fsub_rn(y, __fsub_rn(t, kRound))) == 0.5f;
        sum += __float_as_uint(t) - kRoundBits;
        top = max(top, __float_as_uint(y));
      }
      const bool bad = half || top >= kTooBig;
      const unsigned room = 0x7FFFFFu - (bits & 0x7FFFFFu);  // largest total that stays
      if (bad || sum > room) sum = room + 1u;
      // sums of lanes up to each; room + 1 <= 2^23 a lane, so nothing wraps
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += t;
      }
      const unsigned stop = __ballot_sync(0xffffffffu, sum > room);
      take = stop ? __ffs(stop) - 1 : 32;
      const unsigned total = __shfl_sync(0xffffffffu, sum, max(take, 1) - 1);
      if (take > 0) acc = __uint_as_float(bits + total);
      lo = min(hi, lo + take * kOrdV);
    }
    if (take < 32) {
      const int e = min(hi, lo + (take < 4 ? 2 : 1) * kOrdV);
      acc = add_in_order(v, lo, e, acc);
      lo = e;
    }
  }
  return acc;
}

// One sweep; sweep index and done flag live in the scratch words, so launches
// after convergence return at once.
//
// A CTA owns 256 consecutive rows, whose edges are one contiguous range: all
// threads stage the range's contributions tile by tile in shared memory
// (coalesced indices, 16 gathers in flight per thread), and each thread then
// adds its own row's part in CSR order; long parts are added by the row's warp
// (ordered_sum).  What bounds a sweep is the longest row's chain of dependent
// adds.  RMAT, 250,007 vertices, edge factor 16, 24 sweeps: with one thread per
// row loading its own edges the chain held an L2 round trip per few edges (820 us
// per sweep, 0.06 instructions issued per cycle, 16.9 ms per call); staged, and
// one thread adding a row, 2.6 ms per call; with ordered_sum 1.4 ms.
__global__ void __launch_bounds__(kNoAllocBlock, 6) k_na_sweep(NoAllocArgs a) {
  __shared__ int s_it, s_last;
  __shared__ double red[kNoAllocBlock / 32];
  __shared__ float s_val[kNoAllocTile];
  if (threadIdx.x == 0) {
    const int done = *(volatile int *)(a.words + 2);
    s_it = done ? -1 : *(volatile int *)(a.words + 1);
  }
  __syncthreads();
  const int it = s_it;
  if (it < 0) return;
  const float *cin = (it & 1) ? a.c1 : a.c0;
  float *cout = (it & 1) ? a.c0 : a.c1;
  const int r0 = blockIdx.x * kNoAllocBlock, v = r0 + threadIdx.x;
  const bool has = v < a.m;
  const int first = a.rowptr[r0], end = a.rowptr[min(a.m, r0 + kNoAllocBlock)];
  const int e0 = has ? a.rowptr[v] : end, e1 = has ? a.rowptr[v + 1] : end;
  const float so = has ? a.s[v] : 0.f;
  const int od = has ? a.outdeg[v] : 1;
  float total = 0.f;
  constexpr int kPer = kNoAllocTile / kNoAllocBlock;
  for (long long t = first; t < end; t += kNoAllocTile) {
    const int n = (int)min((long long)kNoAllocTile, end - t);
    int c[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int i = q * kNoAllocBlock + threadIdx.x;
      c[q] = i < n ? a.col[t + i] : -1;
    }
    float x[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) x[q] = c[q] >= 0 ? cin[c[q]] : 0.f;
    __syncthreads();  // the previous tile has been added
#pragma unroll
    for (int q = 0; q < kPer; ++q) s_val[q * kNoAllocBlock + threadIdx.x] = x[q];
    __syncthreads();
    const int lo = (int)max(0LL, e0 - t), hi = (int)min((long long)n, e1 - t);
    unsigned longs = __ballot_sync(0xffffffffu, hi - lo > kOrdMin);
    if (hi - lo <= kOrdMin) total = add_in_order(s_val, lo, hi, total);
    __syncwarp();
    for (; longs; longs &= longs - 1) {
      const int src = __ffs(longs) - 1;
      const float sum = ordered_sum(s_val, __shfl_sync(0xffffffffu, lo, src),
                                    __shfl_sync(0xffffffffu, hi, src),
                                    __shfl_sync(0xffffffffu, total, src), threadIdx.x & 31);
      if ((threadIdx.x & 31) == src) total = sum;
    }
  }
  double err = 0.0;
  if (has) {
    const float sn = __fadd_rn(a.base, __fmul_rn(a.damp, total));
    a.s[v] = sn;
    cout[v] = __fdiv_rn(sn, __int2float_rn(od));
    err = (double)fabsf(__fsub_rn(sn, so));
  }
  err = warp_sum_d(err);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = err;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kNoAllocBlock / 32; ++w) t += red[w];
    a.cta_err[blockIdx.x] = t;
    __threadfence();
    s_last = atomicAdd(a.words, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (s_last && threadIdx.x < 32) {
    __threadfence();
    double t = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += 32) t += __ldcg(a.cta_err + i);
    t = warp_sum_d(t);
    if (threadIdx.x == 0) {
      a.hist[it] = t;
      atomicExch(a.words, 0);
      a.words[1] = it + 1;
      if (t < a.tol || it + 1 >= a.max_iter) a.words[2] = 1;
      __threadfence();
    }
  }
}

std::mutex g_setup_mu;
unsigned char *g_scratch_ptr[64] = {nullptr};

// Device address of the scratch array on the current device, looked up once.
int scratch_for_current_device(unsigned char **out) {
  int dev = 0;
  GPR_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    gpr::set_error("gpr_pagerank_noalloc: device index %d out of range", dev);
    return GPR_EINVAL;
  }
  std::lock_guard<std::mutex> lock(g_setup_mu);
  if (!g_scratch_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      gpr::set_error("gpr_pagerank_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      return GPR_ECUDA;
    }
    g_scratch_ptr[dev] = static_cast<unsigned char *>(p);
  }
  *out = g_scratch_ptr[dev];
  return GPR_OK;
}

}  // namespace

extern "C" {

long long gpr_pagerank_noalloc_max_vertices(void) { return kNoAllocMaxVertices; }

int gpr_pagerank_noalloc(int m, int nnz, const int *d_rowptr, const int *d_col,
                         const int *d_outdeg, float *d_scores, const gpr_pr_opts *opts,
                         gpr_pr_stats *stats, void *stream) {
  GPR_ENTRY_BEGIN
  gpr_pr_opts o;
  if (opts) o = *opts;
  else gpr_pr_opts_default(&o);
  if (m < 0 || nnz < 0 || (m == 0 && nnz != 0) ||
      (m > 0 && (!d_rowptr || !d_outdeg || !d_scores)) || (nnz > 0 && !d_col)) {
    gpr::set_error("gpr_pagerank_noalloc: invalid arguments (m=%d nnz=%d)", m, nnz);
    return GPR_EINVAL;
  }
  if (m > kNoAllocMaxVertices) {
    gpr::set_error("gpr_pagerank_noalloc: m=%d exceeds the fixed scratch limit of %d vertices",
                   m, kNoAllocMaxVertices);
    return GPR_EINVAL;
  }
  if (o.max_iter < 0 || o.max_iter > kNoAllocMaxIter || !(o.tol >= 0.0) ||
      !(o.damping >= 0.f && o.damping <= 1.f)) {
    gpr::set_error("gpr_pagerank_noalloc: invalid options (max_iter %d must be in [0, %d])",
                   o.max_iter, kNoAllocMaxIter);
    return GPR_EINVAL;
  }
  gpr_pr_stats st;
  memset(&st, 0, sizeof(st));
  if (m == 0) {
    // no vertices: the sweeps are empty and their residuals 0
    st.iterations = gpr::empty_graph_sweeps(o.tol, o.max_iter);
    if (stats) *stats = st;
    return GPR_OK;
  }
  const auto t0 = std::chrono::steady_clock::now();
  unsigned char *base = nullptr;
  GPR_TRY(scratch_for_current_device(&base));
  cudaStream_t s = (cudaStream_t)stream;
  NoAllocArgs a;
  a.m = m;
  a.rowptr = d_rowptr;
  a.col = d_col;
  a.outdeg = d_outdeg;
  a.s = d_scores;
  a.c0 = reinterpret_cast<float *>(base + kOffContrib0);
  a.c1 = reinterpret_cast<float *>(base + kOffContrib1);
  a.cta_err = reinterpret_cast<double *>(base + kOffCtaErr);
  a.hist = reinterpret_cast<double *>(base + kOffHist);
  a.words = reinterpret_cast<int *>(base + kOffWords);
  a.damp = o.damping;
  a.base = (1.0f - o.damping) / (float)m;  // src/pr/omp_base.cc:16
  a.tol = o.tol;
  a.max_iter = o.max_iter;
  const unsigned grid = (unsigned)((m + kNoAllocBlock - 1) / kNoAllocBlock);
  GPR_CUDA(cudaMemsetAsync(a.words, 0, sizeof(int) * 8, s));
  k_na_validate<<<148 * 8, 256, 0, s>>>(m, nnz, d_rowptr, d_col, d_outdeg, a.words);
  GPR_CUDA(cudaGetLastError());
  int words[4];
  GPR_CUDA(cudaMemcpyAsync(words, a.words, sizeof(words), cudaMemcpyDeviceToHost, s));
  GPR_CUDA(cudaStreamSynchronize(s));
  if (words[3]) {
    gpr::set_error("gpr_pagerank_noalloc: malformed CSR (flags 0x%x)", words[3]);
    return GPR_EINVAL;
  }
  if (o.max_iter == 0) {
    if (stats) *stats = st;
    return GPR_OK;
  }
  k_na_prologue<<<grid, kNoAllocBlock, 0, s>>>(a);
  GPR_CUDA(cudaGetLastError());
  int launches = 2, issued = 0, done = 0;
  while (!done && issued < o.max_iter) {
    for (int q = 0; q < 8 && issued < o.max_iter; ++q, ++issued) {
      k_na_sweep<<<grid, kNoAllocBlock, 0, s>>>(a);
      ++launches;
    }
    GPR_CUDA(cudaGetLastError());
    GPR_CUDA(cudaMemcpyAsync(words, a.words, sizeof(words), cudaMemcpyDeviceToHost, s));
    GPR_CUDA(cudaStreamSynchronize(s));
    done = words[2];
  }
  st.iterations = words[1];
  if (st.iterations > 0) {
    // on the caller's stream: no device-wide synchronisation
    GPR_CUDA(cudaMemcpyAsync(&st.residual, a.hist + st.iterations - 1, sizeof(double),
                             cudaMemcpyDeviceToHost, s));
    GPR_CUDA(cudaStreamSynchronize(s));
  }
  st.gpu_launches = launches;
  st.solve_ms =
      std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  st.loop_ms = st.solve_ms;
  if (stats) *stats = st;
  return GPR_OK;
  GPR_ENTRY_END("gpr_pagerank_noalloc")
}

}  // extern "C"
