// Error state, scratch pool, device-wide scans and FP64 reductions.
#include <cuda.h>

#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "context.cuh"
#include "scan.cuh"

static thread_local char g_err[512] = "";

extern "C" const char* xk_version(void) { return "xkgpu 0.1 (sm_103a)"; }
extern "C" const char* xk_last_error(void) { return g_err; }

xk_status xk_set_cuda_error(cudaError_t e, const char* file, int line) {
  snprintf(g_err, sizeof(g_err), "CUDA error %d (%s) at %s:%d", (int)e, cudaGetErrorString(e), file, line);
  return XK_ERR_CUDA;
}
xk_status xk_set_error(xk_status code, const char* msg) {
  snprintf(g_err, sizeof(g_err), "%s", msg);
  return code;
}

int xk_sm_count() {
  constexpr int MAX_DEV = 64;
  static std::atomic<int> cache[MAX_DEV];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 1;
  if (dev >= MAX_DEV) {
    int n = 0;
    return (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) ? n : 1;
  }
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
  cache[dev].store(n, std::memory_order_relaxed);
  return n;
}

// --------------------------------------------------------------------------- scratch

// Id of the calling thread's current context (CUDA 12's cuCtxGetId, reached
// through the runtime's driver entry points so that the library needs no
// libcuda at link time); false when there is no current context yet or the
// driver does not offer the calls.
namespace {
using PfnCtxGetCurrent = CUresult (*)(CUcontext*);
using PfnCtxGetId = CUresult (*)(CUcontext, unsigned long long*);
}  // namespace

bool xk_context_id(unsigned long long* id) {
  static PfnCtxGetCurrent get_current = nullptr;
  static PfnCtxGetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    void* f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<PfnCtxGetCurrent>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<PfnCtxGetId>(f);
  });
  CUcontext c = nullptr;
  if (!get_current || !get_id || get_current(&c) != CUDA_SUCCESS || !c) return false;
  return get_id(c, id) == CUDA_SUCCESS;
}

xk_status xk_context_here(unsigned long long* id) {
  if (xk_context_id(id)) return XK_OK;
  RelaxedCapture relaxed;
  XK_CUDA(cudaFree(nullptr));
  if (xk_context_id(id)) return XK_OK;
  int dev = 0;  // a driver without ids: one context per device
  XK_CUDA(cudaGetDevice(&dev));
  *id = ~0ULL - (unsigned long long)dev;
  return XK_OK;
}

namespace {
// the pool of each context, never given back: calls on other threads may be using it
struct ScratchPool {
  cudaMemPool_t pool = nullptr;
  void drop() {}
};
std::mutex g_pool_mutex;
PerContext<ScratchPool>& scratch_pools() {
  static PerContext<ScratchPool>* const pools = new PerContext<ScratchPool>;
  return *pools;
}

// the current device's pool, made on first use; null if there is none to be had
cudaMemPool_t scratch_pool(bool make) {
  int dev = 0;
  unsigned long long id = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || !xk_context_id(&id)) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  ScratchPool* g = scratch_pools().find(id);
  if (g && g->pool) return g->pool;
  if (!make || (!g && !(g = scratch_pools().add(id)))) return nullptr;
  RelaxedCapture relaxed;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  uint64_t keep = XK_SCRATCH_KEEP;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    if (pool) cudaMemPoolDestroy(pool);
    cudaGetLastError();
    return nullptr;
  }
  return g->pool = pool;
}
}  // namespace

xk_status xk_scratch_alloc(void** out, size_t bytes, cudaStream_t s) {
  if (bytes < 1) bytes = 1;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  XK_CUDA(cudaStreamIsCapturing(s, &cap));
  cudaMemPool_t pool = cap == cudaStreamCaptureStatusNone ? scratch_pool(true) : nullptr;
  XK_CUDA(pool ? cudaMallocFromPoolAsync(out, bytes, pool, s) : cudaMallocAsync(out, bytes, s));
  return XK_OK;
}

extern "C" xk_status xk_scratch_trim(int64_t keep_bytes) {
  if (keep_bytes < 0) return xk_set_error(XK_ERR_ARG, "xk_scratch_trim: keep_bytes");
  if (cudaMemPool_t pool = scratch_pool(false)) {
    RelaxedCapture relaxed;
    XK_CUDA(cudaMemPoolTrimTo(pool, (size_t)keep_bytes));
  }
  return XK_OK;
}

// --------------------------------------------------------------------------- read-back

namespace {
// a pinned buffer and an event per thread and context
struct Readback {
  int64_t* host = nullptr;
  cudaEvent_t event = nullptr;
  bool pending = false;  // begun and not ended
  void drop() {
    if (event) cudaEventDestroy(event);
    if (host) cudaFreeHost(host);
  }
};
thread_local PerContext<Readback> g_reads;
thread_local Readback* g_begun = nullptr;
}  // namespace

xk_status xk_read_begin(const int64_t* dev, int words, cudaStream_t s) {
  if (words > XK_READ_WORDS) return xk_set_error(XK_ERR_ARG, "xk_read_begin: words");
  Readback* r;
  XK_TRY(g_reads.here(&r));
  if (!r->host || !r->event) {
    RelaxedCapture relaxed;
    if (!r->host) XK_CUDA(cudaHostAlloc((void**)&r->host, sizeof(int64_t) * XK_READ_WORDS, cudaHostAllocDefault));
    if (!r->event) XK_CUDA(cudaEventCreateWithFlags(&r->event, cudaEventDisableTiming));
  }
  if (r->pending) {  // a call failed in between: its copy may still be on its way into the buffer
    XK_CUDA(cudaEventSynchronize(r->event));
    r->pending = false;
  }
  XK_CUDA(cudaMemcpyAsync(r->host, dev, sizeof(int64_t) * words, cudaMemcpyDeviceToHost, s));
  XK_CUDA(cudaEventRecord(r->event, s));
  r->pending = true;
  g_begun = r;
  return XK_OK;
}

xk_status xk_read_end(int64_t* host, int words) {
  Readback* r = g_begun;
  XK_CUDA(cudaEventSynchronize(r->event));
  r->pending = false;
  for (int k = 0; k < words; ++k) host[k] = r->host[k];
  return XK_OK;
}

// --------------------------------------------------------------------------- scan

namespace {
template <typename TI>
__global__ void k_tile_sums(const TI* __restrict__ in, long long n, int64_t* __restrict__ bsum) {
  __shared__ int64_t wt[SCAN_T / 32];
  long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_I;
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i)
    if (base + i < n) s += (int64_t)in[base + i];
  int64_t tot;
  block_exclusive_scan<int64_t>(s, wt, &tot);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void k_scan_bsums(int64_t* bsum, long long nb, int64_t* total) {
  __shared__ int64_t wt[SCAN_T / 32];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (long long b0 = 0; b0 < nb; b0 += SCAN_T) {
    long long i = b0 + threadIdx.x;
    int64_t v = (i < nb) ? bsum[i] : 0;
    int64_t tot;
    int64_t ex = block_exclusive_scan<int64_t>(v, wt, &tot);
    int64_t c = carry;
    if (i < nb) bsum[i] = c + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry = c + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

template <typename TI, typename TO>
__global__ void k_tile_scan(const TI* __restrict__ in, TO* __restrict__ out, long long n,
                            const int64_t* __restrict__ bsum) {
  __shared__ int64_t wt[SCAN_T / 32];
  long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_I;
  int64_t loc[SCAN_I];
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i) {
    loc[i] = (base + i < n) ? (int64_t)in[base + i] : 0;
    s += loc[i];
  }
  int64_t ex = block_exclusive_scan<int64_t>(s, wt, nullptr) + bsum[blockIdx.x];
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i) {
    if (base + i < n) out[base + i] = (TO)ex;
    ex += loc[i];
  }
}

}  // namespace

xk_status xk_exclusive_scan_i32(const int32_t* in, int32_t* out, long long n, int64_t* total_dev,
                                cudaStream_t s, XkScratch* S) {
  if (n <= 0) {
    if (total_dev) XK_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(int64_t), s));
    return XK_OK;
  }
  if (in < out + n && out < in + n) return xk_set_error(XK_ERR_ARG, "scan: input and output overlap");
  XkScratch own(s);
  const size_t sums = sizeof(int64_t) * (size_t)scan_sums(n, 1), words = sizeof(int) * (size_t)scan_words(n, 1);
  char* buf = nullptr;
  XK_TRY((S ? *S : own).get(&buf, (long long)(sums + words)));
  XK_CUDA(cudaMemsetAsync(buf + sums, 0, words, s));
  return scan_launch(ScanI32{in, out, n, total_dev}, n, 1, reinterpret_cast<int64_t*>(buf),
                     reinterpret_cast<int*>(buf + sums), s);
}

long long xk_scan_tiles(long long n) { return n <= 0 ? 0 : (n + SCAN_TILE - 1) / SCAN_TILE; }

xk_status xk_exclusive_scan_i32_scratch(const int32_t* in, int32_t* out, long long n, int64_t* total_dev,
                                        int64_t* bsum, long long bsum_cap, cudaStream_t s) {
  if (n <= 0) {
    if (total_dev) XK_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(int64_t), s));
    return XK_OK;
  }
  long long nb = xk_scan_tiles(n);
  if (!bsum || nb > bsum_cap) return xk_set_error(XK_ERR_CAPACITY, "scan: block-sum scratch too small");
  k_tile_sums<int32_t><<<(unsigned)nb, SCAN_T, 0, s>>>(in, n, bsum);
  k_scan_bsums<<<1, SCAN_T, 0, s>>>(bsum, nb, total_dev);
  k_tile_scan<int32_t, int32_t><<<(unsigned)nb, SCAN_T, 0, s>>>(in, out, n, bsum);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

// --------------------------------------------------------------------------- FP64 sum of squares

namespace {
constexpr int N2_BLOCKS = 304;  // 2 x 152 SMs; fixed so that the summation order is fixed
constexpr int N2_T = 256;

__global__ void k_sumsq_partial(const double* __restrict__ x, long long n, double* __restrict__ part) {
  __shared__ double sm[N2_T];
  double acc = 0.0;
  for (long long i = (long long)blockIdx.x * N2_T + threadIdx.x; i < n; i += (long long)N2_BLOCKS * N2_T)
    acc = fma(x[i], x[i], acc);
  sm[threadIdx.x] = acc;
  __syncthreads();
  for (int w = N2_T / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sm[0];
}

__global__ void k_sum_final(const double* __restrict__ part, int np, double* __restrict__ out) {
  __shared__ double sm[512];
  double a = 0.0;
  for (int i = threadIdx.x; i < np; i += 512) a += part[i];
  sm[threadIdx.x] = a;
  __syncthreads();
  for (int w = 256; w > 0; w >>= 1) {
    if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sm[0];
}
}  // namespace

// Partials buffer for the fixed-order reductions; one per device, set up on the
// first call (cudaMalloc outside any capture).
static double* g_part[64] = {nullptr};

xk_status xk_partials_buffer(double** out) {
  int dev = 0;
  XK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return xk_set_error(XK_ERR_ARG, "device ordinal out of range");
  if (!g_part[dev]) XK_CUDA(cudaMalloc((void**)&g_part[dev], sizeof(double) * N2_BLOCKS));
  *out = g_part[dev];
  return XK_OK;
}

xk_status xk_sumsq_into(const double* x, long long n, double* out, cudaStream_t s) {
  double* part = nullptr;
  xk_status st = xk_partials_buffer(&part);
  if (st != XK_OK) return st;
  k_sumsq_partial<<<N2_BLOCKS, N2_T, 0, s>>>(x, n, part);
  k_sum_final<<<1, 512, 0, s>>>(part, N2_BLOCKS, out);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_norm2(const double* x, int64_t n, double* out, xk_stream s) {
  if (!x || !out || n < 0) return xk_set_error(XK_ERR_ARG, "xk_norm2: bad arguments");
  return xk_sumsq_into(x, n, out, (cudaStream_t)s);
}
