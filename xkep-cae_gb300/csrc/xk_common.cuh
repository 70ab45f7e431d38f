// Shared device/host helpers for the xkgpu kernels (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/xkgpu.h"

#define XK_HD __host__ __device__ __forceinline__
#define XK_D __device__ __forceinline__

// ---------------------------------------------------------------------------
// Exactly rounded double operations.  The parts of the path whose results are
// compared bit for bit with the reference (AABBs, closest point, gap, active
// set, midpoint prescreen) use these so that nvcc cannot contract a*b+c into
// an FMA; the reference's NumPy arithmetic rounds every product and sum.
// ---------------------------------------------------------------------------
#ifdef __CUDA_ARCH__
XK_D double xadd(double a, double b) { return __dadd_rn(a, b); }
XK_D double xsub(double a, double b) { return __dsub_rn(a, b); }
XK_D double xmul(double a, double b) { return __dmul_rn(a, b); }
XK_D double xdiv(double a, double b) { return __ddiv_rn(a, b); }
XK_D double xsqrt(double a) { return __dsqrt_rn(a); }
#else
inline double xadd(double a, double b) { return a + b; }
inline double xsub(double a, double b) { return a - b; }
inline double xmul(double a, double b) { return a * b; }
inline double xdiv(double a, double b) { return a / b; }
inline double xsqrt(double a) { return sqrt(a); }
#endif

// einsum('ij,ij->i') order measured for the reference's NumPy: (p0 + p2) + p1
XK_HD double xdot_es(const double* a, const double* b) {
  return xadd(xadd(xmul(a[0], b[0]), xmul(a[2], b[2])), xmul(a[1], b[1]));
}
// np.sum(axis=1) / np.linalg.norm order: (p0 + p1) + p2
XK_HD double xdot_seq(const double* a, const double* b) {
  return xadd(xadd(xmul(a[0], b[0]), xmul(a[1], b[1])), xmul(a[2], b[2]));
}
XK_HD void xcross(const double* a, const double* b, double* c) {
  c[0] = xsub(xmul(a[1], b[2]), xmul(a[2], b[1]));
  c[1] = xsub(xmul(a[2], b[0]), xmul(a[0], b[2]));
  c[2] = xsub(xmul(a[0], b[1]), xmul(a[1], b[0]));
}
// np.clip(x, 0, 1): NaN propagates
XK_HD double xclip01(double x) { return x < 0.0 ? 0.0 : (x > 1.0 ? 1.0 : x); }

// ---------------------------------------------------------------------------
// Generic small-vector helpers for the non-exact (FP64 plain or FP32 mixed) math.
// ---------------------------------------------------------------------------
template <typename T>
XK_HD T dot3(const T* a, const T* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
template <typename T>
XK_HD void cross3(const T* a, const T* b, T* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

template <typename T>
XK_HD T my_sqrt(T x);
template <>
XK_HD double my_sqrt<double>(double x) { return sqrt(x); }
template <>
XK_HD float my_sqrt<float>(float x) { return sqrtf(x); }
template <typename T>
XK_HD T my_abs(T x) { return x < T(0) ? -x : x; }

// Precision policy: P == XK_FP64 computes everything in double; P == XK_MIXED
// computes the bulk in float and keeps the rotation frames, the axial strain,
// the contact gap and all reductions in double.
template <int P>
struct Prec;
template <>
struct Prec<XK_FP64> { typedef double T; };
template <>
struct Prec<XK_MIXED> { typedef float T; };

// Double <-> float conversions in integer arithmetic.  On this GPU the conversion instructions issue
// at the FP64 rate (about 1.8 per clock per SM, like a double add, against about 100 float adds),
// and the integer operations at the full rate.  Both give the bits of the IEEE conversion (round to
// nearest, ties to even, for double -> float; exact for float -> double): the fields are moved as
// integers, and a result or input that is not a normal number (denormal, overflow, inf, nan) takes
// the conversion instruction.
XK_D float xk_d2f(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned e = (hi >> 20) & 0x7ffu;  // biased exponent; a normal float result needs e in [897, 1150]
  if (e - 897u > 253u) {
    if (((hi & 0x7fffffffu) | lo) == 0u) return __uint_as_float(hi & 0x80000000u);  // +-0
    return __double2float_rn(x);
  }
  const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);  // the top 23 of the 52 mantissa bits
  const unsigned r = lo & 0x1fffffffu;                     // the 29 bits rounded away
  const unsigned up = (r > 0x10000000u || (r == 0x10000000u && (m & 1u))) ? 1u : 0u;
  // a carry out of the mantissa raises the exponent (and past the largest float gives inf), as rounding does
  return __uint_as_float(((hi & 0x80000000u) | ((e - 896u) << 23) | m) + up);
}
XK_D double xk_f2d(float v) {
  const unsigned f = __float_as_uint(v);
  const unsigned e = (f >> 23) & 0xffu;
  if (e - 1u > 253u) {
    if ((f & 0x7fffffffu) == 0u) return __hiloint2double((int)(f & 0x80000000u), 0);  // +-0
    return (double)v;
  }
  return __hiloint2double((int)((f & 0x80000000u) | ((e + 896u) << 20) | ((f & 0x7fffffu) >> 3)), (int)(f << 29));
}

// FP64 on the FP64 pipe is scarce (about two operations per clock and SM; a divide or a square root takes some
// ten of them).  1/x and 1/sqrt(x) for x in the ordinary range: the approximate instruction, which sees the upper 32
// bits of x (1 - x r and 1 - x y^2 below 2^-19.9 and 2^-19.0 over 2^32 operands on this GPU), and one step of third
// order, r + r (e + e^2) and y + y e (1/2 + 3/8 e): three and five operations, where two Newton-Raphson steps take
// four and seven.  Not correctly rounded: the step leaves 2^-59.8 of r, and of y 2^-58 and half the rounding of x y;
// measured over those operands, at most 0.508 units of the last place of r and 1.0 of y.
XK_D double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
XK_D double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// x in [2^lo, 2^hi), tested on the high word: false for zero, negative values, infinities and NaN
template <int LO, int HI>
XK_D bool in_range64(double x) {
  return (unsigned)(__double2hiint(x) - ((1023 + LO) << 20)) < (unsigned)((HI - LO) << 20);
}
// x in [1 - 2^-32, 1 + 2^-30): a unit vector's square up to rounding, where 1/sqrt(x) = 3/2 - x/2 to 2^-61
XK_D bool near_one64(double x) {
  return (unsigned long long)(__double_as_longlong(x) - 0x3fefffffffe00000LL) < 0x600000ULL;
}

// The correctly rounded quotient and square root (the bits of the operators) on fewer FP64 operations, after
// Markstein ("Computation of elementary functions on the IBM RISC System/6000 processor", 1990): q = RN(x r), r the
// reciprocal, leaves the remainder x - d q, and RN(q + rem r) is x / d.  With D, R the mantissas of d and r as whole
// numbers (R D = 2^105) and r off by t units of its last place: a quotient next to a tie is at least 1 / (2 D) units
// from it, q half a unit, and the last step is off by t / (2 R), so it rounds correctly for t < R / D = 2^105 / D^2.
// Two Newton-Raphson steps give t < 1/2 + 2^-26 (rcp64 alone 0.508, too much for one divisor in a hundred), and
// 2^105 / D^2 is above 1/2 + 2^-21 unless the upper 20 bits of the mantissa are ones.
// The square root likewise from g = RN(x y) and its exact remainder: near a tie the step's error is below 2^-52.7
// units, and the few operands whose root lies that close (x = N (N + 1) - c, c small, N (N + 1) = c modulo a power of
// two) have been tried one by one.  A divisor's reciprocal serves several quotients.  Operands outside the range
// where the remainders are exact, and divisors of ones, take the operators, out of line.
__noinline__ static __device__ double div64_plain(double x, double d) { return x / d; }
__noinline__ static __device__ double sqrt64_plain(double x) { return sqrt(x); }
struct Divisor64 {
  double d, r;
  bool ok;
};
XK_D bool mag_in64(double x) {  // |x| in [2^-300, 2^300)
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) - (723u << 20) < (600u << 20);
}
XK_D Divisor64 divisor64(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  r = fma(r, fma(-d, r, 1.0), r);
  r = fma(r, fma(-d, r, 1.0), r);
  return {d, r, mag_in64(d) && (__double2hiint(d) & 0xfffff) != 0xfffff};
}
XK_D double div64(double x, const Divisor64& q) {
  if (!(q.ok && mag_in64(x))) return x == 0.0 && q.ok ? x : div64_plain(x, q.d);
  const double y = x * q.r;
  return fma(fma(-q.d, y, x), q.r, y);
}
XK_D double div64(double x, double d) { return div64(x, divisor64(d)); }
// v / d for a divisor next to one, d = 1 - k 2^-53 (k <= 16) or 1 + k 2^-52 (k < 8): as RN(v + v (1 - d)), one
// operation, which leaves out v (1 - d)^2, below 2^-45 units of the last place of v.  That decides the rounding where
// v (1 - d) lies on a tie or within 2^-45 of one (v = 1/2, d = 1 - 2^-53: a contact at 60 degrees), and v may be so
// close to a power of two that the quotient changes binade.  With m the mantissa of v and n = |1 - d| 2^53 <= 16, the
// product m n is within 512 of a multiple of 2^32 in both cases; where its lower word says so (one value in four
// million, and those of few bits, zeros, infinities) `sure` falls, and the caller takes the operator.  The whole test
// of m n takes ten times the integer operations: 632,000 exact narrowphases 299 us, this 277.
XK_D bool next_to_one64(double d) {
  return (unsigned long long)(__double_as_longlong(d) - 0x3feffffffffffff0LL) < 0x18ULL;
}
XK_D unsigned units_from_one64(double d) {
  const int k = (int)(__double_as_longlong(d) - 0x3ff0000000000000LL);
  return (unsigned)(k < 0 ? -k : 2 * k);
}
XK_D double div_next_to_one64(double v, double d, unsigned n, bool& sure) {
  sure = n == 0 || (unsigned)__double2loint(v) * n + 512u >= 1024u;
  return fma(v, 1.0 - d, v);
}
XK_D double sqrt64(double x) {
  if (!in_range64<-300, 300>(x)) return x == 0.0 ? x : sqrt64_plain(x);
  const double y = rsqrt64(x), g = x * y;
  return fma(fma(-g, g, x), 0.5 * y, g);
}

// Eight floats from a 32-byte aligned read-only address in one 256-bit load.
XK_D void ldg8(const float* __restrict__ p, float* v) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(p));
}

// Eight floats to a 32-byte aligned address in one 256-bit store.
XK_D void stg8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// ---------------------------------------------------------------------------
// Launch helpers
// ---------------------------------------------------------------------------
static inline int xk_blocks(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 0x7fffffffLL) b = 0x7fffffffLL;
  return (int)b;
}

#define XK_CHECK_LAUNCH()                                      \
  do {                                                         \
    cudaError_t e__ = cudaGetLastError();                      \
    if (e__ != cudaSuccess) return xk_set_cuda_error(e__, __FILE__, __LINE__); \
  } while (0)

#define XK_CUDA(call)                                          \
  do {                                                         \
    cudaError_t e__ = (call);                                  \
    if (e__ != cudaSuccess) return xk_set_cuda_error(e__, __FILE__, __LINE__); \
  } while (0)

xk_status xk_set_cuda_error(cudaError_t e, const char* file, int line);
xk_status xk_set_error(xk_status code, const char* msg);

// SM count of the current device, read once per device ordinal (1 when it cannot be read).
int xk_sm_count();

// Id of the calling thread's current context; false when there is none yet.
bool xk_context_id(unsigned long long* id);

// Stream-ordered scratch (freed with cudaFreeAsync) from a memory pool of this library's own, one per device: the
// default pool gives freed memory back to the system at every synchronisation, and a detection has five of them,
// each followed by allocations that map it again.  The pool holds on to at most XK_SCRATCH_KEEP bytes between
// calls; xk_scratch_trim gives those back too.  While s is being captured the default pool is used.
constexpr size_t XK_SCRATCH_KEEP = 256u << 20;
xk_status xk_scratch_alloc(void** out, size_t bytes, cudaStream_t s);

// The scratch of one call: get() carves aligned pieces from the block that reserve() allocated, or allocates
// what does not fit; everything is freed with the object, in stream order.
struct XkScratch {
  cudaStream_t s;
  void* p[24];
  int n = 0;
  char* base = nullptr;
  size_t size = 0, used = 0;
  explicit XkScratch(cudaStream_t st) : s(st) {}
  XkScratch(const XkScratch&) = delete;
  static size_t padded(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
  xk_status take(void** out, size_t bytes) {
    if (n >= (int)(sizeof(p) / sizeof(p[0]))) return xk_set_error(XK_ERR_OVERFLOW, "scratch table full");
    const xk_status r = xk_scratch_alloc(out, bytes, s);
    if (r == XK_OK) p[n++] = *out;
    return r;
  }
  xk_status reserve(size_t bytes) {
    size = padded(bytes);
    used = 0;
    return take((void**)&base, size);
  }
  template <typename T>
  xk_status get(T** out, long long count) {
    const size_t bytes = padded(sizeof(T) * (size_t)(count < 1 ? 1 : count));
    if (used + bytes <= size) {
      *out = reinterpret_cast<T*>(base + used);
      used += bytes;
      return XK_OK;
    }
    return take((void**)out, bytes);
  }
  ~XkScratch() {
    for (int i = 0; i < n; ++i) cudaFreeAsync(p[i], s);
  }
};

#define XK_TRY(x)                 \
  do {                            \
    xk_status r__ = (x);          \
    if (r__ != XK_OK) return r__; \
  } while (0)

// Up to XK_READ_WORDS words of device memory to the host in two steps, so that the kernels queued in between run
// while the host waits for the words and prepares what follows (a wait for the whole stream leaves the GPU idle
// for as long as the host needs to come back).  Each begin is followed by its end, on the same thread and device.
constexpr int XK_READ_WORDS = 8;
xk_status xk_read_begin(const int64_t* dev, int words, cudaStream_t s);
xk_status xk_read_end(int64_t* host, int words);

// Device-wide exclusive scan (util.cu) into another array, its scratch from S or of its own.
xk_status xk_exclusive_scan_i32(const int32_t* in, int32_t* out, long long n, int64_t* total_dev,
                                cudaStream_t s, XkScratch* S = nullptr);
// Number of block sums the scans use for n elements, and the int32 scan with a
// caller-provided block-sum array of bsum_cap words (same result, in place allowed;
// allocates nothing).
long long xk_scan_tiles(long long n);
xk_status xk_exclusive_scan_i32_scratch(const int32_t* in, int32_t* out, long long n, int64_t* total_dev,
                                        int64_t* bsum, long long bsum_cap, cudaStream_t s);
