// One-pass exclusive scan with decoupled look-back (Merrill and Garland, "Single-pass Parallel Prefix Scan with
// Decoupled Look-back", NVIDIA technical report NVR-2016-002), over whatever an operation loads and into whatever
// it stores, so that a flag, its scan and the compaction by it are one kernel.
//
// Tiles take their index from a ticket
// counter in the order they start, so a tile waits only on tiles that are already running and never on a
// later one.  Each tile publishes its aggregate (flag 1); the first warp then looks back over a window of
// 32 predecessors at a time (one flag per lane, ballots to find the nearest inclusive prefix, flag 2, and
// any predecessor that has not published), adds the window's aggregates up to that prefix with a warp sum,
// and publishes the tile's inclusive prefix.  The wait on a predecessor that has not published yet is
// bounded: past SPIN polls the tile sums the inputs before it itself (the same prefix: integer
// sums do not depend on their order), so the result never depends on the wait.  Earlier tiles may have stored by
// then: what an operation stores must not be what its one() reads.
//
// One launch runs up to SCAN_CHANNELS independent scans (blockIdx.y).  An operation has, per channel c,
//   long long size(int c) const                      how many values
//   int64_t one(int c, long long i) const            the value at i < size
//   void eight(int c, long long i, int64_t* v) const the values at i ... i + 7, all below size
//   void store(int c, long long i, int n, int64_t prefix, const int64_t* v) const
//                                                    n values from i on, prefix = the sum before i
//   void total(int c, int64_t sum) const
#pragma once

#include "xk_common.cuh"

constexpr int SCAN_T = 256;
constexpr int SCAN_I = 8;
constexpr int SCAN_TILE = SCAN_T * SCAN_I;
constexpr int SCAN_SPIN_LIMIT = 1 << 20;
constexpr int SCAN_CHANNELS = 2;

template <typename T>
__device__ T block_exclusive_scan(T v, T* warp_tot, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = (lane < (SCAN_T / 32)) ? warp_tot[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < (SCAN_T / 32)) warp_tot[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  T before = (warp > 0) ? warp_tot[warp - 1] : T(0);
  if (total) *total = warp_tot[SCAN_T / 32 - 1];
  return before + x - v;
}

XK_D int scan_flag(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

template <typename Op, int SPIN>
__global__ void __launch_bounds__(SCAN_T) k_scan_onepass(const __grid_constant__ Op op, long long nb_max,
                                                         int64_t* __restrict__ sums, int* __restrict__ words) {
  __shared__ int64_t wt[SCAN_T / 32];
  __shared__ long long s_tile;
  __shared__ int64_t s_prefix;
  __shared__ int s_fallback;
  const int c = blockIdx.y;
  const long long n = op.size(c), nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  int64_t* agg = sums + 2 * nb_max * c;
  int64_t* inc = agg + nb_max;
  int* flag = words + (nb_max + 1) * c;
  if (threadIdx.x == 0) {
    s_tile = (long long)atomicAdd(reinterpret_cast<unsigned*>(flag + nb_max), 1u);
    s_fallback = 0;
  }
  __syncthreads();
  const long long t = s_tile;
  if (t >= nb) {  // the longer channel has more tiles
    if (n == 0 && t == 0 && threadIdx.x == 0) op.total(c, 0);
    return;
  }
  const long long base = t * SCAN_TILE + (long long)threadIdx.x * SCAN_I;
  int64_t loc[SCAN_I];
  if (base + SCAN_I <= n) {
    op.eight(c, base, loc);
  } else {
#pragma unroll
    for (int i = 0; i < SCAN_I; ++i) loc[i] = (base + i < n) ? op.one(c, base + i) : 0;
  }
  int64_t s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_I; ++i) s += loc[i];
  int64_t tile_tot;
  int64_t ex = block_exclusive_scan<int64_t>(s, wt, &tile_tot);
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (t == 0) {
      if (lane == 0) {
        inc[0] = tile_tot;
        __threadfence();
        atomicExch(&flag[0], 2);
        s_prefix = 0;
      }
    } else {
      if (lane == 0) {
        agg[t] = tile_tot;
        __threadfence();
        atomicExch(&flag[t], 1);
      }
      int64_t p = 0;
      long long j = t - 1;  // the window covers tiles j, j - 1, ..., j - 31 (lane k: tile j - k)
      int spins = 0;
      bool fell_back = false;
      while (true) {
        const long long k = j - lane;
        const int f = k >= 0 ? scan_flag(flag + k) : 2;  // before tile 0: an inclusive prefix of 0
        const unsigned m_inc = __ballot_sync(0xffffffffu, f == 2);
        const int stop = m_inc ? __ffs(m_inc) - 1 : 32;  // nearest inclusive prefix in the window
        const unsigned need = stop == 32 ? 0xffffffffu : ((1u << stop) - 1u);
        if (__ballot_sync(0xffffffffu, f == 0) & need) {  // a nearer predecessor has not published
          if (++spins > SPIN) {
            fell_back = true;
            break;
          }
          continue;
        }
        __threadfence();
        // published values are read past L1 (other tiles' lines may sit there stale)
        int64_t v = 0;
        if (k >= 0) {
          if (lane < stop) v = __ldcg(agg + k);
          else if (lane == stop) v = __ldcg(inc + k);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        p += v;
        if (stop < 32) break;
        j -= 32;
      }
      if (lane == 0) {
        if (fell_back) {
          s_fallback = 1;
        } else {
          inc[t] = p + tile_tot;
          __threadfence();
          atomicExch(&flag[t], 2);
          s_prefix = p;
        }
      }
    }
  }
  __syncthreads();
  if (s_fallback) {  // the prefix from the inputs before this tile
    int64_t q = 0;
    for (long long k = threadIdx.x; k < t * SCAN_TILE; k += SCAN_T) q += op.one(c, k);
    int64_t all;
    block_exclusive_scan<int64_t>(q, wt, &all);
    if (threadIdx.x == 0) {
      s_prefix = all;
      inc[t] = all + tile_tot;
      __threadfence();
      atomicExch(&flag[t], 2);
    }
    __syncthreads();
  }
  if (base < n) op.store(c, base, n - base < SCAN_I ? (int)(n - base) : SCAN_I, ex + s_prefix, loc);
  if (t == nb - 1 && threadIdx.x == 0) op.total(c, s_prefix + tile_tot);
}

// int32 array in, exclusive prefixes out (another array); *sum (nullable) = the sum of all
struct ScanI32 {
  const int32_t* in;
  int32_t* out;
  long long n;
  int64_t* sum;
  XK_D long long size(int) const { return n; }
  XK_D int64_t one(int, long long i) const { return in[i]; }
  XK_D void eight(int, long long i, int64_t* v) const {
    if ((reinterpret_cast<uintptr_t>(in + i) & 15) == 0) {  // two vector loads
      const int4* q = reinterpret_cast<const int4*>(in + i);
      const int4 x = q[0], y = q[1];
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
      v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
      return;
    }
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) v[k] = in[i + k];
  }
  XK_D void store(int, long long i, int k, int64_t prefix, const int64_t* v) const {
#pragma unroll
    for (int j = 0; j < SCAN_I; ++j) {
      if (j < k) out[i + j] = (int32_t)prefix;
      prefix += v[j];
    }
  }
  XK_D void total(int, int64_t s) const {
    if (sum) *sum = s;
  }
};

// The words of one launch, for scans of at most n values: sums, and words that are zero at its start.
inline long long scan_tiles(long long n) { return (n + SCAN_TILE - 1) / SCAN_TILE; }
inline long long scan_sums(long long n, int channels) { return 2 * scan_tiles(n) * channels; }
inline long long scan_words(long long n, int channels) { return (scan_tiles(n) + 1) * channels; }

// n = the longest channel's size (> 0).
template <typename Op, int SPIN = SCAN_SPIN_LIMIT>
xk_status scan_launch(const Op& op, long long n, int channels, int64_t* sums, int* zeroed_words, cudaStream_t s) {
  const long long nb = scan_tiles(n);
  k_scan_onepass<Op, SPIN><<<dim3((unsigned)nb, channels), SCAN_T, 0, s>>>(op, nb, sums, zeroed_words);
  XK_CHECK_LAUNCH();
  return XK_OK;
}
