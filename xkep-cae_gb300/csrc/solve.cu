// The Newton step's linear system on the device: LinearSolveProcess
// (xkep_cae/contact/solver/_newton_steps.py:338-366) solves K du = -R with the
// Dirichlet DOFs' rows and columns replaced by the identity by a sparse direct
// factorisation on the host.  Here the system stays where the assembly left it,
// K = K_beam (6x6 blocks over the nodes) + K_c (3x3 blocks over the nodes'
// translational DOFs), and is solved by BiCGStab with a block-Jacobi
// preconditioner (each node's 6x6 diagonal block, inverted once per matrix).
// Every reduction is a fixed-order two-pass sum (block partial sums in a fixed
// grid, then one block), so a solve gives the same bits run after run; the
// iteration's scalars stay in device memory, so a solve issues no host
// synchronisation until its convergence checks.
#include <math.h>

#include "xk_common.cuh"

namespace {

constexpr int SV_T = 256;
constexpr int SV_BLOCKS = 304;  // 2 x 152 SMs: the fixed grid of the two-pass reductions

template <typename T>
__global__ void k_spmv(xk_system A, const double* __restrict__ x, double* __restrict__ y) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= 6LL * A.n_nodes) return;
  const int v = (int)(g / 6), d = (int)(g % 6);
  if (A.fixed && A.fixed[g]) {  // Dirichlet row: identity
    y[g] = x[g];
    return;
  }
  const T* kb = (const T*)A.kb_vals;
  double acc = 0.0;
  // the stored blocks (u, v), u < v, transposed: row v's blocks left of the diagonal
  for (int q = A.kb_low_ptr[v]; q < A.kb_low_ptr[v + 1]; ++q) {
    const int b = A.kb_low_blk[q];
    const int u = A.kb_blk_row[b];
    const T* blk = kb + 36LL * b + d;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const long long col = 6LL * u + j;
      if (!(A.fixed && A.fixed[col])) acc = fma((double)blk[6 * j], x[col], acc);
    }
  }
  for (int b = A.kb_row_ptr[v]; b < A.kb_row_ptr[v + 1]; ++b) {
    const int w = A.kb_col[b];
    const T* blk = kb + 36LL * b + 6 * d;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const long long col = 6LL * w + j;
      if (!(A.fixed && A.fixed[col])) acc = fma((double)blk[j], x[col], acc);
    }
  }
  if (d < 3 && A.kc_vals) {
    const T* kc = (const T*)A.kc_vals;
    // the stored blocks (u, v), u < v, are also the blocks (v, u): row v's entries left of the diagonal
    for (int q = A.kc_low_ptr[v]; q < A.kc_low_ptr[v + 1]; ++q) {
      const int b = A.kc_low_blk[q];
      const int u = A.kc_blk_row[b];
      const T* blk = kc + 9LL * b + 3 * d;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const long long col = 6LL * u + j;
        if (!(A.fixed && A.fixed[col])) acc = fma((double)blk[j], x[col], acc);
      }
    }
    for (int b = A.kc_row_ptr[v]; b < A.kc_row_ptr[v + 1]; ++b) {
      const int w = A.kc_col[b];
      const T* blk = kc + 9LL * b + 3 * d;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const long long col = 6LL * w + j;
        if (!(A.fixed && A.fixed[col])) acc = fma((double)blk[j], x[col], acc);
      }
    }
  }
  y[g] = acc;
}

// inverse of each node's 6x6 diagonal block (K_beam's, plus K_c's translational one), Dirichlet DOFs
// as identity rows and columns; Gauss-Jordan with partial pivoting in double
template <typename T>
__global__ void k_block_jacobi(xk_system A, double* __restrict__ dinv) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= A.n_nodes) return;
  double M[6][12];
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 12; ++j) M[i][j] = (j - 6 == i) ? 1.0 : 0.0;
  const T* kb = (const T*)A.kb_vals;
  for (int b = A.kb_row_ptr[v]; b < A.kb_row_ptr[v + 1]; ++b)
    if (A.kb_col[b] == v)
      for (int i = 0; i < 6; ++i)
        for (int j = 0; j < 6; ++j) M[i][j] += (double)kb[36LL * b + 6 * i + j];
  if (A.kc_vals) {
    const T* kc = (const T*)A.kc_vals;
    for (int b = A.kc_row_ptr[v]; b < A.kc_row_ptr[v + 1]; ++b)
      if (A.kc_col[b] == v)
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j) M[i][j] += (double)kc[9LL * b + 3 * i + j];
  }
  if (A.fixed)
    for (int i = 0; i < 6; ++i)
      if (A.fixed[6LL * v + i])
        for (int j = 0; j < 6; ++j) {
          M[i][j] = (i == j) ? 1.0 : 0.0;
          M[j][i] = (i == j) ? 1.0 : 0.0;
        }
  for (int c = 0; c < 6; ++c) {
    int piv = c;
    for (int r = c + 1; r < 6; ++r)
      if (fabs(M[r][c]) > fabs(M[piv][c])) piv = r;
    if (piv != c)
      for (int j = 0; j < 12; ++j) {
        const double t = M[c][j];
        M[c][j] = M[piv][j];
        M[piv][j] = t;
      }
    const double p = M[c][c];
    const double ip = fabs(p) > 0.0 ? 1.0 / p : 0.0;  // a singular block leaves that part unpreconditioned
    for (int j = 0; j < 12; ++j) M[c][j] *= ip;
    for (int r = 0; r < 6; ++r)
      if (r != c) {
        const double f = M[r][c];
        for (int j = 0; j < 12; ++j) M[r][j] -= f * M[c][j];
      }
  }
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 6; ++j) dinv[36LL * v + 6 * i + j] = M[i][6 + j];
}

__global__ void k_apply_block_jacobi(int n_nodes, const double* __restrict__ dinv, const double* __restrict__ r,
                                     double* __restrict__ z) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= 6LL * n_nodes) return;
  const int v = (int)(g / 6), d = (int)(g % 6);
  const double* D = dinv + 36LL * v + 6 * d;
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < 6; ++j) acc = fma(D[j], r[6LL * v + j], acc);
  z[g] = acc;
}

// block partial sums of up to two dot products: part[2 b + k] = sum over the block's grid-stride share
__global__ void k_dot2(long long n, const double* __restrict__ a0, const double* __restrict__ b0,
                       const double* __restrict__ a1, const double* __restrict__ b1, double* __restrict__ part) {
  __shared__ double red[2][SV_T];
  double s0 = 0.0, s1 = 0.0;
  for (long long i = (long long)blockIdx.x * SV_T + threadIdx.x; i < n; i += (long long)SV_BLOCKS * SV_T) {
    s0 = fma(a0[i], b0[i], s0);
    if (a1) s1 = fma(a1[i], b1[i], s1);
  }
  red[0][threadIdx.x] = s0;
  red[1][threadIdx.x] = s1;
  __syncthreads();
  for (int w = SV_T / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[0][threadIdx.x] += red[0][threadIdx.x + w];
      red[1][threadIdx.x] += red[1][threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = red[0][0];
    part[2 * blockIdx.x + 1] = red[1][0];
  }
}

// BiCGStab's scalar updates from the dot results; sc holds
// [0] rho, [1] alpha, [2] omega, [3] beta, [4] scratch, [5] ||r||^2 (and the two sums of a k_dot2)
enum { S_RHO = 0, S_ALPHA, S_OMEGA, S_BETA, S_D0, S_D1, S_RR, S_BB, S_N };

__device__ void sum_parts(const double* __restrict__ part, double* out0, double* out1) {
  __shared__ double red[2][SV_T];
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < SV_BLOCKS; i += SV_T) {
    a += part[2 * i];
    b += part[2 * i + 1];
  }
  red[0][threadIdx.x] = a;
  red[1][threadIdx.x] = b;
  __syncthreads();
  for (int w = SV_T / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[0][threadIdx.x] += red[0][threadIdx.x + w];
      red[1][threadIdx.x] += red[1][threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *out0 = red[0][0];
    *out1 = red[1][0];
  }
}

// MODE 0: sc[D0], sc[D1] <- the two sums.  MODE 1 (after (rh, r)): beta = (rho_new / rho) (alpha / omega),
// rho = rho_new.  MODE 2 (after (rh, v)): alpha = rho / (rh, v).  MODE 3 (after (t, s), (t, t)):
// omega = (t, s) / (t, t).  MODE 4: ||r||^2 -> sc[RR].
template <int MODE>
__global__ void k_scalars(const double* __restrict__ part, double* __restrict__ sc) {
  __shared__ double d0, d1;
  sum_parts(part, &d0, &d1);
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (MODE == 0) {
    sc[S_D0] = d0;
    sc[S_D1] = d1;
  } else if (MODE == 1) {
    const double rho_new = d0;
    sc[S_BETA] = (sc[S_RHO] != 0.0 && sc[S_OMEGA] != 0.0) ? (rho_new / sc[S_RHO]) * (sc[S_ALPHA] / sc[S_OMEGA]) : 0.0;
    sc[S_RHO] = rho_new;
  } else if (MODE == 2) {
    sc[S_ALPHA] = d0 != 0.0 ? sc[S_RHO] / d0 : 0.0;
  } else if (MODE == 3) {
    sc[S_OMEGA] = d1 != 0.0 ? d0 / d1 : 0.0;
  } else {
    sc[S_RR] = d0;
  }
}

// p = r + beta (p - omega v)
__global__ void k_update_p(long long n, const double* __restrict__ r, const double* __restrict__ v,
                           double* __restrict__ p, const double* __restrict__ sc) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  p[i] = r[i] + sc[S_BETA] * (p[i] - sc[S_OMEGA] * v[i]);
}
// x += alpha y; s = r - alpha v
__global__ void k_update_xs(long long n, double* __restrict__ x, const double* __restrict__ y,
                            const double* __restrict__ r, const double* __restrict__ v, double* __restrict__ s,
                            const double* __restrict__ sc) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = sc[S_ALPHA];
  x[i] = fma(a, y[i], x[i]);
  s[i] = fma(-a, v[i], r[i]);
}
// x += omega z; r = s - omega t
__global__ void k_update_xr(long long n, double* __restrict__ x, const double* __restrict__ z,
                            const double* __restrict__ s, const double* __restrict__ t, double* __restrict__ r,
                            const double* __restrict__ sc) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double w = sc[S_OMEGA];
  x[i] = fma(w, z[i], x[i]);
  r[i] = fma(-w, t[i], s[i]);
}
// r = b - r (r holds A x on entry), rh = r, p = v = 0; scalars rho = alpha = omega = 1
__global__ void k_init(long long n, const double* __restrict__ b, double* __restrict__ r, double* __restrict__ rh,
                       double* __restrict__ p, double* __restrict__ v, double* __restrict__ sc) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    sc[S_RHO] = 1.0;
    sc[S_ALPHA] = 1.0;
    sc[S_OMEGA] = 1.0;
    sc[S_BETA] = 0.0;
  }
  if (i >= n) return;
  const double ri = b[i] - r[i];
  r[i] = ri;
  rh[i] = ri;
  p[i] = 0.0;
  v[i] = 0.0;
}

template <typename T>
xk_status spmv(const xk_system& A, const double* x, double* y, cudaStream_t st) {
  k_spmv<T><<<xk_blocks(6LL * A.n_nodes, SV_T), SV_T, 0, st>>>(A, x, y);
  return XK_OK;
}

xk_status spmv_any(const xk_system& A, const double* x, double* y, cudaStream_t st) {
  if (A.precision == XK_FP64) return spmv<double>(A, x, y, st);
  return spmv<float>(A, x, y, st);
}

xk_status dot2(long long n, const double* a0, const double* b0, const double* a1, const double* b1, double* part,
               cudaStream_t st) {
  k_dot2<<<SV_BLOCKS, SV_T, 0, st>>>(n, a0, b0, a1, b1, part);
  return XK_OK;
}

}  // namespace

static bool kc_complete(const xk_system* A) {
  return A->kb_blk_row && A->kb_low_ptr && A->kb_low_blk &&
         (!A->kc_vals || (A->kc_row_ptr && A->kc_col && A->kc_blk_row && A->kc_low_ptr && A->kc_low_blk));
}

extern "C" xk_status xk_system_spmv(const xk_system* A, const double* x, double* y, xk_stream s) {
  if (!A || !x || !y || !A->kb_row_ptr || !A->kb_col || !A->kb_vals || !kc_complete(A))
    return xk_set_error(XK_ERR_ARG, "xk_system_spmv: null argument");
  if (A->n_nodes <= 0) return XK_OK;
  spmv_any(*A, x, y, (cudaStream_t)s);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_system_block_jacobi(const xk_system* A, double* dinv, xk_stream s) {
  if (!A || !dinv || !A->kb_row_ptr || !A->kb_col || !A->kb_vals || !kc_complete(A))
    return xk_set_error(XK_ERR_ARG, "xk_system_block_jacobi: null argument");
  if (A->n_nodes <= 0) return XK_OK;
  if (A->precision == XK_FP64)
    k_block_jacobi<double><<<xk_blocks(A->n_nodes, 64), 64, 0, (cudaStream_t)s>>>(*A, dinv);
  else
    k_block_jacobi<float><<<xk_blocks(A->n_nodes, 64), 64, 0, (cudaStream_t)s>>>(*A, dinv);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

namespace {

// One BiCGStab iteration on stream st (scalars on the device).
void bicgstab_iteration(const xk_system& A, long long n, int nb, const double* dinv, double* x, double* r,
                        const double* rh, double* p, double* v, double* y, double* sv, double* z, double* t,
                        double* part, double* sc, cudaStream_t st) {
  dot2(n, rh, r, nullptr, nullptr, part, st);
  k_scalars<1><<<1, SV_T, 0, st>>>(part, sc);  // beta, rho
  k_update_p<<<nb, SV_T, 0, st>>>(n, r, v, p, sc);
  k_apply_block_jacobi<<<nb, SV_T, 0, st>>>(A.n_nodes, dinv, p, y);
  spmv_any(A, y, v, st);
  dot2(n, rh, v, nullptr, nullptr, part, st);
  k_scalars<2><<<1, SV_T, 0, st>>>(part, sc);  // alpha
  k_update_xs<<<nb, SV_T, 0, st>>>(n, x, y, r, v, sv, sc);
  k_apply_block_jacobi<<<nb, SV_T, 0, st>>>(A.n_nodes, dinv, sv, z);
  spmv_any(A, z, t, st);
  dot2(n, t, sv, t, t, part, st);
  k_scalars<3><<<1, SV_T, 0, st>>>(part, sc);  // omega
  k_update_xr<<<nb, SV_T, 0, st>>>(n, x, z, sv, t, r, sc);
}

// ||r||^2 into sc[S_RR]
void residual_sq(long long n, const double* r, double* part, double* sc, cudaStream_t st) {
  dot2(n, r, r, nullptr, nullptr, part, st);
  k_scalars<4><<<1, SV_T, 0, st>>>(part, sc);
}

// A private stream ordered after the caller's, and the graph of one check interval.  On every
// exit, an error return included, the stream is drained before it is destroyed, so that no
// kernel queued on it can still write x or the work vectors after xk_bicgstab has returned.
struct SolveStream {
  cudaStream_t cs = nullptr;
  cudaEvent_t ev = nullptr;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  ~SolveStream() {
    if (cs) cudaStreamSynchronize(cs);
    if (ge) cudaGraphExecDestroy(ge);
    if (g) cudaGraphDestroy(g);
    if (ev) cudaEventDestroy(ev);
    if (cs) cudaStreamDestroy(cs);
  }
};


// ---------------------------------------------------------------------------
// Small systems: the whole iteration in one thread-block cluster.
//
// The iteration above is 13 dependent launches, about 57 us however small the system.  Here 16 CTAs on 16
// SMs hold it together: the nodes are dealt out to the CTAs, a CTA keeps its rows of every vector in shared
// memory, and what the others need (the preconditioned vectors, the products of the dot products) goes through
// global memory between hardware cluster barriers.  A CTA's rows of the matrix are packed once into shared
// memory, without the fixed columns, where they fit.  The convergence checks run on the device: a solve is one
// launch per CL_SLICE iterations (so that no launch runs for long).  Every sum keeps the order of the launches above (a row's terms; 256
// consecutive products by the same tree, then the chunk sums by it), so x, the iteration count and the residual
// are the same bits.
// What bounds an iteration is the chain of dependent FP64 operations (68 clocks each): the longest row of the
// two products (some 120 terms for a core wire's node), then the sums' trees, three divides and the five
// barriers.  No more warps than rows need: a warp issues one FP64 instruction in 64 clocks, so further ones
// only repeat the scalar work (714 unknowns: 25 us an iteration with 16 warps, 21 us with four).  Writing the
// exchanged vectors into the other CTAs' shared memory instead measured the same.
// Line: CL_MAX_N unknowns.  us an iteration, launches against cluster (FP64 / float values): 714 unknowns 58 / 65
// against 21 / 22; 2,058: 62 / 76 against 27 / 27; 3,762: 62 / 73 against 40 / 47; beyond it the rows no longer
// fit shared memory and 16 SMs are too few: 5,550: 62 / 73 against 62 / 66, 7,326: 62 / 73 against 64 / 69.
// ---------------------------------------------------------------------------
constexpr int CL = 16, CL_SLICE = 512;
constexpr int CL_MAX_N = 4032;  // 252 rows a CTA, and below 32 chunks of 256
constexpr int CL_SMEM = 225 * 1024;
constexpr int CL_B = 8;  // terms loaded ahead of their operations; packed rows are padded to a multiple

XK_D void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// The tree of k_dot2 over 256 values (index t + w added to t for w = 128 ... 1) by one warp: y[k] of lane l is
// value l + 32 k.  The sum is in lane 0.
XK_D double warp_tree256(double* y) {
#pragma unroll
  for (int k = 0; k < 4; ++k) y[k] += y[k + 4];
  y[0] += y[2];
  y[1] += y[3];
  double x = y[0] + y[1];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}

struct ClusterSolve {
  const double* b;
  double* x;
  const double* dinv;
  double* work;  // 8 vectors, the chunk sums (not used here), the scalars
  double rtol;
  int start, it0, it1, max_iter, interval;
};

template <typename T, int CL_T>
__global__ void __launch_bounds__(CL_T, 1) k_bicgstab_cluster(const __grid_constant__ xk_system A,
                                                              const __grid_constant__ ClusterSolve a) {
  constexpr int CL_WARPS = CL_T / 32;
  extern __shared__ double sm[];
  __shared__ double s_part[2][32], s_sum[2];
  __shared__ int s_max[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = blockIdx.x;
  const int nn = A.n_nodes, n = 6 * nn;
  const int npc = (nn + CL - 1) / CL;  // nodes per CTA
  const int v0 = rank * npc < nn ? rank * npc : nn, nv = (v0 + npc < nn ? v0 + npc : nn) - v0;
  const int R = 6 * nv, g0 = 6 * v0, RS = 6 * npc;
  // this CTA's rows
  double *r = sm, *rh = r + RS, *p = rh + RS, *v = p + RS, *sv = v + RS, *t = sv + RS, *x = t + RS, *y = x + RS;
  double* dinv = y + RS;         // [6 RS]
  double* full = dinv + 6 * RS;  // [n + 1] the vector that the rows are multiplied with, then a zero
  uint8_t* fx = reinterpret_cast<uint8_t*>(full + n + 1);
  double* const vals = full + n + 1 + (n + 7) / 8;
  double* const W = a.work;
  // exchanged through global memory; each is written again only after a barrier that its readers have passed
  double *gy = W + 4LL * n, *gz = W + 6LL * n, *P0 = W + 5LL * n, *P1 = W + 7LL * n, *P2 = W + 3LL * n, *P3 = W;
  double* const sc = W + 8LL * n + 2 * SV_BLOCKS;
  const int chunks = (n + SV_T - 1) / SV_T;
  int half = 1;  // half the power of two that holds the chunks
  while (2 * half < chunks) half *= 2;
  for (int i = tid; i < n; i += CL_T) fx[i] = A.fixed ? A.fixed[i] : 0;
  for (int i = tid; i < 6 * R; i += CL_T) dinv[i] = a.dinv[6LL * g0 + i];
  if (tid < 2) s_max[tid] = 0;
  if (tid == 0) full[n] = 0.0;
  __syncthreads();

  // row i of this CTA: the translational rows first (they also carry K_c), so that a warp's rows are alike
  const int nt = 3 * nv;
  auto row_of = [&](int i) { return i < nt ? 6 * (i / 3) + i % 3 : 6 * ((i - nt) / 3) + 3 + (i - nt) % 3; };
  // the terms of k_spmv's row in its order: f(value, column) for every column that is not fixed
  auto walk = [&](int row, auto f) {
    const int w = (g0 + row) / 6, d = (g0 + row) % 6;
    const T* kb = (const T*)A.kb_vals;
    for (int q = A.kb_low_ptr[w]; q < A.kb_low_ptr[w + 1]; ++q) {
      const int bk = A.kb_low_blk[q], c = 6 * A.kb_blk_row[bk];
#pragma unroll
      for (int j = 0; j < 6; ++j)
        if (!fx[c + j]) f(kb[36LL * bk + d + 6 * j], c + j);
    }
    for (int bk = A.kb_row_ptr[w]; bk < A.kb_row_ptr[w + 1]; ++bk) {
      const int c = 6 * A.kb_col[bk];
#pragma unroll
      for (int j = 0; j < 6; ++j)
        if (!fx[c + j]) f(kb[36LL * bk + 6 * d + j], c + j);
    }
    if (d < 3 && A.kc_vals) {
      const T* kc = (const T*)A.kc_vals;
      for (int q = A.kc_low_ptr[w]; q < A.kc_low_ptr[w + 1]; ++q) {
        const int bk = A.kc_low_blk[q], c = 6 * A.kc_blk_row[bk];
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (!fx[c + j]) f(kc[9LL * bk + 3 * d + j], c + j);
      }
      for (int bk = A.kc_row_ptr[w]; bk < A.kc_row_ptr[w + 1]; ++bk) {
        const int c = 6 * A.kc_col[bk];
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (!fx[c + j]) f(kc[9LL * bk + 3 * d + j], c + j);
      }
    }
  };
  // Packed rows: a panel of the rotational rows and one of the translational rows, each padded to its longest
  // row with zero times the zero past the vector; term e of a panel's row i at e * nt + i.  A panel that does not
  // fit is read from the block matrices instead.
  for (int i = tid; i < R; i += CL_T) {
    int e = 0;
    if (!fx[g0 + row_of(i)]) walk(row_of(i), [&](T, int) { ++e; });
    atomicMax(&s_max[i < nt ? 1 : 0], e);
  }
  __syncthreads();
  const long long room = (CL_SMEM - (reinterpret_cast<char*>(vals) - reinterpret_cast<char*>(sm))) / 10 - 8;
  const int len_r = (s_max[0] + CL_B - 1) / CL_B * CL_B, len_t = (s_max[1] + CL_B - 1) / CL_B * CL_B;
  const bool pack_r = (long long)len_r * nt <= room, pack_t = pack_r && (long long)(len_r + len_t) * nt <= room;
  uint16_t* const cols = reinterpret_cast<uint16_t*>(vals + (pack_r ? (long long)(len_r + (pack_t ? len_t : 0)) * nt : 0));
  for (int i = tid; i < R; i += CL_T) {
    const bool tr = i < nt;
    if (tr ? !pack_t : !pack_r) continue;
    const int at = tr ? len_r * nt + i : i - nt, len = tr ? len_t : len_r;
    int e = 0;
    if (!fx[g0 + row_of(i)])
      walk(row_of(i), [&](T val, int c) {
        vals[at + e * nt] = (double)val;
        cols[at + e * nt] = (uint16_t)c;
        ++e;
      });
    for (; e < len; ++e) {
      vals[at + e * nt] = 0.0;
      cols[at + e * nt] = (uint16_t)n;
    }
  }
  __syncthreads();

  auto matvec = [&](int i, int row) {
    if (fx[g0 + row]) return full[g0 + row];
    double acc = 0.0;
    const bool tr = i < nt;
    if (tr ? pack_t : pack_r) {
      const double* z = vals + (tr ? len_r * nt + i : i - nt);
      const uint16_t* c = cols + (z - vals);
      const int len = tr ? len_t : len_r;
      double z0[CL_B], w0[CL_B];
      if (len > 0) {
#pragma unroll
        for (int j = 0; j < CL_B; ++j) {
          z0[j] = z[j * nt];
          w0[j] = full[c[j * nt]];
        }
      }
      for (int e = CL_B; e <= len; e += CL_B) {  // the next terms are on their way while these are added
        double z1[CL_B], w1[CL_B];
        z += CL_B * nt;
        c += CL_B * nt;
        if (e < len) {
#pragma unroll
          for (int j = 0; j < CL_B; ++j) {
            z1[j] = z[j * nt];
            w1[j] = full[c[j * nt]];
          }
        }
#pragma unroll
        for (int j = 0; j < CL_B; ++j) acc = fma(z0[j], w0[j], acc);
#pragma unroll
        for (int j = 0; j < CL_B; ++j) {
          z0[j] = z1[j];
          w0[j] = w1[j];
        }
      }
    } else {
      walk(row, [&](T val, int col) { acc = fma((double)val, full[col], acc); });
    }
    return acc;
  };
  auto precondition = [&](const double* src, int row) {  // k_apply_block_jacobi
    const double* D = dinv + 6 * row;
    const double* s = src + 6 * (row / 6);
    double acc = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) acc = fma(D[j], s[j], acc);
    return acc;
  };
  auto fetch = [&](const double* src) {
    for (int i = tid; i < n; i += CL_T) full[i] = __ldcg(src + i);
    __syncthreads();
  };
  // the sums of one or two exchanged product vectors, in every CTA the same bits
  auto sums = [&](const double* Pa, const double* Pb, double& sa, double& sb) {
    const int k = Pb ? 2 : 1;
    for (int c = warp; c < chunks * k; c += CL_WARPS) {
      const double* P = c < chunks ? Pa : Pb;
      const int q = c < chunks ? c : c - chunks;
      double z[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = SV_T * q + lane + 32 * j;
        z[j] = i < n ? __ldcg(P + i) : 0.0;
      }
      const double s = warp_tree256(z);
      if (lane == 0) s_part[c < chunks ? 0 : 1][q] = s;
    }
    __syncthreads();
    if (warp < k) {  // the tree of sum_parts without its zeros
      double s = lane < chunks ? s_part[warp][lane] : 0.0;
      for (int o = half; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) s_sum[warp] = s;
    }
    __syncthreads();
    sa = s_sum[0];
    if (Pb) sb = s_sum[1];
  };

  double rho, alpha, omega, rho_next, bb, rr = 0.0, unused;
  if (a.start) {
    for (int i = tid; i < n; i += CL_T) full[i] = a.x[i];
    __syncthreads();
    for (int i = tid; i < R; i += CL_T) {
      const int row = row_of(i), g = g0 + row;
      const double ri = a.b[g] - matvec(i, row);
      r[row] = ri;
      rh[row] = ri;
      p[row] = 0.0;
      v[row] = 0.0;
      x[row] = full[g];
      P0[g] = ri * ri;
      P1[g] = a.b[g] * a.b[g];
    }
    cluster_sync();
    sums(P0, P1, rho_next, bb);
    bb = bb > 0.0 ? bb : 1.0;
    rho = alpha = omega = 1.0;
  } else {
    rho = sc[0];
    alpha = sc[1];
    omega = sc[2];
    rho_next = sc[3];
    bb = sc[4];
    for (int row = tid; row < R; row += CL_T) {
      const int g = g0 + row;
      r[row] = W[g];
      rh[row] = W[1LL * n + g];
      p[row] = W[2LL * n + g];
      v[row] = W[3LL * n + g];
      x[row] = a.x[g];
    }
  }
  cluster_sync();  // the state and the first products have been read by all
  double ao = div64(alpha, omega);
  int it = a.it0;
  while (it < a.it1) {
    const int k = a.max_iter - it < a.interval ? a.max_iter - it : a.interval;
    for (int q = 0; q < k; ++q) {
      const double beta = (rho != 0.0 && omega != 0.0) ? div64(rho_next, rho) * ao : 0.0;
      rho = rho_next;
      for (int row = tid; row < R; row += CL_T) p[row] = r[row] + beta * (p[row] - omega * v[row]);
      __syncthreads();
      for (int row = tid; row < R; row += CL_T) gy[g0 + row] = y[row] = precondition(p, row);
      cluster_sync();
      fetch(gy);
      for (int i = tid; i < R; i += CL_T) {
        const int row = row_of(i);
        const double z = matvec(i, row);
        v[row] = z;
        P0[g0 + row] = rh[row] * z;
      }
      cluster_sync();
      double d0, d1 = 0.0;
      sums(P0, nullptr, d0, unused);
      alpha = d0 != 0.0 ? div64(rho, d0) : 0.0;
      for (int row = tid; row < R; row += CL_T) {
        x[row] = fma(alpha, y[row], x[row]);
        sv[row] = fma(-alpha, v[row], r[row]);
      }
      __syncthreads();
      for (int row = tid; row < R; row += CL_T) gz[g0 + row] = y[row] = precondition(sv, row);
      cluster_sync();
      fetch(gz);
      for (int i = tid; i < R; i += CL_T) {
        const int row = row_of(i);
        const double z = matvec(i, row);
        t[row] = z;
        P0[g0 + row] = z * sv[row];
        P1[g0 + row] = z * z;
      }
      cluster_sync();
      sums(P0, P1, d0, d1);
      omega = d1 != 0.0 ? div64(d0, d1) : 0.0;
      const bool check = q == k - 1;
      for (int row = tid; row < R; row += CL_T) {
        x[row] = fma(omega, y[row], x[row]);
        const double ri = fma(-omega, t[row], sv[row]);
        r[row] = ri;
        P2[g0 + row] = rh[row] * ri;
        if (check) P3[g0 + row] = ri * ri;
      }
      cluster_sync();
      ao = div64(alpha, omega);
      sums(P2, check ? P3 : nullptr, rho_next, rr);
    }
    it += k;
    if (!(sqrt(rr / bb) > a.rtol)) break;  // converged (or a NaN): the same in every CTA
  }
  cluster_sync();  // the last sums have been read by all before the state goes out
  for (int row = tid; row < R; row += CL_T) {
    const int g = g0 + row;
    W[g] = r[row];
    W[1LL * n + g] = rh[row];
    W[2LL * n + g] = p[row];
    W[3LL * n + g] = v[row];
    a.x[g] = x[row];
  }
  if (rank == 0 && tid == 0) {
    sc[0] = rho;
    sc[1] = alpha;
    sc[2] = omega;
    sc[3] = rho_next;
    sc[4] = bb;
    sc[5] = rr;
    sc[6] = (double)it;
  }
}

// One slice of a solve; false where a cluster of this size cannot be launched here.
template <typename T, int CL_T>
bool cluster_slice(const xk_system& A, const ClusterSolve& a, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CL);
  cfg.blockDim = dim3(CL_T);
  cfg.dynamicSmemBytes = CL_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int resident = 0;
  const auto kernel = k_bicgstab_cluster<T, CL_T>;
  if ((a.start &&
       (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&resident, kernel, &cfg) != cudaSuccess || resident < 1)) ||
      cudaLaunchKernelEx(&cfg, kernel, A, a) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

// a thread per row
template <typename T>
bool cluster_slice_any(const xk_system& A, const ClusterSolve& a, cudaStream_t st) {
  const int rows = 6 * ((A.n_nodes + CL - 1) / CL);
  return rows <= 128 ? cluster_slice<T, 128>(A, a, st) : cluster_slice<T, 256>(A, a, st);
}

}  // namespace

extern "C" xk_status xk_bicgstab(const xk_system* A, const double* b, double* x, const double* dinv, double* work,
                                 int32_t max_iter, int32_t check_every, double rtol, int32_t* iters, double* rel_res,
                                 xk_stream s) {
  if (!A || !b || !x || !dinv || !work || max_iter < 0 || check_every < 1 || !A->kb_row_ptr || !A->kb_col ||
      !A->kb_vals || !kc_complete(A))
    return xk_set_error(XK_ERR_ARG, "xk_bicgstab: bad arguments");
  cudaStream_t st = (cudaStream_t)s;
  const long long n = 6LL * A->n_nodes;
  if (iters) *iters = 0;
  if (rel_res) *rel_res = 0.0;
  if (n == 0) return XK_OK;
  double* r = work;
  double* rh = r + n;
  double* p = rh + n;
  double* v = p + n;
  double* y = v + n;
  double* sv = y + n;
  double* z = sv + n;
  double* t = z + n;
  double* part = t + n;          // [2 * SV_BLOCKS]
  double* sc = part + 2 * SV_BLOCKS;  // [S_N]
  const int nb = xk_blocks(n, SV_T);
  const int interval = check_every < max_iter ? check_every : (max_iter > 0 ? max_iter : 1);
  if (n <= CL_MAX_N && max_iter > 0) {  // one launch per slice of whole check intervals
    ClusterSolve a{b, x, dinv, work, rtol, 1, 0, 0, max_iter, interval};
    const int slice = interval * (interval < CL_SLICE ? CL_SLICE / interval : 1);
    while (true) {
      a.it1 = max_iter - a.it0 < slice ? max_iter : a.it0 + slice;
      if (!(A->precision == XK_FP64 ? cluster_slice_any<double>(*A, a, st) : cluster_slice_any<float>(*A, a, st))) {
        if (a.start) break;  // no such cluster here: the launches below
        return xk_set_error(XK_ERR_CUDA, "xk_bicgstab: cluster launch failed");
      }
      double h[7];
      XK_CUDA(cudaMemcpyAsync(h, sc, sizeof(h), cudaMemcpyDeviceToHost, st));
      XK_CUDA(cudaStreamSynchronize(st));
      a.it0 = (int)h[6];
      a.start = 0;
      const double res_c = sqrt(h[5] / h[4]);
      if (iters) *iters = a.it0;
      if (rel_res) *rel_res = res_c;
      if (a.it0 >= max_iter || !(res_c > rtol)) return XK_OK;
    }
  }
  // ||b||^2 and r = b - A x
  dot2(n, b, b, nullptr, nullptr, part, st);
  k_scalars<0><<<1, SV_T, 0, st>>>(part, sc);
  double bb_rr[2];
  XK_CUDA(cudaMemcpyAsync(bb_rr, sc + S_D0, sizeof(double), cudaMemcpyDeviceToHost, st));
  spmv_any(*A, x, r, st);
  k_init<<<nb, SV_T, 0, st>>>(n, b, r, rh, p, v, sc);
  XK_CHECK_LAUNCH();
  XK_CUDA(cudaStreamSynchronize(st));
  const double bb = bb_rr[0] > 0.0 ? bb_rr[0] : 1.0;
  int it = 0;
  double res = 1.0;
  // every check interval (check_every iterations and the residual norm) is one CUDA graph, captured on
  // a private stream; if capture is not possible the same kernels are launched one by one
  SolveStream ss;
  XK_CUDA(cudaStreamCreateWithFlags(&ss.cs, cudaStreamNonBlocking));
  XK_CUDA(cudaEventCreateWithFlags(&ss.ev, cudaEventDisableTiming));
  XK_CUDA(cudaEventRecord(ss.ev, st));
  XK_CUDA(cudaStreamWaitEvent(ss.cs, ss.ev, 0));
  auto chunk = [&](int k, cudaStream_t cs) {
    for (int q = 0; q < k; ++q) bicgstab_iteration(*A, n, nb, dinv, x, r, rh, p, v, y, sv, z, t, part, sc, cs);
    residual_sq(n, r, part, sc, cs);
  };
  if (max_iter >= interval &&
      cudaStreamBeginCapture(ss.cs, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
    chunk(interval, ss.cs);
    if (cudaStreamEndCapture(ss.cs, &ss.g) != cudaSuccess ||
        cudaGraphInstantiate(&ss.ge, ss.g, 0) != cudaSuccess) {
      ss.ge = nullptr;
      cudaGetLastError();  // capture not possible here: launch one by one
    }
  } else {
    cudaGetLastError();
  }
  while (it < max_iter) {
    const int k = (max_iter - it) < interval ? (max_iter - it) : interval;
    if (ss.ge && k == interval) XK_CUDA(cudaGraphLaunch(ss.ge, ss.cs));
    else chunk(k, ss.cs);
    XK_CHECK_LAUNCH();
    it += k;
    double rr = 0.0;
    XK_CUDA(cudaMemcpyAsync(&rr, sc + S_RR, sizeof(double), cudaMemcpyDeviceToHost, ss.cs));
    XK_CUDA(cudaStreamSynchronize(ss.cs));
    res = sqrt(rr / bb);
    if (!(res > rtol)) break;  // converged (or a NaN, reported through rel_res)
  }
  XK_CUDA(cudaEventRecord(ss.ev, ss.cs));
  XK_CUDA(cudaStreamWaitEvent(st, ss.ev, 0));  // the caller's stream sees x
  if (iters) *iters = it;
  if (rel_res) *rel_res = res;
  return XK_OK;
}

// ---------------------------------------------------------------------------
// The system as dense blocks of a block-tridiagonal matrix, for a direct solve
// on the device.  Nodes are renumbered by pos[] (an ordering along the strand
// axis) and grouped bn to a block; a row of DOFs of node v, DOF d sits in
// block row I = pos[v] / bn at local row 6 (pos[v] % bn) + d.  One thread per
// DOF row writes every entry of its row (K_beam's blocks, then K_c's added on
// the translational part, the mass term on the diagonal), so no entry has two
// writers.  Dirichlet rows and columns become the identity.  A coupling more
// than one block row away cannot be stored: it sets *overflow.
namespace {

template <typename T>
__global__ void k_blocktri(xk_system A, const int32_t* __restrict__ pos, int bn, int nb,
                           const double* __restrict__ mass, double mass_coef, double* __restrict__ D,
                           double* __restrict__ Lo, double* __restrict__ Up, int32_t* __restrict__ overflow) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= 6LL * A.n_nodes) return;
  const int v = (int)(g / 6), d = (int)(g % 6);
  const long long b = 6LL * bn;
  const int pv = pos[v];
  const int I = pv / bn;
  const long long r = 6LL * (pv % bn) + d;
  const long long row_off = (long long)I * b * b + r * b;
  auto at = [&](int w, int j) -> double* {
    const int pw = pos[w];
    const int J = pw / bn;
    const long long c = 6LL * (pw % bn) + j;
    if (J == I) return D + row_off + c;
    if (J == I - 1) return Lo + row_off + c;
    if (J == I + 1) return Up + row_off + c;
    return nullptr;
  };
  if (A.fixed && A.fixed[g]) {  // Dirichlet row: identity (the rest of the row stays zero)
    D[row_off + 6LL * (pv % bn) + d] = 1.0;
    return;
  }
  bool lost = false;
  const T* kb = (const T*)A.kb_vals;
  for (int q = A.kb_low_ptr[v]; q < A.kb_low_ptr[v + 1]; ++q) {  // stored (u, v), u < v, transposed
    const int bk = A.kb_low_blk[q];
    const int u = A.kb_blk_row[bk];
    const T* blk = kb + 36LL * bk + d;
    for (int j = 0; j < 6; ++j) {
      if (A.fixed && A.fixed[6LL * u + j]) continue;
      double* p = at(u, j);
      if (p) *p += (double)blk[6 * j];
      else lost = true;
    }
  }
  for (int bk = A.kb_row_ptr[v]; bk < A.kb_row_ptr[v + 1]; ++bk) {
    const int w = A.kb_col[bk];
    const T* blk = kb + 36LL * bk + 6 * d;
    for (int j = 0; j < 6; ++j) {
      if (A.fixed && A.fixed[6LL * w + j]) continue;
      double* p = at(w, j);
      if (p) *p += (double)blk[j];
      else lost = true;
    }
  }
  if (d < 3 && A.kc_vals) {
    const T* kc = (const T*)A.kc_vals;
    for (int q = A.kc_low_ptr[v]; q < A.kc_low_ptr[v + 1]; ++q) {  // stored (u, v), u < v, also (v, u)
      const int bk = A.kc_low_blk[q];
      const int u = A.kc_blk_row[bk];
      const T* blk = kc + 9LL * bk + 3 * d;
      for (int j = 0; j < 3; ++j) {
        if (A.fixed && A.fixed[6LL * u + j]) continue;
        double* p = at(u, j);
        if (p) *p += (double)blk[j];
        else lost = true;
      }
    }
    for (int bk = A.kc_row_ptr[v]; bk < A.kc_row_ptr[v + 1]; ++bk) {
      const int w = A.kc_col[bk];
      const T* blk = kc + 9LL * bk + 3 * d;
      for (int j = 0; j < 3; ++j) {
        if (A.fixed && A.fixed[6LL * w + j]) continue;
        double* p = at(w, j);
        if (p) *p += (double)blk[j];
        else lost = true;
      }
    }
  }
  if (mass) D[row_off + 6LL * (pv % bn) + d] += mass_coef * mass[g];
  if (lost) atomicExch(overflow, 1);
}

}  // namespace

extern "C" xk_status xk_system_blocktri(const xk_system* A, const int32_t* pos, int32_t bn, int32_t nb,
                                        const double* mass, double mass_coef, double* D, double* Lo, double* Up,
                                        int32_t* overflow, xk_stream s) {
  if (!A || !pos || bn < 1 || nb < 1 || !D || !Lo || !Up || !overflow || !A->kb_row_ptr || !A->kb_col ||
      !A->kb_vals || !kc_complete(A) || (long long)bn * nb < A->n_nodes)
    return xk_set_error(XK_ERR_ARG, "xk_system_blocktri: bad arguments");
  cudaStream_t st = (cudaStream_t)s;
  const long long b = 6LL * bn;
  const size_t bytes = (size_t)nb * b * b * sizeof(double);
  XK_CUDA(cudaMemsetAsync(D, 0, bytes, st));
  XK_CUDA(cudaMemsetAsync(Lo, 0, bytes, st));
  XK_CUDA(cudaMemsetAsync(Up, 0, bytes, st));
  XK_CUDA(cudaMemsetAsync(overflow, 0, sizeof(int32_t), st));
  if (A->n_nodes == 0) return XK_OK;
  const int nbk = xk_blocks(6LL * A->n_nodes, SV_T);
  if (A->precision == XK_FP64)
    k_blocktri<double><<<nbk, SV_T, 0, st>>>(*A, pos, bn, nb, mass, mass_coef, D, Lo, Up, overflow);
  else
    k_blocktri<float><<<nbk, SV_T, 0, st>>>(*A, pos, bn, nb, mass, mass_coef, D, Lo, Up, overflow);
  XK_CHECK_LAUNCH();
  return XK_OK;
}
