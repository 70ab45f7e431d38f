// Learned pruning of broadphase candidate pairs: per-candidate features, a
// small MLP (F = 8 inputs -> 64 -> 64 -> 64 -> 1, ReLU, BF16 weights and
// activations, FP32 accumulation), its training kernels (forward with stored
// activations, backward, deterministic weight-gradient reduction, Adam) and the
// selection / pair-table compaction that apply it at detection time.
//
// Inference runs on the tensor cores, in two forms: tcgen05.mma with the
// activations and accumulators in TMEM, five tiles of 128 candidates per SM (the default), and
// mma.sync m16n8k16 (BF16 -> FP32), where a warp takes 16 candidates and each
// layer's accumulator fragments are re-packed in registers as the next layer's
// A operand.  Training runs
// in FP32 register tiles on BF16-rounded operands, which is the same
// arithmetic up to the order of the float sums.
#include <cuda_bf16.h>

#include "xk_common.cuh"

namespace {

constexpr int MF = XK_MLP_IN, MH = XK_MLP_HIDDEN, NP = XK_MLP_PARAMS, NA = XK_MLP_ACT;
constexpr int O_W1 = 0, O_B1 = O_W1 + MH * MF, O_W2 = O_B1 + MH, O_B2 = O_W2 + MH * MH, O_W3 = O_B2 + MH,
              O_B3 = O_W3 + MH * MH, O_W4 = O_B3 + MH, O_B4 = O_W4 + MH;
static_assert(O_B4 + 1 == NP, "parameter layout");
static_assert(NA == 3 * MH, "activation layout");

XK_D float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

XK_D uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x (low half) = lo
  return *reinterpret_cast<uint32_t*>(&v);
}

XK_D float bf16_at(const uint16_t* w, int i) {
  return __uint_as_float(((uint32_t)w[i]) << 16);
}

// D = A * B + D for one m16n8k16 tile (A row-major 16x16, B "col" 16x8, BF16 in, FP32 accumulate).
XK_D void mma_bf16(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------------ features

// Current gap of a candidate over (r_a + r_b), in float, from the segment differences a3 = a1 - a0,
// b3 = b1 - b0, w3 = a0 - b0: the clamped closest-point parameters of _closest_point_segments_batch
// (geometry/_compute.py:55-151) in float, each product and sum rounded on its own (no contraction),
// so that a NumPy float32 restatement gives the same value; near-parallel pairs (det <= 1e-3 ac)
// take s = 0.
XK_D float current_gap_f(const float* a3, const float* b3, const float* w3, float rsf) {
  auto dotf = [](const float* p, const float* q) {
    return __fadd_rn(__fadd_rn(__fmul_rn(p[0], q[0]), __fmul_rn(p[1], q[1])), __fmul_rn(p[2], q[2]));
  };
  auto clampf = [](float v) { return v < 0.f ? 0.f : (v > 1.f ? 1.f : v); };
  const float a = dotf(a3, a3), b = dotf(a3, b3), c = dotf(b3, b3), d = dotf(a3, w3), e = dotf(b3, w3);
  const float ac = __fmul_rn(a, c);
  const float det = __fsub_rn(ac, __fmul_rn(b, b));
  float s, t;
  if (!(det > __fmul_rn(1e-3f, ac))) {
    s = 0.f;
    t = c > 0.f ? clampf(__fdiv_rn(e, c)) : 0.f;
  } else {
    const float su = __fdiv_rn(__fsub_rn(__fmul_rn(b, e), __fmul_rn(c, d)), det);
    const float tu = __fdiv_rn(__fsub_rn(__fmul_rn(a, e), __fmul_rn(b, d)), det);
    s = clampf(su);
    t = clampf(tu);
    if (su < 0.f || su > 1.f) t = c > 0.f ? clampf(__fdiv_rn(__fadd_rn(__fmul_rn(b, s), e), c)) : 0.f;
    if (tu < 0.f || tu > 1.f) {
      s = a > 0.f ? clampf(__fdiv_rn(__fsub_rn(__fmul_rn(b, t), d), a)) : 0.f;
      t = c > 0.f ? clampf(__fdiv_rn(__fadd_rn(__fmul_rn(b, s), e), c)) : 0.f;
    }
  }
  float D[3];
  for (int q = 0; q < 3; ++q) D[q] = __fsub_rn(__fadd_rn(w3[q], __fmul_rn(s, a3[q])), __fmul_rn(t, b3[q]));
  return __fdiv_rn(__fsub_rn(__fsqrt_rn(dotf(D, D)), rsf), rsf);
}

// start[s] = the first row of the old table (sorted by (ea, eb)) whose ea >= s, s in [0, ne]
__global__ void k_table_seg_start(xk_pairs p, long long ne, int32_t* __restrict__ start) {
  const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s > ne) return;
  long long lo = 0, hi = p.n;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (p.ea[mid] < s) lo = mid + 1; else hi = mid;
  }
  start[s] = (int32_t)lo;
}

// Difference of two positions held as float hi/lo pairs (the node records): the hi and lo parts
// subtracted separately and then added, each operation rounded on its own.
XK_D float split_diff(const float* p, const float* q, int c) {
  return __fadd_rn(__fsub_rn(p[c], q[c]), __fsub_rn(p[3 + c], q[3 + c]));
}

__global__ void k_features(xk_mesh m, const float* __restrict__ n32, const int32_t* __restrict__ cands, long long n,
                           xk_pairs old, const int32_t* __restrict__ ostart, float* __restrict__ feat,
                           uint8_t* __restrict__ hist) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int ea = cands[2 * i], eb = cands[2 * i + 1];
  const int nd[4] = {m.conn[2 * ea], m.conn[2 * ea + 1], m.conn[2 * eb], m.conn[2 * eb + 1]};
  float x[4][6];  // x_hi (3), x_lo (3) of the four nodes
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4* r = reinterpret_cast<const float4*>(n32 + (long long)nd[k] * XK_NODE32_STRIDE);
    const float4 p = __ldg(r), q = __ldg(r + 1);
    x[k][0] = p.x; x[k][1] = p.y; x[k][2] = p.z; x[k][3] = p.w; x[k][4] = q.x; x[k][5] = q.y;
  }
  const float rsf = xk_d2f(xadd(m.radii[ea], m.radii[eb]));
  // position differences from the split records (no double arithmetic), then everything in float with
  // each operation rounded on its own
  float dm[3], da[3], db[3], dw[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    da[c] = split_diff(x[1], x[0], c);
    db[c] = split_diff(x[3], x[2], c);
    dw[c] = split_diff(x[0], x[2], c);
    // m_a - m_b = ((a0 - b0) + (a1 - b1)) / 2
    dm[c] = __fmul_rn(0.5f, __fadd_rn(dw[c], split_diff(x[1], x[3], c)));
  }
  auto dotf = [](const float* p, const float* q) {
    return __fadd_rn(__fadd_rn(__fmul_rn(p[0], q[0]), __fmul_rn(p[1], q[1])), __fmul_rn(p[2], q[2]));
  };
  const float sep = __fsqrt_rn(dotf(dm, dm));
  const float lna = __fsqrt_rn(dotf(da, da)), lnb = __fsqrt_rn(dotf(db, db));
  float den = __fmul_rn(lna, lnb);
  if (!(den >= 1e-30f)) den = (den != den) ? den : 1e-30f;
  float f[MF];
  f[0] = __fdiv_rn(sep, rsf);
  f[1] = __fdiv_rn(fabsf(dotf(da, db)), den);
  f[2] = __fdiv_rn(__fadd_rn(lna, lnb), __fmul_rn(2.0f, rsf));
  const int la = m.layer ? m.layer[ea] : -1, lb = m.layer ? m.layer[eb] : -1;
  const bool have = la >= 0 && lb >= 0;
  const int dl = la > lb ? la - lb : lb - la;
  f[3] = have ? __fdiv_rn((float)(dl < 3 ? dl : 3), 3.0f) : 0.f;
  f[4] = (have && (la == 0 || lb == 0)) ? 1.f : 0.f;
  // previous-step gap: the pair in the old table (sorted by (ea, eb)), searched among the rows of ea
  long long lo = ostart[ea], hi = (long long)ostart[ea + 1] - 1, at = -1;
  while (lo <= hi) {
    const long long mid = (lo + hi) >> 1;
    const int ob = old.eb[mid];
    if (ob == eb) { at = mid; break; }
    if (ob < eb) lo = mid + 1; else hi = mid - 1;
  }
  float g5;
  if (at >= 0) {
    g5 = __fdiv_rn((float)old.gap[at], rsf);
  } else {  // no previous gap: the current one, in float (feature accuracy is enough)
    g5 = current_gap_f(da, db, dw, rsf);
  }
  g5 = g5 < -2.0f ? -2.0f : (g5 > 8.0f ? 8.0f : g5);
  f[5] = g5;
  f[6] = at >= 0 ? 1.f : 0.f;
  f[7] = 0.f;
  float4* o = reinterpret_cast<float4*>(feat + MF * i);
  o[0] = make_float4(f[0], f[1], f[2], f[3]);
  o[1] = make_float4(f[4], f[5], f[6], f[7]);
  uint8_t h = 0;
  if (at >= 0) {
    const long long c = old.cap;
    h = (old.status[at] != 0 || old.p_n[at] > 0.0 || old.k_pen[at] > 0.0 || old.z_t[at] != 0.0 ||
         old.z_t[c + at] != 0.0) ? 1 : 0;
  }
  hist[i] = h;
}

// ------------------------------------------------------------------ inference (tensor cores)

constexpr int FW_WARPS = 4;

__global__ void __launch_bounds__(32 * FW_WARPS) k_mlp_forward_mma(const uint16_t* __restrict__ P,
                                                                   const float* __restrict__ feat, long long n,
                                                                   float* __restrict__ logit) {
  __shared__ __align__(16) uint16_t W[NP + 7];
  for (int i = threadIdx.x; i < NP; i += blockDim.x) W[i] = P[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const long long tiles = (n + 15) / 16;
  const uint32_t* W32 = reinterpret_cast<const uint32_t*>(W);
  for (long long tile = (long long)blockIdx.x * FW_WARPS + (threadIdx.x >> 5); tile < tiles;
       tile += (long long)gridDim.x * FW_WARPS) {
    const long long r0 = tile * 16 + g, r1 = r0 + 8;
    uint32_t a[4][4];
    {
      float2 x0 = r0 < n ? *reinterpret_cast<const float2*>(feat + MF * r0 + 2 * t) : make_float2(0.f, 0.f);
      float2 x1 = r1 < n ? *reinterpret_cast<const float2*>(feat + MF * r1 + 2 * t) : make_float2(0.f, 0.f);
      a[0][0] = pack_bf16(x0.x, x0.y);
      a[0][1] = pack_bf16(x1.x, x1.y);
      a[0][2] = 0u;  // k = 8..15: no inputs
      a[0][3] = 0u;
    }
    float c[8][4];
    // layer 1: K = 16 (8 inputs + zero padding)
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int j = nt * 8 + 2 * t;
      c[nt][0] = c[nt][2] = bf16_at(W, O_B1 + j);
      c[nt][1] = c[nt][3] = bf16_at(W, O_B1 + j + 1);
      mma_bf16(c[nt], a[0], W32[(O_W1 + (nt * 8 + g) * MF + 2 * t) >> 1], 0u);
    }
    // layers 2 and 3: K = 64 as 4 k-tiles; the relu'd, rounded accumulators are the next A operand
#pragma unroll
    for (int layer = 0; layer < 2; ++layer) {
      const int ow = layer == 0 ? O_W2 : O_W3, ob = layer == 0 ? O_B2 : O_B3;
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        a[kt][0] = pack_bf16(fmaxf(c[2 * kt][0], 0.f), fmaxf(c[2 * kt][1], 0.f));
        a[kt][1] = pack_bf16(fmaxf(c[2 * kt][2], 0.f), fmaxf(c[2 * kt][3], 0.f));
        a[kt][2] = pack_bf16(fmaxf(c[2 * kt + 1][0], 0.f), fmaxf(c[2 * kt + 1][1], 0.f));
        a[kt][3] = pack_bf16(fmaxf(c[2 * kt + 1][2], 0.f), fmaxf(c[2 * kt + 1][3], 0.f));
      }
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const int j = nt * 8 + 2 * t;
        c[nt][0] = c[nt][2] = bf16_at(W, ob + j);
        c[nt][1] = c[nt][3] = bf16_at(W, ob + j + 1);
        const int row = ow + (nt * 8 + g) * MH;
#pragma unroll
        for (int kt = 0; kt < 4; ++kt)
          mma_bf16(c[nt], a[kt], W32[(row + kt * 16 + 2 * t) >> 1], W32[(row + kt * 16 + 8 + 2 * t) >> 1]);
      }
    }
    // output: logit = b4 + sum_k bf16(relu(z3_k)) w4_k, the row sum over the quad
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int j = nt * 8 + 2 * t;
      const float w0 = bf16_at(W, O_W4 + j), w1 = bf16_at(W, O_W4 + j + 1);
      s0 += bf16r(fmaxf(c[nt][0], 0.f)) * w0 + bf16r(fmaxf(c[nt][1], 0.f)) * w1;
      s1 += bf16r(fmaxf(c[nt][2], 0.f)) * w0 + bf16r(fmaxf(c[nt][3], 0.f)) * w1;
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (t == 0) {
      const float b4 = bf16_at(W, O_B4);
      if (r0 < n) logit[r0] = s0 + b4;
      if (r1 < n) logit[r1] = s1 + b4;
    }
  }
}

// ------------------------------------------------------------------ inference (tcgen05, TMEM operands and accumulators)
//
// One CTA per SM, persistent over tiles of 128 candidates, five tiles in flight: 128 threads (four warps, a
// thread per candidate) run one tile's three layers, each group of four warps with its own 64-column TMEM
// accumulator, 32-column TMEM operand, mbarrier and named barrier.  A layer is tcgen05.mma (kind::f16, BF16 in,
// FP32 accumulate, M 128, N 64, K 16 per instruction) with the activations as the A operand in TMEM (a lane per
// candidate, two BF16 values per column) and the weights in shared memory in the canonical K-major layout without
// swizzle: 8-row x 16-byte core matrices (row r of a core at +16 r), cores adjacent along K LBO = 128 B
// apart, 8-row groups SBO apart.  A group's first thread issues the MMAs and commits to the mbarrier; the
// four warps read their 32 lanes back with tcgen05.ld, apply ReLU, round to BF16 and store the next operand
// with tcgen05.st.  The next tile's first layer runs while this tile's output sums are taken.
// What bounds it is latency: a tile is three dependent rounds.  Activations that go through TMEM need neither
// shared-memory stores, nor the proxy fence, nor the tensor core's reads of A from shared memory (which at
// N 64 take longer than the MMA itself), and one barrier a round is left of two.
// Measured at 3,197,900 candidates: operands staged in shared memory, five CTAs an SM 124 us, this 85.5 us (656
// TFLOP/s; of 164k clocks the tensor pipe is busy 35 %, the issue slots 52 %, the ALU 50 %: 96 conversions and
// 64 unpackings a candidate).  The logits are the same bits.
// Every wait is bounded: on expiry the kernel sets *err, skips the group's remaining work, and still frees its
// TMEM.

constexpr int TC_SLOTS = 5;
constexpr int TC_T = 128 * TC_SLOTS;
// columns: the accumulators, then the operands, then the constant operand of the biases
constexpr uint32_t TC_COLS = 512, TC_A = 64 * TC_SLOTS, TC_ONES = TC_A + 32 * TC_SLOTS;
static_assert(TC_ONES + 8 <= TC_COLS, "TMEM columns");
// instruction descriptor: D f32 (bit 4), A bf16 (bits 7-9 = 1), B bf16 (bits 10-12 = 1),
// K-major A and B (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28
constexpr uint32_t TC_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
constexpr long long TC_SPIN = 1LL << 22;

XK_D uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start >> 4 (bits 0-13), LBO >> 4 (16-29), SBO >> 4 (32-45),
// fixed 0b001 at bits 46-48, no base offset, relative LBO, no swizzle (bits 61-63 = 0)
XK_D uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

XK_D void tc_mma(uint32_t dtmem, uint32_t atmem, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      :
      : "r"(dtmem), "r"(atmem), "l"(bdesc), "r"(TC_IDESC), "r"(accumulate)
      : "memory");
}

XK_D void tc_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
               : "memory");
}

// bounded wait for the mbarrier phase `parity`; false on expiry
XK_D bool tc_wait(uint32_t mbar, uint32_t parity) {
  for (long long it = 0; it < TC_SPIN; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// 16 consecutive fp32 columns of this thread's TMEM lane
XK_D void tc_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 8 or 16 consecutive 32-bit columns of this thread's TMEM lane
XK_D void tc_st8(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
XK_D void tc_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

XK_D void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
XK_D void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
XK_D void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
XK_D void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
XK_D void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// a barrier of the 128 threads of one group; the disjunction of their predicates, the same in all of them
XK_D bool group_or(int id, bool pred) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "barrier.cta.red.or.aligned.pred q, %1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(any)
      : "r"(id), "r"((uint32_t)pred)
      : "memory");
  return any != 0;
}

// byte offset of element (row, k) (16-bit elements) in a K-major no-swizzle tile with K columns
XK_D uint32_t core_off(int row, int k, int K) {
  return (uint32_t)((row >> 3) * (K / 8) * 128 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// The biases ride in the MMAs: layer 1's operand has a constant-one column
// (k = 8) matched by b1 in W1's padding, and layers 2 and 3 add one K-16 MMA
// of a constant operand (k = 0 is 1) against a bias tile (column 0 = b).  The
// BF16 biases times 1 are exact in the FP32 accumulator.
struct __align__(128) TcSmem {
  uint16_t w1[64 * 16];  // [W1 | b1 | 0] as N 64 x K 16
  uint16_t w2[64 * 64];
  uint16_t w3[64 * 64];
  uint16_t bb2[64 * 16];  // column 0 = b2
  uint16_t bb3[64 * 16];  // column 0 = b3
  float w4[64];
  float b4;
  uint64_t mbar[TC_SLOTS];
  uint32_t tmem;
};

// two floats -> bf16x2 (lo in the low half), each max(x, 0) rounded to nearest even
XK_D uint32_t pack_relu_bf16(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

__global__ void __launch_bounds__(TC_T, 1) k_mlp_forward_tc(const uint16_t* __restrict__ P,
                                                            const float* __restrict__ feat, long long n,
                                                            float* __restrict__ logit, int* __restrict__ err) {
  __shared__ TcSmem sm;
  const int slot = threadIdx.x >> 7, tid = threadIdx.x & 127, warp = tid >> 5;
  // weights in the operand layout (N rows = outputs, K = inputs), biases as float
  constexpr uint16_t BF16_ONE = 0x3F80;
  for (int i = threadIdx.x; i < 64 * 16; i += TC_T) {
    const int nn = i >> 4, k = i & 15;
    const uint16_t v = k < MF ? P[O_W1 + nn * MF + k] : k == MF ? P[O_B1 + nn] : (uint16_t)0;
    const uint32_t o = core_off(nn, k, 16);
    *reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(sm.w1) + o) = v;
    *reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(sm.bb2) + o) = k == 0 ? P[O_B2 + nn] : (uint16_t)0;
    *reinterpret_cast<uint16_t*>(reinterpret_cast<char*>(sm.bb3) + o) = k == 0 ? P[O_B3 + nn] : (uint16_t)0;
  }
  // W2, W3: one 16-byte core-matrix row (8 consecutive k of output nn) per copy; the
  // parameter offsets of both are multiples of 8 elements
  static_assert(O_W2 % 8 == 0 && O_W3 % 8 == 0, "16-byte weight rows");
  for (int i = threadIdx.x; i < 64 * 8; i += TC_T) {
    const int nn = i >> 3, kc = i & 7;
    const uint32_t o = core_off(nn, 8 * kc, 64);
    *reinterpret_cast<uint4*>(reinterpret_cast<char*>(sm.w2) + o) = *reinterpret_cast<const uint4*>(P + O_W2 + 8 * i);
    *reinterpret_cast<uint4*>(reinterpret_cast<char*>(sm.w3) + o) = *reinterpret_cast<const uint4*>(P + O_W3 + 8 * i);
  }
  if (threadIdx.x < 64) sm.w4[threadIdx.x] = bf16_at(P, O_W4 + threadIdx.x);
  if (threadIdx.x == 0) sm.b4 = bf16_at(P, O_B4);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&sm.mbar[slot])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sm.tmem)),
                 "r"(TC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem;
  const uint32_t lanes = (uint32_t)(32 * warp) << 16;  // this warp's 32 TMEM lanes
  if (slot == 0) {  // the constant operand: 1 at k = 0
    const uint32_t v[8] = {BF16_ONE, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    tc_st8(tmem + lanes + TC_ONES, v);
    tc_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t mbar = smem_u32(&sm.mbar[slot]);
  const uint32_t acc = tmem + 64u * slot, opnd = tmem + TC_A + 32u * slot;
  const long long tiles = (n + 127) / 128, stride = (long long)gridDim.x * TC_SLOTS;
  long long tile = blockIdx.x + (long long)gridDim.x * slot;
  // features of this thread's row of a tile (zero beyond n); the next tile's are loaded while
  // the current tile runs its layers
  float4 x_lo, x_hi;
  auto load_row = [&](long long t) {
    const long long row = t * 128 + tid;
    x_lo = x_hi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < tiles && row < n) {
      const float4* f4 = reinterpret_cast<const float4*>(feat + MF * row);
      x_lo = __ldcs(f4);
      x_hi = __ldcs(f4 + 1);
    }
  };
  auto stage = [&] {  // layer-1 operand: the features rounded to bf16, the one for b1, zeros
    const uint32_t v[8] = {pack_bf16(x_lo.x, x_lo.y), pack_bf16(x_lo.z, x_lo.w), pack_bf16(x_hi.x, x_hi.y),
                           pack_bf16(x_hi.z, x_hi.w), BF16_ONE, 0u, 0u, 0u};
    tc_st8(opnd + lanes, v);
    tc_wait_st();
  };
  uint32_t phase = 0;
  bool bad = false;  // a wait of this thread has expired
  // the group's operand is stored (and its accumulator read): its first thread issues a layer's MMAs.
  // False, in all threads of the group, once a wait of any of them has expired.
  auto issue = [&](int layer) {
    tc_fence_before();
    if (group_or(1 + slot, bad)) return false;
    tc_fence_after();
    if (tid == 0) {
      if (layer == 0) {
        tc_mma(acc, opnd, tc_desc(smem_u32(sm.w1), 128, 256), 0u);
      } else {
        const uint32_t w = smem_u32(layer == 1 ? sm.w2 : sm.w3);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) tc_mma(acc, opnd + 8u * ks, tc_desc(w + ks * 256, 128, 1024), ks > 0 ? 1u : 0u);
        tc_mma(acc, tmem + TC_ONES, tc_desc(smem_u32(layer == 1 ? sm.bb2 : sm.bb3), 128, 256), 1u);
      }
      tc_commit(mbar);
    }
    __syncwarp();
    return true;
  };
  float z[64];
  auto fetch = [&] {  // wait for the layer and read this candidate's accumulator row
    bad |= !tc_wait(mbar, phase);
    phase ^= 1u;
    __syncwarp();
    tc_fence_after();
#pragma unroll
    for (int k = 0; k < 4; ++k) tc_ld16(acc + lanes + 16u * k, z + 16 * k);
    tc_wait_ld();
#pragma unroll
    for (int k = 0; k < 64; ++k) asm volatile("" : "+f"(z[k]));  // nothing that uses a value moves before the wait
  };
  load_row(tile);
  bool go = tile < tiles;  // the same in the whole group
  if (go) {
    stage();
    load_row(tile + stride);
    go = issue(0);
  }
  while (go) {
#pragma unroll 1
    for (int layer = 1; layer < 3 && go; ++layer) {
      fetch();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] = pack_relu_bf16(z[32 * h + 2 * c], z[32 * h + 2 * c + 1]);
        tc_st16(opnd + lanes + 16u * h, v);
      }
      tc_wait_st();
      go = issue(layer);
    }
    if (!go) break;
    fetch();
    // the last layer's MMAs have read the operand and its accumulator is in registers: the next tile begins
    const long long row = tile * 128 + tid;
    tile += stride;
    if (tile < tiles) {
      stage();
      load_row(tile + stride);
      go = issue(0);
    } else {
      go = false;
    }
    float out = 0.f;
#pragma unroll
    for (int j = 0; j < 64; j += 2) {
      const uint32_t h = pack_relu_bf16(z[j], z[j + 1]);
      out = fmaf(__uint_as_float(h << 16), sm.w4[j], out);
      out = fmaf(__uint_as_float(h & 0xFFFF0000u), sm.w4[j + 1], out);
    }
    if (!bad && row < n) logit[row] = out + sm.b4;
  }
  if (bad) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TC_COLS) : "memory");
}

// ------------------------------------------------------------------ training
//
// Activations and deltas are stored plane-major: value q of sample i at [q * n + i].
// The layers' products (n x 64 by 64 x 64, FP32 on BF16-rounded weights and activations) run as register tiles:
// a CTA of 128 threads takes 128 samples, each thread eight samples by eight outputs from operands in shared
// memory, 64 multiply-adds for sixteen loaded values.  One sample per thread, as before, loads a weight for
// every multiply-add, and what bounds that is the 128 bytes per clock that shared memory returns to the
// registers.  Every sum keeps its order (k ascending from zero), so activations, logits and deltas are the same
// bits.  Tensor cores are no way here: another order of the sums rounds one activation in 20,000 to the other
// bfloat16 neighbour, which moves the logits by more than float rounding.
// Measured at 201,347 samples, one sample per thread against this: forward 161 -> 113 us, backward
// 423 -> 159 us, weight gradients 963 -> 142 us (94,000 of 234,000 clocks of the forward are its multiply-adds).

constexpr int TR_T = 128;   // threads, and samples of a tile
constexpr int TR_LD = 132;  // row stride of a tile [value][sample]: rows 4 banks apart, 16-byte aligned
struct TrainTile {
  float v[MH][TR_LD];
};

// Weight matrix in shared memory for tile_mul: the eight outputs og + 8 j of thread group og (whose results then go
// to rows one apart) stand at columns 4 og ... 4 og + 3 and 32 + 4 og ..., so that a warp's two 16-byte loads
// meet every bank once.
XK_D int tile_col(int out) { return 32 * (out >> 5) + 4 * (out & 7) + ((out >> 3) & 3); }

// acc[i][j] = sum_k A[k][8 sg + i] B[k][og + 8 j], k ascending
template <int K>
XK_D void tile_mul(const float (*A)[TR_LD], const float (*B)[MH], int sg, int og, float (*acc)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    const float4 a0 = *reinterpret_cast<const float4*>(&A[k][8 * sg]);
    const float4 a1 = *reinterpret_cast<const float4*>(&A[k][8 * sg + 4]);
    const float4 b0 = *reinterpret_cast<const float4*>(&B[k][4 * og]);
    const float4 b1 = *reinterpret_cast<const float4*>(&B[k][32 + 4 * og]);
    const float x[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float w[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(w[j], x[i], acc[i][j]);
  }
}

struct TrainFwdSmem {
  float w1[MF][MH], w2[MH][MH], w3[MH][MH];
  float b1[MH], b2[MH], b3[MH], w4[MH];
  TrainTile a;
};

__global__ void __launch_bounds__(TR_T, 3) k_mlp_train_fwd(const float* __restrict__ theta,
                                                           const float* __restrict__ feat, long long n,
                                                           float* __restrict__ act, float* __restrict__ logit) {
  extern __shared__ __align__(16) unsigned char raw[];
  TrainFwdSmem& sm = *reinterpret_cast<TrainFwdSmem*>(raw);
  const int tid = threadIdx.x;
  for (int i = tid; i < MH * MF; i += TR_T) sm.w1[i % MF][tile_col(i / MF)] = bf16r(theta[O_W1 + i]);
  for (int i = tid; i < MH * MH; i += TR_T) {
    sm.w2[i % MH][tile_col(i / MH)] = bf16r(theta[O_W2 + i]);
    sm.w3[i % MH][tile_col(i / MH)] = bf16r(theta[O_W3 + i]);
  }
  if (tid < MH) {
    sm.b1[tid] = bf16r(theta[O_B1 + tid]);
    sm.b2[tid] = bf16r(theta[O_B2 + tid]);
    sm.b3[tid] = bf16r(theta[O_B3 + tid]);
    sm.w4[tid] = bf16r(theta[O_W4 + tid]);
  }
  const float b4 = bf16r(theta[O_B4]);
  const int og = tid & 7, sg = tid >> 3;  // outputs og + 8 j, samples 8 sg + i
  for (long long s0 = (long long)blockIdx.x * TR_T; s0 < n; s0 += (long long)gridDim.x * TR_T) {
    const int ns = n - s0 < TR_T ? (int)(n - s0) : TR_T;
    __syncthreads();  // the weights are in place; the last tile has been read
#pragma unroll
    for (int k = 0; k < MF; ++k) sm.a.v[k][tid] = tid < ns ? bf16r(feat[MF * (s0 + tid) + k]) : 0.f;
    __syncthreads();
#pragma unroll 1
    for (int layer = 0; layer < 3; ++layer) {
      float acc[8][8];
      if (layer == 0) tile_mul<MF>(sm.a.v, sm.w1, sg, og, acc);
      else tile_mul<MH>(sm.a.v, layer == 1 ? sm.w2 : sm.w3, sg, og, acc);
      const float* b = layer == 0 ? sm.b1 : (layer == 1 ? sm.b2 : sm.b3);
      __syncthreads();  // every thread has read the layer's inputs
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float bj = b[og + 8 * j];
        float z[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) z[i] = bf16r(fmaxf(acc[i][j] + bj, 0.f));
        float4* o = reinterpret_cast<float4*>(&sm.a.v[og + 8 * j][8 * sg]);
        o[0] = make_float4(z[0], z[1], z[2], z[3]);
        o[1] = make_float4(z[4], z[5], z[6], z[7]);
      }
      __syncthreads();
      if (tid < ns) {
#pragma unroll 8
        for (int j = 0; j < MH; ++j) act[(long long)(layer * MH + j) * n + s0 + tid] = sm.a.v[j][tid];
      }
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < MH; ++k) s += sm.a.v[k][tid] * sm.w4[k];
    if (tid < ns) logit[s0 + tid] = s + b4;
  }
}

struct TrainBwdSmem {
  float w2[MH][MH], w3[MH][MH];  // [j][k]: the rows that delta_j is multiplied with
  float w4[MH];
  double red[TR_T];
  TrainTile d;
};

// Loss part of the tile, delta of the output (g) and the deltas of the three hidden layers.  The loss and the
// sigmoid are taken in double from one exponential: with e = exp(-|l|), softplus(l) = max(l, 0) + log1p(e) and
// sigmoid(l) = 1 / (1 + e) or e / (1 + e).
__global__ void __launch_bounds__(TR_T, 3) k_mlp_train_bwd(const float* __restrict__ theta,
                                                           const float* __restrict__ act,
                                                           const float* __restrict__ logit,
                                                           const float* __restrict__ y, const float* __restrict__ w,
                                                           long long n, float* __restrict__ dvec,
                                                           float* __restrict__ gout, double* __restrict__ loss_part) {
  extern __shared__ __align__(16) unsigned char raw[];
  TrainBwdSmem& sm = *reinterpret_cast<TrainBwdSmem*>(raw);
  const int tid = threadIdx.x;
  for (int i = tid; i < MH * MH; i += TR_T) {
    sm.w2[i / MH][tile_col(i % MH)] = bf16r(theta[O_W2 + i]);
    sm.w3[i / MH][tile_col(i % MH)] = bf16r(theta[O_W3 + i]);
  }
  if (tid < MH) sm.w4[tid] = bf16r(theta[O_W4 + tid]);
  const int og = tid & 7, sg = tid >> 3;
  const Divisor64 dn = divisor64((double)n);
  for (long long t = blockIdx.x; t * TR_T < n; t += gridDim.x) {
    const long long s0 = t * TR_T, i = s0 + tid;
    const bool live = i < n;
    // which of this sample's activations are positive, as bits: 32 loads in flight a thread, all of them before
    // the tile's arithmetic (a load between the sums waited out its latency: 475 us)
    uint32_t pos[NA / 32];
#pragma unroll
    for (int q = 0; q < NA / 32; ++q) {
      pos[q] = 0u;
      if (live) {
        float v[32];
#pragma unroll
        for (int b = 0; b < 32; ++b) v[b] = act[(long long)(32 * q + b) * n + i];
#pragma unroll
        for (int b = 0; b < 32; ++b) pos[q] |= (v[b] > 0.f ? 1u : 0u) << b;
      }
    }
    float g = 0.f;
    double li = 0.0;
    if (live) {
      const double l = (double)logit[i], yi = (double)y[i], wi = (double)w[i];
      const double e = exp(-fabs(l)), sig = (l >= 0.0 ? 1.0 : e) * rcp64(1.0 + e);
      li = div64(wi * ((l > 0.0 ? l : 0.0) + log1p(e) - yi * l), dn);
      g = (float)div64(wi * (sig - yi), dn);
      gout[i] = g;
    }
    __syncthreads();  // the weights are in place; the last tile has been read
    sm.red[tid] = li;
#pragma unroll
    for (int k = 0; k < MH; ++k) {
      const float v = (pos[4 + k / 32] >> (k % 32)) & 1u ? g * sm.w4[k] : 0.f;
      if (live) dvec[(long long)(2 * MH + k) * n + i] = v;
      sm.d.v[k][tid] = v;
    }
    __syncthreads();
#pragma unroll
    for (int layer = 1; layer >= 0; --layer) {  // d2 = (W3^T d3) masked, then d1 = (W2^T d2) masked
      float acc[8][8];
      tile_mul<MH>(sm.d.v, layer == 1 ? sm.w3 : sm.w2, sg, og, acc);
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float4* o = reinterpret_cast<float4*>(&sm.d.v[og + 8 * j][8 * sg]);
        o[0] = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
        o[1] = make_float4(acc[4][j], acc[5][j], acc[6][j], acc[7][j]);
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < MH; ++k) {
        const float v = (pos[2 * layer + k / 32] >> (k % 32)) & 1u ? sm.d.v[k][tid] : 0.f;
        if (live) dvec[(long long)(layer * MH + k) * n + i] = v;
        if (layer == 1) sm.d.v[k][tid] = v;
      }
      __syncthreads();
    }
    for (int h = TR_T / 2; h > 0; h >>= 1) {
      if (tid < h) sm.red[tid] += sm.red[tid + h];
      __syncthreads();
    }
    if (tid == 0) loss_part[t] = sm.red[0];
  }
}

// Weight gradients: a CTA sums a chunk of samples for every parameter in sample order, two warps with the 64 x 64
// products d2 a1^T and two with d3 a2^T as 8 x 8 tiles a thread (four samples at a time from [value][sample] rows
// in shared memory), then its share of the small ones; a second kernel adds the chunks' sums in a fixed order.
// The chunk follows from n alone, so that the sums' order does too: the samples dealt out in whole tiles to WG_CTAS
// CTAs (what this GPU's 152 SMs hold, three each), or to as many rounds of them as leave no chunk above WG_MOST
// samples, which bounds the float chains of additions.  Chunks of 1,024 whatever n left a few thousand samples to one
// or two CTAs (1,200 samples: 600 us) and fill the last round by chance (500,001 samples: the gradient 1,100 us).
constexpr int WG_T = 128, WG_S = 32, WG_LD = 36, WG_CTAS = 456, WG_MOST = 1024;
static_assert(WG_MOST % WG_S == 0, "whole tiles");
static_assert(NA % 64 == 0 && WG_T == 128, "row loads: 16 rows a warp and round");
constexpr int WG_A = MF + NA;  // rows x0 a1 a2 a3
struct WgradSmem {
  float d[NA][WG_LD];  // d1 d2 d3
  float a[WG_A][WG_LD];
  float g[WG_LD];
};
long long wgrad_chunk(long long n) {
  const long long rounds = (n + WG_CTAS * WG_MOST - 1) / (WG_CTAS * WG_MOST);
  const long long per = (n + WG_CTAS * rounds - 1) / (WG_CTAS * rounds);
  return (per + WG_S - 1) / WG_S * WG_S;
}

__global__ void __launch_bounds__(WG_T, 3) k_mlp_wgrad(const float* __restrict__ feat, const float* __restrict__ act,
                                                       const float* __restrict__ dvec, const float* __restrict__ g,
                                                       long long n, long long chunk, float* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char raw[];
  WgradSmem& sm = *reinterpret_cast<WgradSmem*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = warp >> 1;                      // 0: d2 a1^T, 1: d3 a2^T
  const int tr = (tid & 63) >> 3, tc = tid & 7;    // this thread's rows tr + 8 i and columns tc + 8 j
  const float(*D)[WG_LD] = sm.d + MH * (1 + half);
  const float(*A)[WG_LD] = sm.a + MF + MH * half;
  float acc[8][8], w1[4] = {0.f, 0.f, 0.f, 0.f}, b0 = 0.f, b1 = 0.f, w4 = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  const int r1 = tid >> 1, c1 = 4 * (tid & 1);     // this thread's part of d1 x0^T: row r1, columns c1 ... c1 + 3
  const long long c0 = (long long)blockIdx.x * chunk, ce = c0 + chunk < n ? c0 + chunk : n;
  for (long long s0 = c0; s0 < ce; s0 += WG_S) {
    const bool in = s0 + lane < ce;
    __syncthreads();
#pragma unroll
    for (int q0 = warp; q0 < NA; q0 += 16 * (WG_T / 32)) {  // 32 loads in flight a thread
      float vd[16], va[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const long long at = (long long)(q0 + 4 * q) * n + s0 + lane;
        vd[q] = in ? dvec[at] : 0.f;
        va[q] = in ? act[at] : 0.f;
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        sm.d[q0 + 4 * q][lane] = vd[q];
        sm.a[MF + q0 + 4 * q][lane] = va[q];
      }
    }
#pragma unroll
    for (int e = tid; e < WG_S * MF; e += WG_T) {
      const int q = e % MF, s = e / MF;
      sm.a[q][s] = s0 + s < ce ? bf16r(feat[MF * (s0 + s) + q]) : 0.f;
    }
    if (warp == 0) sm.g[lane] = in ? g[s0 + lane] : 0.f;
    __syncthreads();
    // samples past the chunk add zero times zero
#pragma unroll 1
    for (int s = 0; s < WG_S; s += 4) {
      float4 x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = *reinterpret_cast<const float4*>(&A[tc + 8 * j][s]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 d = *reinterpret_cast<const float4*>(&D[tr + 8 * i][s]);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          acc[i][j] = fmaf(d.w, x[j].w, fmaf(d.z, x[j].z, fmaf(d.y, x[j].y, fmaf(d.x, x[j].x, acc[i][j]))));
      }
      const float4 d1 = *reinterpret_cast<const float4*>(&sm.d[r1][s]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(&sm.a[c1 + j][s]);
        w1[j] = fmaf(d1.w, v.w, fmaf(d1.z, v.z, fmaf(d1.y, v.y, fmaf(d1.x, v.x, w1[j]))));
      }
      const float4 e0 = *reinterpret_cast<const float4*>(&sm.d[tid][s]);
      b0 = (((b0 + e0.x) + e0.y) + e0.z) + e0.w;
      const float4 gs = *reinterpret_cast<const float4*>(&sm.g[s]);
      if (tid < MH) {  // bias row 128 + tid, and w4
        const float4 e1 = *reinterpret_cast<const float4*>(&sm.d[WG_T + tid][s]);
        b1 = (((b1 + e1.x) + e1.y) + e1.z) + e1.w;
        const float4 v = *reinterpret_cast<const float4*>(&sm.a[MF + 2 * MH + tid][s]);
        w4 = fmaf(gs.w, v.w, fmaf(gs.z, v.z, fmaf(gs.y, v.y, fmaf(gs.x, v.x, w4))));
      } else if (tid == MH) {
        b1 = (((b1 + gs.x) + gs.y) + gs.z) + gs.w;  // b4
      }
    }
  }
  float* o = partial + (long long)blockIdx.x * NP;
  float* m = o + (half == 0 ? O_W2 : O_W3);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) m[(tr + 8 * i) * MH + tc + 8 * j] = acc[i][j];
#pragma unroll
  for (int j = 0; j < 4; ++j) o[O_W1 + r1 * MF + c1 + j] = w1[j];
  o[tid < MH ? O_B1 + tid : O_B2 + tid - MH] = b0;
  if (tid < MH) {
    o[O_B3 + tid] = b1;
    o[O_W4 + tid] = w4;
  } else if (tid == MH) {
    o[O_B4] = b1;
  }
}

// grad[p] = the sum of the chunks' partials: SP_G groups of consecutive chunks, each in order, then the groups in
// order.  One more block adds the tiles' loss parts in a fixed tree.
constexpr int SP_P = 32, SP_G = 8;
__global__ void __launch_bounds__(SP_P * SP_G) k_sum_partials(const float* __restrict__ partial, int nb,
                                                              float* __restrict__ grad,
                                                              const double* __restrict__ loss_part, long long nl,
                                                              float* __restrict__ loss) {
  __shared__ float part[SP_G][SP_P];
  __shared__ double red[SP_P * SP_G];
  const int tid = threadIdx.x, col = tid % SP_P, grp = tid / SP_P;
  if (blockIdx.x == gridDim.x - 1) {
    double s = 0.0;
    for (long long b = tid; b < nl; b += SP_P * SP_G) s += loss_part[b];
    red[tid] = s;
    __syncthreads();
    for (int h = SP_P * SP_G / 2; h > 0; h >>= 1) {
      if (tid < h) red[tid] += red[tid + h];
      __syncthreads();
    }
    if (tid == 0) *loss = (float)red[0];
    return;
  }
  const int p = blockIdx.x * SP_P + col;
  const int per = (nb + SP_G - 1) / SP_G, b0 = grp * per, b1 = b0 + per < nb ? b0 + per : nb;
  float s = 0.f;
  if (p < NP) {
#pragma unroll 8
    for (int b = b0; b < b1; ++b) s += partial[(long long)b * NP + p];
  }
  part[grp][col] = s;
  __syncthreads();
  if (grp == 0 && p < NP) {
    for (int q = 1; q < SP_G; ++q) s += part[q][col];
    grad[p] = s;
  }
}

// a persistent grid of tiles: as many CTAs as the SMs hold, at most one per tile
int train_grid(long long n, int per_sm) {
  const long long tiles = (n + TR_T - 1) / TR_T, cap = (long long)per_sm * xk_sm_count();
  return (int)(tiles < cap ? tiles : cap);
}

// Adam with the float32 roundings of the oracle's NumPy expressions (no contraction).
__global__ void k_adam(float* __restrict__ theta, const float* __restrict__ grad, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float ob1, float b2, float ob2, float bc1, float bc2,
                       float eps, uint16_t* __restrict__ out_bf16) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NP) return;
  const float gr = grad[p];
  const float mm = __fadd_rn(__fmul_rn(b1, m[p]), __fmul_rn(ob1, gr));
  const float vv = __fadd_rn(__fmul_rn(b2, v[p]), __fmul_rn(__fmul_rn(ob2, gr), gr));
  const float mh = __fdiv_rn(mm, bc1), vh = __fdiv_rn(vv, bc2);
  const float th = __fsub_rn(theta[p], __fdiv_rn(__fmul_rn(lr, mh), __fadd_rn(__fsqrt_rn(vh), eps)));
  m[p] = mm;
  v[p] = vv;
  theta[p] = th;
  if (out_bf16) {
    __nv_bfloat16 h = __float2bfloat16_rn(th);
    out_bf16[p] = *reinterpret_cast<uint16_t*>(&h);
  }
}

__global__ void k_to_bf16(const float* __restrict__ theta, uint16_t* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NP) return;
  __nv_bfloat16 h = __float2bfloat16_rn(theta[p]);
  out[p] = *reinterpret_cast<uint16_t*>(&h);
}

// ------------------------------------------------------------------ selection and table compaction

// keep flag of candidate i; a scoring that reported an expired tensor-core wait (*err != 0) keeps every
// candidate, since its scores are undefined
__global__ void k_keep_flags(long long n, const float* __restrict__ logit, const uint8_t* __restrict__ hist,
                             float thr, int invert, const int32_t* __restrict__ err, int32_t* __restrict__ flag) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const int keep = (logit[i] >= thr || (hist && hist[i]) || (err && *err)) ? 1 : 0;
    flag[i] = invert ? 1 - keep : keep;
  }
}

__global__ void k_scatter_cands(long long n, const int32_t* __restrict__ cands, const int32_t* __restrict__ flag,
                                const int32_t* __restrict__ off, int32_t* __restrict__ kept) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && flag[i]) {
    const long long o = off[i];
    kept[2 * o] = cands[2 * i];
    kept[2 * o + 1] = cands[2 * i + 1];
  }
}

__global__ void k_old_keep(xk_pairs p, const int32_t* __restrict__ kept, long long nk, int32_t* __restrict__ flag) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= p.n) return;
  const long long c = p.cap;
  const bool pristine = p.status[j] == 0 && p.p_n[j] == 0.0 && p.k_pen[j] == 0.0 && p.z_t[j] == 0.0 &&
                        p.z_t[c + j] == 0.0;
  int keep = 1;
  if (pristine) {
    const int ea = p.ea[j], eb = p.eb[j];
    long long lo = 0, hi = nk - 1;
    keep = 0;
    while (lo <= hi) {
      const long long mid = (lo + hi) >> 1;
      const int a = kept[2 * mid], b = kept[2 * mid + 1];
      if (a == ea && b == eb) { keep = 1; break; }
      if (a < ea || (a == ea && b < eb)) lo = mid + 1; else hi = mid - 1;
    }
  }
  flag[j] = keep;
}

__global__ void k_compact_table(xk_pairs in, const int32_t* __restrict__ flag, const int32_t* __restrict__ off,
                                xk_pairs out) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= in.n || !flag[j]) return;
  const long long o = off[j], ci = in.cap, co = out.cap;
  out.ea[o] = in.ea[j];
  out.eb[o] = in.eb[j];
  out.s[o] = in.s[j];
  out.t[o] = in.t[j];
  out.gap[o] = in.gap[j];
  for (int c = 0; c < 3; ++c) {
    out.normal[c * co + o] = in.normal[c * ci + j];
    out.t1[c * co + o] = in.t1[c * ci + j];
    out.t2[c * co + o] = in.t2[c * ci + j];
  }
  out.lambda_n[o] = in.lambda_n[j];
  out.k_pen[o] = in.k_pen[j];
  out.k_t[o] = in.k_t[j];
  out.p_n[o] = in.p_n[j];
  out.z_t[o] = in.z_t[j];
  out.z_t[co + o] = in.z_t[ci + j];
  out.q_trial_norm[o] = in.q_trial_norm[j];
  out.dissipation[o] = in.dissipation[j];
  out.status[o] = in.status[j];
  out.stick[o] = in.stick[j];
}

}  // namespace

// ------------------------------------------------------------------ entry points

extern "C" xk_status xk_prune_features(const xk_mesh* m, const float* node32, const int32_t* cands, int64_t n,
                                       const xk_pairs* old, float* feat, uint8_t* hist, xk_stream s) {
  if (!m || !old || (n > 0 && (!cands || !feat || !hist || !node32)) || n < 0)
    return xk_set_error(XK_ERR_ARG, "xk_prune_features: bad arguments");
  if (n == 0) return XK_OK;
  cudaStream_t st = (cudaStream_t)s;
  const long long ne = m->n_elems;
  XkScratch S(st);  // the library's pool: the default one maps its memory again after every synchronisation (0.1 ms)
  int32_t* ostart;
  XK_TRY(S.get(&ostart, ne + 2));
  k_table_seg_start<<<xk_blocks(ne + 1, 256), 256, 0, st>>>(*old, ne, ostart);
  k_features<<<xk_blocks(n, 256), 256, 0, st>>>(*m, node32, cands, n, *old, ostart, feat, hist);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_mlp_forward(const uint16_t* params_bf16, const float* feat, int64_t n, float* logit,
                                    xk_stream s) {
  if (!params_bf16 || n < 0 || (n > 0 && (!feat || !logit)))
    return xk_set_error(XK_ERR_ARG, "xk_mlp_forward: bad arguments");
  if (n == 0) return XK_OK;
  const long long tiles = (n + 15) / 16;
  long long blocks = (tiles + FW_WARPS - 1) / FW_WARPS;
  if (blocks > 152 * 16) blocks = 152 * 16;  // grid-stride beyond 16 blocks per SM
  k_mlp_forward_mma<<<(int)blocks, 32 * FW_WARPS, 0, (cudaStream_t)s>>>(params_bf16, feat, n, logit);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_mlp_forward_tcgen05(const uint16_t* params_bf16, const float* feat, int64_t n, float* logit,
                                            int* err, xk_stream s) {
  if (!params_bf16 || !err || n < 0 || (n > 0 && (!feat || !logit)))
    return xk_set_error(XK_ERR_ARG, "xk_mlp_forward_tcgen05: bad arguments");
  if ((reinterpret_cast<uintptr_t>(params_bf16) & 15) || (reinterpret_cast<uintptr_t>(feat) & 15))
    return xk_set_error(XK_ERR_ARG, "xk_mlp_forward_tcgen05: params and feat must be 16-byte aligned");
  if (n == 0) return XK_OK;
  // one CTA per SM (it takes all of the SM's TMEM); tiles go round the CTAs, then round their groups, so that
  // few tiles spread over many SMs
  const long long tiles = (n + 127) / 128;
  const int sms = xk_sm_count(), blocks = (int)(tiles < sms ? tiles : sms);
  k_mlp_forward_tc<<<blocks, TC_T, 0, (cudaStream_t)s>>>(params_bf16, feat, n, logit, err);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_mlp_train_forward(const float* theta, const float* feat, int64_t n, float* act,
                                          float* logit, xk_stream s) {
  if (!theta || n < 0 || (n > 0 && (!feat || !act || !logit)))
    return xk_set_error(XK_ERR_ARG, "xk_mlp_train_forward: bad arguments");
  if (n == 0) return XK_OK;
  XK_CUDA(cudaFuncSetAttribute(k_mlp_train_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainFwdSmem)));
  k_mlp_train_fwd<<<train_grid(n, 3), TR_T, sizeof(TrainFwdSmem), (cudaStream_t)s>>>(theta, feat, n, act, logit);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_mlp_backward(const float* theta, const float* feat, const float* act, const float* logit,
                                     const float* y, const float* w, int64_t n, float* dvec, float* g, float* grad,
                                     float* loss, xk_stream s) {
  if (!theta || !grad || !loss || n <= 0 || !feat || !act || !logit || !y || !w || !dvec || !g)
    return xk_set_error(XK_ERR_ARG, "xk_mlp_backward: bad arguments");
  cudaStream_t st = (cudaStream_t)s;
  const long long tiles = (n + TR_T - 1) / TR_T, chunk = wgrad_chunk(n);
  const int nb_w = (int)((n + chunk - 1) / chunk);
  XK_CUDA(cudaFuncSetAttribute(k_mlp_train_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainBwdSmem)));
  XK_CUDA(cudaFuncSetAttribute(k_mlp_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WgradSmem)));
  double* lpart = nullptr;
  float* part = nullptr;
  XK_CUDA(cudaMallocAsync((void**)&lpart, sizeof(double) * tiles, st));
  cudaError_t e = cudaMallocAsync((void**)&part, sizeof(float) * (size_t)nb_w * NP, st);
  if (e != cudaSuccess) {
    cudaFreeAsync(lpart, st);
    return xk_set_cuda_error(e, __FILE__, __LINE__);
  }
  k_mlp_train_bwd<<<train_grid(n, 3), TR_T, sizeof(TrainBwdSmem), st>>>(theta, act, logit, y, w, n, dvec, g, lpart);
  k_mlp_wgrad<<<nb_w, WG_T, sizeof(WgradSmem), st>>>(feat, act, dvec, g, n, chunk, part);
  k_sum_partials<<<(NP + SP_P - 1) / SP_P + 1, SP_P * SP_G, 0, st>>>(part, nb_w, grad, lpart, tiles, loss);
  e = cudaGetLastError();
  cudaFreeAsync(lpart, st);
  cudaFreeAsync(part, st);
  if (e != cudaSuccess) return xk_set_cuda_error(e, __FILE__, __LINE__);
  return XK_OK;
}

extern "C" xk_status xk_mlp_adam(float* theta, const float* grad, float* m, float* v, int step, double lr,
                                 double beta1, double beta2, double eps, uint16_t* theta_bf16, xk_stream s) {
  if (!theta || !grad || !m || !v || step < 1) return xk_set_error(XK_ERR_ARG, "xk_mlp_adam: bad arguments");
  // each constant is formed in double and rounded to float once
  const float ob1 = (float)(1.0 - beta1), ob2 = (float)(1.0 - beta2);
  const float bc1 = (float)(1.0 - pow(beta1, step)), bc2 = (float)(1.0 - pow(beta2, step));
  k_adam<<<(NP + 255) / 256, 256, 0, (cudaStream_t)s>>>(theta, grad, m, v, (float)lr, (float)beta1, ob1,
                                                        (float)beta2, ob2, bc1, bc2, (float)eps, theta_bf16);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_mlp_to_bf16(const float* theta, uint16_t* out, xk_stream s) {
  if (!theta || !out) return xk_set_error(XK_ERR_ARG, "xk_mlp_to_bf16: bad arguments");
  k_to_bf16<<<(NP + 255) / 256, 256, 0, (cudaStream_t)s>>>(theta, out);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_prune_select(const int32_t* cands, int64_t n, const float* logit, const uint8_t* hist,
                                     float threshold, int invert, const int32_t* score_error, int32_t* kept,
                                     int64_t* n_kept, int32_t* score_failed, xk_stream s) {
  if (!n_kept || n < 0 || (n > 0 && (!cands || !logit || !kept)))
    return xk_set_error(XK_ERR_ARG, "xk_prune_select: bad arguments");
  *n_kept = 0;
  if (score_failed) *score_failed = 0;
  if (n == 0) return XK_OK;
  cudaStream_t st = (cudaStream_t)s;
  XkScratch S(st);
  int32_t* flag;
  int64_t* tot;  // [count, scoring error word]
  XK_TRY(S.reserve(8 * (size_t)n + 8 * (size_t)(n / 256) + 8192));
  XK_TRY(S.get(&flag, 2 * n));
  XK_TRY(S.get(&tot, 2));
  cudaError_t e = cudaSuccess;
  int32_t* off = flag + n;
  k_keep_flags<<<xk_blocks(n, 256), 256, 0, st>>>(n, logit, hist, threshold, invert, score_error, flag);
  xk_status r = xk_exclusive_scan_i32(flag, off, n, tot, st, &S);
  if (r == XK_OK) {
    k_scatter_cands<<<xk_blocks(n, 256), 256, 0, st>>>(n, cands, flag, off, kept);
    int64_t h[2] = {0, 0};
    e = cudaGetLastError();
    // the count and the scoring's error word come back in one copy
    if (e == cudaSuccess && score_error)
      e = cudaMemcpyAsync(tot + 1, score_error, sizeof(int32_t), cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, tot, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      r = xk_set_cuda_error(e, __FILE__, __LINE__);
    } else {
      *n_kept = h[0];
      if (score_failed && score_error) *score_failed = (int32_t)(h[1] & 0xffffffff);
    }
  }
  return r;
}

extern "C" xk_status xk_pairs_drop_pristine(const xk_pairs* in, const int32_t* kept, int64_t n_kept, xk_pairs* out,
                                            xk_stream s) {
  if (!in || !out || n_kept < 0 || (n_kept > 0 && !kept))
    return xk_set_error(XK_ERR_ARG, "xk_pairs_drop_pristine: bad arguments");
  cudaStream_t st = (cudaStream_t)s;
  out->n = 0;
  if (in->n == 0) return XK_OK;
  int32_t* flag = nullptr;
  int64_t* tot = nullptr;
  const long long n = in->n;
  XK_CUDA(cudaMallocAsync((void**)&flag, sizeof(int32_t) * 2 * n, st));
  cudaError_t e = cudaMallocAsync((void**)&tot, sizeof(int64_t), st);
  if (e != cudaSuccess) {
    cudaFreeAsync(flag, st);
    return xk_set_cuda_error(e, __FILE__, __LINE__);
  }
  int32_t* off = flag + n;
  k_old_keep<<<xk_blocks(n, 256), 256, 0, st>>>(*in, kept, n_kept, flag);
  xk_status r = xk_exclusive_scan_i32(flag, off, n, tot, st);
  int64_t h = 0;
  if (r == XK_OK) {
    e = cudaMemcpyAsync(&h, tot, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) r = xk_set_cuda_error(e, __FILE__, __LINE__);
  }
  if (r == XK_OK && h > out->cap) r = xk_set_error(XK_ERR_CAPACITY, "xk_pairs_drop_pristine: out->cap too small");
  if (r == XK_OK) {
    k_compact_table<<<xk_blocks(n, 256), 256, 0, st>>>(*in, flag, off, *out);
    e = cudaGetLastError();
    if (e != cudaSuccess) r = xk_set_cuda_error(e, __FILE__, __LINE__);
    else out->n = (int32_t)h;
  }
  cudaFreeAsync(flag, st);
  cudaFreeAsync(tot, st);
  return r;
}
