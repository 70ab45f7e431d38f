// Broadphase and pair-list update.
//
// The reference bins AABBs into a hash grid (xkep_cae/contact/_broadphase.py:52-87)
// and keeps the pairs whose closed AABBs overlap (:93-96); its output is the
// set of all overlapping pairs, whatever the cell size.  Here every segment is
// binned once, by the cell of its box's lower corner (counting sort by cell, each cell's entries then
// in ascending order).
// A box j can overlap box i only if its lower corner lies in [lo_i - E, hi_i]
// per axis, E the largest extent of any box on that axis.  Cells are numbered with
// the axis of the largest extent running fastest, so the range is a few rows of
// cells whose entries are contiguous; a warp per segment i walks those rows and tests every
// entry j > i: screened on float boxes rounded outward, tested on the exact
// double AABBs, filtered, compacted with ballot/popc into a fixed-size slot list
// of the segment.  Each pair is found once, from its lower-numbered segment, in
// a single walk: a second kernel sorts each slot list and applies the midpoint
// prescreen (whose margin is a mean over all candidates), a third writes the
// kept pairs out in (i, j) order.  A slot list that overflows is detected at the
// end and the walk is repeated with longer lists.  Filters follow
// DetectCandidatesProcess (_manager_process.py:200-217,260-286).
//
// FP64 operations are what these kernels must not spend (1.6 per clock and SM): cell numbers and ranges are
// computed once per segment by its own thread, not by every lane of the warp that walks it (96 operations a
// lane there: most of the walk's 558 us at 98,592 segments, 189 us now); the radius sums of the margin are skipped
// where every radius is the same; the prescreen decides in float from split midpoints (slot ranking 96 -> 58 us).
#include <atomic>
#include <cstddef>
#include <cstdio>

#include "merge.cuh"

namespace {

constexpr int BP_T = 128;  // 4 warps per block, one warp per segment

struct Grid {
  double origin[3], inv[3];  // lower corner, 1 / cell size
  double emax[3];            // largest box extent on each axis
  int dims[3], stride[3];    // cells per axis; stride 1 on axis f
  int f;
  int uniform;               // every radius is `radius`
  double radius;
};

// Words shared by the broadphase kernels, all zero at the start.
struct Words {
  unsigned long long lo_max[3];   // max of the inverted lower corners, order-preserving (the min, inverted)
  unsigned long long hi_max[3];   // max of the upper corners
  unsigned long long ext_max[3];  // max of the extents (bits of doubles >= 0)
  unsigned long long r_lo, r_hi;  // radii: max of the inverted and of the plain ones
  double ext_sum[3];              // sums of the extents (they set the cell size: any order will do)
  double margin;                  // of the prescreen
  unsigned int ticket, ticket2;
  // read back by the host
  long long raw, pre, longest, kept;
};

XK_D unsigned long long enc_min(double x) {  // order-preserving map of doubles to u64
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
XK_D double dec_min(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

// A segment's midpoint in float hi / lo parts with its half length and radius: the prescreen's float form.
struct __align__(32) MidF {
  float hi[3], half, lo[3], r;
};

// cells of cell_size, or (cell_size <= 0) of these fractions of the mean extent on each axis: short on the
// axis that runs fastest, where a row's length costs nothing, and on the others so that a segment's rows are
// some 25 (one batch of the walk's lanes); coarsened while there would be more than cap_cells cells
constexpr float CELL_FAST = 0.125f, CELL_OTHER = 0.5f;
XK_D void make_grid(const Words& w, long long ne, long long cap_cells, double cell_size, Grid* g) {
  // The walk is right for any cell size and count (cell coordinates are clamped and grow with the position), so
  // these are taken in float: one thread does this, and an FP64 divide takes it a microsecond.
  float span[3], cell[3], e[3];
  for (int c = 0; c < 3; ++c) {
    const double lo = dec_min(~w.lo_max[c]), hi = dec_min(w.hi_max[c]);
    g->origin[c] = lo;
    g->emax[c] = __longlong_as_double((long long)w.ext_max[c]);
    e[c] = xk_d2f(g->emax[c]);
    span[c] = xk_d2f(hi - lo);
  }
  const int f = (e[2] >= e[0] && e[2] >= e[1]) ? 2 : (e[1] >= e[0] ? 1 : 0);
  const int a = f == 0 ? 1 : 0, b = f == 2 ? 1 : 2;
  float n[3];
  for (int c = 0; c < 3; ++c) {
    cell[c] = cell_size > 0.0 ? xk_d2f(cell_size) : (c == f ? CELL_FAST : CELL_OTHER) * (xk_d2f(w.ext_sum[c]) / (float)ne);
    cell[c] = fmaxf(cell[c], span[c] * 9.5367432e-7f);  // at most 2^20 cells on an axis
    n[c] = span[c] > 0.f ? span[c] / cell[c] : 0.f;
    if (!(n[c] >= 0.f && n[c] <= 2097152.f)) n[c] = 0.f;  // extents that are not finite: one cell
  }
  for (int it = 0; it < 400 && (n[0] + 1.f) * (n[1] + 1.f) * (n[2] + 1.f) > 0.999f * (float)cap_cells; ++it)
    for (int c = 0; c < 3; ++c) n[c] *= 0.8f;
  for (int c = 0; c < 3; ++c) {
    g->dims[c] = (int)n[c] + 1;
    g->inv[c] = n[c] > 0.f ? xk_f2d(n[c] / span[c]) : 0.0;
  }
  g->f = f;
  g->stride[f] = 1;
  g->stride[a] = g->dims[f];
  g->stride[b] = g->dims[f] * g->dims[a];
  g->uniform = w.r_hi == ~w.r_lo;
  g->radius = dec_min(w.r_hi);
}

// box: the FP64 boxes, six doubles per segment (lower corner, upper corner); boxf: the same boxes in
// float, rounded outward (lower corner down, upper corner up), as two float4 per segment (32 bytes): a
// conservative screen for the sweep, which then tests the FP64 boxes.  mid: per segment its midpoint and
// half length in the operation order of the midpoint prescreen (_manager_process.py:265-272), so that
// the prescreen of a pair reads these 32 bytes of each segment and gives the same values; midf: the same in
// float parts.  The extremes and sums go over the block, then by one atomic each into w; the last block forms
// the grid.
// AABB_T: some 60 FP64 operations a segment, so few segments go in small CTAs to many SMs' pipes.
template <int AABB_T>
__global__ void __launch_bounds__(AABB_T) k_aabb(xk_mesh m, const double* __restrict__ u, double margin,
                                                 double* __restrict__ box, float4* __restrict__ boxf,
                                                 double4_32a* __restrict__ mid, MidF* __restrict__ midf,
                                                 Words* __restrict__ w, long long cap_cells, double cell_size,
                                                 Grid* __restrict__ grid) {
  constexpr int AABB_W = AABB_T / 32;
  __shared__ unsigned long long s_max[11][AABB_W];
  __shared__ double s_sum[3][AABB_W];
  __shared__ bool s_last;
  const int e = blockIdx.x * AABB_T + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long mx[11] = {};  // as Words: inverted lower corners, upper corners, extents, radii
  double sum[3] = {0.0, 0.0, 0.0};
  if (e < m.n_elems) {
    const int a = m.conn[2 * e], b = m.conn[2 * e + 1];
    const double rad = m.radii[e], ex = xadd(rad, margin);
    float lf[3], hf[3];
    double ma[3], da[3];
    MidF mf;
    for (int c = 0; c < 3; ++c) {
      double x0 = u ? xadd(m.X[3LL * a + c], u[6LL * a + c]) : m.X[3LL * a + c];
      double x1 = u ? xadd(m.X[3LL * b + c], u[6LL * b + c]) : m.X[3LL * b + c];
      ma[c] = xmul(0.5, xadd(x0, x1));
      da[c] = xsub(x1, x0);
      double lo = xsub(x0 < x1 ? x0 : x1, ex);
      double hi = xadd(x0 < x1 ? x1 : x0, ex);
      box[6LL * e + c] = lo;
      box[6LL * e + 3 + c] = hi;
      lf[c] = __double2float_rd(lo);
      hf[c] = __double2float_ru(hi);
      mf.hi[c] = xk_d2f(ma[c]);
      mf.lo[c] = xk_d2f(ma[c] - xk_f2d(mf.hi[c]));
      mx[c] = ~enc_min(lo);
      mx[3 + c] = enc_min(hi);
      sum[c] = fmax(hi - lo, 0.0);  // >= 0 (a negative margin may turn a box round): the bits order as the values
      mx[6 + c] = (unsigned long long)__double_as_longlong(sum[c]);
    }
    mx[9] = ~enc_min(rad);
    mx[10] = enc_min(rad);
    // the spare fourth word carries the element's layer (-1 without layers), read by the walk's filter
    boxf[2LL * e] = make_float4(lf[0], lf[1], lf[2], __int_as_float(m.layer ? m.layer[e] : -1));
    boxf[2LL * e + 1] = make_float4(hf[0], hf[1], hf[2], 0.f);
    double4_32a me;
    me.x = ma[0];
    me.y = ma[1];
    me.z = ma[2];
    me.w = xmul(0.5, xsqrt(xdot_seq(da, da)));
    mid[e] = me;
    mf.half = xk_d2f(me.w);
    mf.r = xk_d2f(rad);
    midf[e] = mf;
  }
#pragma unroll
  for (int k = 0; k < 11; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long y = __shfl_down_sync(0xffffffffu, mx[k], o);
      mx[k] = y > mx[k] ? y : mx[k];
    }
    if (lane == 0) s_max[k][warp] = mx[k];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    for (int o = 16; o > 0; o >>= 1) sum[c] += __shfl_down_sync(0xffffffffu, sum[c], o);
    if (lane == 0) s_sum[c][warp] = sum[c];
  }
  __syncthreads();
  if (threadIdx.x < 11) {
    unsigned long long v = s_max[threadIdx.x][0];
    for (int q = 1; q < AABB_W; ++q) v = s_max[threadIdx.x][q] > v ? s_max[threadIdx.x][q] : v;
    atomicMax(reinterpret_cast<unsigned long long*>(w) + threadIdx.x, v);
  } else if (threadIdx.x >= 32 && threadIdx.x < 35) {
    const int c = threadIdx.x - 32;
    double v = 0.0;
    for (int q = 0; q < AABB_W; ++q) v += s_sum[c][q];
    atomicAdd(&w->ext_sum[c], v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&w->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    const volatile unsigned long long* v = reinterpret_cast<const volatile unsigned long long*>(w);
    Words c;
    unsigned long long* d = reinterpret_cast<unsigned long long*>(&c);
    for (int k = 0; k < 14; ++k) d[k] = v[k];
    make_grid(c, m.n_elems, cap_cells, cell_size, grid);
  }
}

XK_D int cell_coord(const Grid& g, int c, double x) {
  const int ci = (int)floor((x - g.origin[c]) * g.inv[c]);
  return ci < 0 ? 0 : (ci >= g.dims[c] ? g.dims[c] - 1 : ci);
}

// Per segment: its cell (of its box's lower corner) with the cells' counts, and its range of the walk, the
// cells of [lo - E, hi] (widened by a relative 1e-12 against rounding): first cell, steps along the fast
// axis, rows along the other two.
__global__ void k_cell_count(const double* __restrict__ box, long long ne, const Grid* __restrict__ gp,
                             int32_t* __restrict__ ecell, int32_t* __restrict__ ccnt, int4* __restrict__ range) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const Grid g = *gp;
  int lin = 0, base = 0, n[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double lo = box[6 * e + c], hi = box[6 * e + 3 + c];
    lin += cell_coord(g, c, lo) * g.stride[c];
    const int c0 = cell_coord(g, c, xsub(xsub(lo, g.emax[c]), 1e-12 * (fabs(lo) + g.emax[c])));
    n[c] = cell_coord(g, c, hi) - c0;
    base += c0 * g.stride[c];
  }
  ecell[e] = lin;
  atomicAdd(&ccnt[lin], 1);
  const int a = g.f == 0 ? 1 : 0, b = g.f == 2 ? 1 : 2;
  const bool any = n[0] >= 0 && n[1] >= 0 && n[2] >= 0;  // a box turned round may have none
  range[e] = any ? make_int4(base, n[g.f] + 1, n[a] + 1, n[b] + 1) : make_int4(0, 0, 0, 0);
}

// counting sort of the segments by cell (the counts run down to zero)
__global__ void k_cell_scatter(long long ne, const int32_t* __restrict__ ecell, const int32_t* __restrict__ cstart,
                               int32_t* __restrict__ ccnt, int32_t* __restrict__ segs) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int c = ecell[e];
  segs[cstart[c] + atomicSub(&ccnt[c], 1) - 1] = (int32_t)e;
}

// The float boxes in the order of the cells, each cell's in ascending order of the segments (each thread finds
// its entry's rank among the cell's; cells of more than CELL_SORTED entries keep the order of the scatter), so
// that a row of cells is read as one run.  The last word of a box is its segment.
constexpr int CELL_SORTED = 64;
__global__ void k_cell_boxes(long long ne, const int32_t* __restrict__ segs, const int32_t* __restrict__ ecell,
                             const int32_t* __restrict__ cstart, const float4* __restrict__ boxf,
                             float4* __restrict__ sorted) {
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= ne) return;
  const int e = segs[x], c = ecell[e], lo = cstart[c], hi = cstart[c + 1];
  long long at = x;
  if (hi - lo <= CELL_SORTED) {
    at = lo;
    for (int y = lo; y < hi; ++y) at += segs[y] < e;
  }
  const float4 l = boxf[2LL * e];
  float4 h = boxf[2LL * e + 1];
  h.w = __int_as_float(e);
  sorted[2 * at] = l;
  sorted[2 * at + 1] = h;
}

// the neighbouring floats above and below x (finite x): the outward-rounded float bounds lf <= lo, hf >= hi
// of a box satisfy lo <= up1(lf) and hi >= dn1(hf), so boxes whose up1/dn1-shrunk float bounds overlap
// certainly overlap in FP64 as well
XK_D float up1(float x) {
  const int b = __float_as_int(x);
  return __int_as_float(x == 0.f ? 1 : (x > 0.f ? b + 1 : b - 1));
}
XK_D float dn1(float x) {
  const int b = __float_as_int(x);
  return __int_as_float(x == 0.f ? (int)0x80000001 : (x > 0.f ? b - 1 : b + 1));
}

// the FP64 boxes of i and j (six doubles at box + 6 k, 16-byte aligned) overlap, closed
XK_D bool overlap(const double* __restrict__ box, int i, int j) {
  const double2* bi = reinterpret_cast<const double2*>(box + 6LL * i);
  const double2* bj = reinterpret_cast<const double2*>(box + 6LL * j);
  const double2 a = __ldg(bi), b = __ldg(bi + 1), c = __ldg(bi + 2);  // lo x,y | lo z, hi x | hi y,z
  const double2 p = __ldg(bj), q = __ldg(bj + 1), r = __ldg(bj + 2);
  return a.x <= q.y && p.x <= b.y && a.y <= r.x && p.y <= c.x && b.x <= r.y && q.x <= c.y;
}

// A warp per segment i.  The rows of its range are taken 32 at a time: lane l reads row l's entry range (its
// cells are consecutive), a warp scan lays the ranges of the rows that have entries out as one list, and the
// warp walks it 64 entries at a time: the rows that begin in a window of 32 entries are a bit mask, so a lane
// finds its entry's row by a population count.  An entry
// j > i is screened on the outward-rounded float boxes (which can never reject an FP64 overlap), tested on
// the FP64 boxes where those are not certain, then the shared-node and same-layer filters apply and hits are
// compacted with ballot/popc into segment i's slot list (the first `cap` of them; cnt[i] counts them all,
// raw[i] the overlaps).  Unless all radii are equal, also the sum of r_i + r_j over its kept candidates (each
// lane sums its own entries in walk order, then a fixed butterfly: rsum[i], for the prescreen margin).
// UNIFORM: all radii equal, no radius sums (predicated off they would still issue on the FP64 pipe).
template <bool UNIFORM>
XK_D void sweep(const xk_mesh& m, const double* __restrict__ box,
                                                   const float4* __restrict__ boxf, const float4* __restrict__ sorted,
                                                   const Grid* __restrict__ gp, const int4* __restrict__ range,
                                                   const int32_t* __restrict__ cstart, int excl_shared,
                                                   int excl_layer, int cap, int32_t* __restrict__ slot,
                                                   int32_t* __restrict__ cnt, int32_t* __restrict__ raw,
                                                   double* __restrict__ rsum, int* offs) {
  const long long ne = m.n_elems;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ne) return;
  const int i = (int)w;
  const int4 rg = range[i];
  const int f = gp->f, sa = gp->stride[f == 0 ? 1 : 0], sb = gp->stride[f == 2 ? 1 : 2];
  const int rows = rg.z * rg.w;
  const int2* conn2 = reinterpret_cast<const int2*>(m.conn);
  const int2 ci = __ldg(conn2 + i);
  const int li = (excl_layer && m.layer) ? m.layer[i] : -1;
  const float4 il = boxf[2LL * i], ih = boxf[2LL * i + 1];
  // an outward float overlap is an FP64 overlap when the boxes shrunk by one float step each still overlap
  // (a <= dn1(b) is up1(a) <= b: both steps are taken on box i); only the rare pair between the two takes the
  // FP64 boxes
  const float ux = up1(up1(il.x)), uy = up1(up1(il.y)), uz = up1(up1(il.z));
  const float vx = dn1(dn1(ih.x)), vy = dn1(dn1(ih.y)), vz = dn1(dn1(ih.z));
  int32_t* const my = slot + (long long)i * cap;
  const unsigned below = (1u << lane) - 1u;
  int n_raw = 0, n_keep = 0;  // n_raw: this lane's overlaps
  double rs = 0.0;
  for (int rb = 0; rb < rows; rb += 32) {
    // this lane's row of the batch and its entry range
    int s0 = 0, n0 = 0;
    const int q0 = rb + lane;
    if (q0 < rows) {
      const int c = rg.x + (q0 % rg.z) * sa + (q0 / rg.z) * sb;
      s0 = cstart[c];
      n0 = cstart[c + rg.y] - s0;
    }
    int incl = n0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int pre = incl - n0;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    // offs[r]: the offset from list position to sorted position of the r-th row that has entries
    const unsigned some = __ballot_sync(0xffffffffu, n0 > 0);
    __syncwarp();
    if (n0 > 0) offs[__popc(some & below)] = s0 - pre;
    __syncwarp();
    int before = -1;  // rows begun before the window, less one
    auto entry = [&](int f0) {  // sorted position of this lane's entry of the window at f0 (any past the list)
      const unsigned d = (unsigned)(pre - f0);
      const unsigned begun = __reduce_or_sync(0xffffffffu, n0 > 0 && d < 32u ? 1u << d : 0u);
      const int r = before + __popc(begun & (below | (1u << lane)));
      before += __popc(begun);
      return offs[r & 31] + f0 + lane;
    };
    auto hit_of = [&](const float4& jl, const float4& jh) {
      if (!(il.x <= jh.x && jl.x <= ih.x && il.y <= jh.y && jl.y <= ih.y && il.z <= jh.z && jl.z <= ih.z))
        return false;
      const bool sure = ux <= jh.x && jl.x <= vx && uy <= jh.y && jl.y <= vy && uz <= jh.z && jl.z <= vz;
      return sure || overlap(box, i, __float_as_int(jh.w));
    };
    auto keep = [&](bool hit, const float4& jl, const float4& jh) {
      if (!hit || (li >= 0 && __float_as_int(jl.w) == li)) return false;
      if (!excl_shared) return true;
      const int2 cj = __ldg(conn2 + __float_as_int(jh.w));
      return !(ci.x == cj.x || ci.x == cj.y || ci.y == cj.x || ci.y == cj.y);
    };
    auto put = [&](bool kept, int j) {
      const unsigned bal = __ballot_sync(0xffffffffu, kept);
      if (kept) {
        if (!UNIFORM) rs = xadd(rs, xadd(m.radii[i], m.radii[j]));  // this lane's entries, in walk order
        const int at = n_keep + __popc(bal & below);
        if (at < cap) my[at] = j;
      }
      n_keep += __popc(bal);
    };
    // two entries per lane and pass, their loads issued together; each lane meets its entries in increasing order
    for (int f0 = 0; f0 < total; f0 += 64) {
      const int pA = entry(f0), pB = entry(f0 + 32);
      const bool inA = f0 + lane < total, inB = f0 + 32 + lane < total;
      float4 al, ah, bl, bh;
      al = bl = make_float4(0.f, 0.f, 0.f, 0.f);
      ah = bh = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
      if (inA) { al = __ldg(sorted + 2LL * pA); ah = __ldg(sorted + 2LL * pA + 1); }
      if (inB) { bl = __ldg(sorted + 2LL * pB); bh = __ldg(sorted + 2LL * pB + 1); }
      const int jA = __float_as_int(ah.w), jB = __float_as_int(bh.w);
      const bool hitA = jA > i && hit_of(al, ah), hitB = jB > i && hit_of(bl, bh);
      n_raw += (int)hitA + (int)hitB;
      const bool keptA = keep(hitA, al, ah), keptB = keep(hitB, bl, bh);
      put(keptA, jA);
      put(keptB, jB);
    }
  }
  n_raw = __reduce_add_sync(0xffffffffu, n_raw);
  if (!UNIFORM) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);  // fixed butterfly order
  }
  if (lane == 0) {
    cnt[i] = n_keep;
    raw[i] = n_raw;
    if (!UNIFORM) rsum[i] = rs;
  }
}

__global__ void __launch_bounds__(BP_T, 8) k_sweep(xk_mesh m, const double* __restrict__ box,
                                                   const float4* __restrict__ boxf, const float4* __restrict__ sorted,
                                                   const Grid* __restrict__ gp, const int4* __restrict__ range,
                                                   const int32_t* __restrict__ cstart, int excl_shared,
                                                   int excl_layer, int cap, int32_t* __restrict__ slot,
                                                   int32_t* __restrict__ cnt, int32_t* __restrict__ raw,
                                                   double* __restrict__ rsum) {
  __shared__ int s_off[BP_T / 32][32];
  int* const offs = s_off[threadIdx.x >> 5];
  if (gp->uniform)
    sweep<true>(m, box, boxf, sorted, gp, range, cstart, excl_shared, excl_layer, cap, slot, cnt, raw, rsum, offs);
  else
    sweep<false>(m, box, boxf, sorted, gp, range, cstart, excl_shared, excl_layer, cap, slot, cnt, raw, rsum, offs);
}

// Totals over the segments (overlaps, candidates before the prescreen, the longest slot list) and the
// prescreen margin: mean(r_a + r_b) / 2 over the candidates after the shared-node and same-layer filters
// (_manager_process.py:275-279) from the per-segment sums, in a fixed order (a tree in every block, the last
// block over the blocks), or the common radius.
// RED_BLOCKS is this GPU's number of SMs, but fixed: the order of the sums follows from it.
constexpr int RED_BLOCKS = 152, RED_T = 256;
__global__ void __launch_bounds__(RED_T) k_totals(const int32_t* __restrict__ cnt, const int32_t* __restrict__ raw,
                                                  const double* __restrict__ rsum, long long ne,
                                                  const Grid* __restrict__ gp, double fixed, double* __restrict__ part,
                                                  Words* __restrict__ w) {
  __shared__ double sm[RED_T];
  __shared__ bool s_last;
  const bool sums = !(fixed > 0.0) && !gp->uniform;
  double acc = 0.0;
  long long c = 0, r = 0;
  int mx = 0;
  for (long long k = (long long)blockIdx.x * RED_T + threadIdx.x; k < ne; k += (long long)RED_BLOCKS * RED_T) {
    const int v = cnt[k];
    c += v;
    r += raw[k];
    mx = v > mx ? v : mx;
    if (sums) acc += rsum[k];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c += __shfl_down_sync(0xffffffffu, c, o);
    r += __shfl_down_sync(0xffffffffu, r, o);
    const int y = __shfl_down_sync(0xffffffffu, mx, o);
    mx = y > mx ? y : mx;
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(reinterpret_cast<unsigned long long*>(&w->pre), (unsigned long long)c);
    atomicAdd(reinterpret_cast<unsigned long long*>(&w->raw), (unsigned long long)r);
    atomicMax(reinterpret_cast<unsigned long long*>(&w->longest), (unsigned long long)mx);
  }
  auto tree = [&](double v) {
    sm[threadIdx.x] = v;
    __syncthreads();
    for (int h = RED_T / 2; h > 0; h >>= 1) {
      if (threadIdx.x < h) sm[threadIdx.x] += sm[threadIdx.x + h];
      __syncthreads();
    }
    return sm[0];
  };
  if (sums) {
    const double v = tree(acc);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&w->ticket2, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double margin = fixed;
  if (!(fixed > 0.0)) {
    const long long n = *(volatile long long*)&w->pre;
    if (sums) {
      __syncthreads();
      const double v = tree(threadIdx.x < RED_BLOCKS ? __ldcg(part + threadIdx.x) : 0.0);
      margin = n > 0 ? xmul(xdiv(v, (double)n), 0.5) : 0.0;
    } else {
      margin = n > 0 ? xmul(xadd(gp->radius, gp->radius), 0.5) : 0.0;
    }
  }
  if (threadIdx.x == 0) {
    w->margin = margin;
    w->ticket2 = 0u;  // the walk may be repeated
  }
}

// Midpoint prescreen of DetectCandidatesProcess (_manager_process.py:260-286) for the pair (i, j), from
// the segments' midpoints and half lengths: keep when max(0, |m_i - m_j| - h_i - h_j) <= r_i + r_j +
// extra, in the reference's operation order.
XK_D bool midpoint_keep(const double4_32a a, const double4_32a b, double ra, double rb, double extra) {
  const double dm[3] = {xsub(a.x, b.x), xsub(a.y, b.y), xsub(a.z, b.z)};
  const double md = xsqrt(xdot_seq(dm, dm));
  double mp = xsub(xsub(md, a.w), b.w);
  mp = (mp > 0.0 || mp != mp) ? mp : 0.0;
  return mp <= xadd(xadd(ra, rb), extra);
}

// The same decision with a float screen first: the separation |m_i - m_j| from the split midpoints against the
// threshold r_i + r_j + extra + h_i + h_j in float decides every pair farther from it than a relative 1e-5 (the
// float roundings of both stay below 1e-6) and than `slack`; the rest, and what is not finite, take the exact
// routine, so the decision is the exact one.  slack: what the split midpoints do not resolve.  A low part is rounded
// at 2^-48 of its position and the difference of two at 2^-47 of the larger, 2^-46 a component in all, so 2^-45 of
// m_i's largest component covers the three (m_j's exceeds it by the separation at most, far below the relative part).
XK_D float split_slack(const MidF& a) {
  return 2.8421709e-14f * fmaxf(fabsf(a.hi[0]), fmaxf(fabsf(a.hi[1]), fabsf(a.hi[2])));
}
XK_D bool midpoint_keep_fast(const MidF& a, const MidF& b, float extra, float slack,
                             const double4_32a* __restrict__ mid, int i, int j, const double* __restrict__ radii,
                             double extra64) {
  const float dx = (a.hi[0] - b.hi[0]) + (a.lo[0] - b.lo[0]), dy = (a.hi[1] - b.hi[1]) + (a.lo[1] - b.lo[1]),
              dz = (a.hi[2] - b.hi[2]) + (a.lo[2] - b.lo[2]);
  const float md = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
  const float thr = ((a.r + b.r) + extra) + (a.half + b.half);
  if (md < fmaf(thr, 0.99999f, -slack)) return true;
  if (md > fmaf(thr, 1.00001f, slack)) return false;
  return midpoint_keep(mid[i], mid[j], radii[i], radii[j], extra64);
}

// A warp per segment: its slot list sorted by j (a rank sort; the j are distinct), the prescreen
// applied (if wanted), written to srt as j (kept) or ~j (dropped); cnt2[i] = kept count.
__global__ void __launch_bounds__(BP_T) k_slots_rank(xk_mesh m, const double4_32a* __restrict__ mid,
                                                     const MidF* __restrict__ midf, const int32_t* __restrict__ slot,
                                                     const int32_t* __restrict__ cnt, int cap, int prescreen,
                                                     const Words* __restrict__ words, int32_t* __restrict__ srt,
                                                     int32_t* __restrict__ cnt2) {
  const long long ne = m.n_elems;
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ne) return;
  const int i = (int)w;
  const int n = cnt[i] < cap ? cnt[i] : cap;
  const int32_t* const my = slot + (long long)i * cap;
  int32_t* const out = srt + (long long)i * cap;
  const MidF mi = midf[i];
  const double ex = words->margin;
  const float exf = xk_d2f(ex), slack = split_slack(mi);
  auto keep = [&](int j) {
    return !prescreen || midpoint_keep_fast(mi, midf[j], exf, slack, mid, i, j, m.radii, ex);
  };
  int kept = 0;
  if (n <= 64) {  // two entries per lane, ranked by shuffle-broadcast comparisons
    const int v0 = lane < n ? my[lane] : 0x7fffffff;
    const int v1 = lane + 32 < n ? my[lane + 32] : 0x7fffffff;
    bool k0 = false, k1 = false;
    if (lane < n) k0 = keep(v0);
    if (lane + 32 < n) k1 = keep(v1);
    int r0 = 0, r1 = 0;
    const int n0 = n < 32 ? n : 32;
    for (int k = 0; k < n0; ++k) {
      const int x = __shfl_sync(0xffffffffu, v0, k);
      r0 += x < v0;
      r1 += x < v1;
    }
    for (int k = 0; k < n - 32; ++k) {
      const int x = __shfl_sync(0xffffffffu, v1, k);
      r0 += x < v0;
      r1 += x < v1;
    }
    if (lane < n) out[r0] = k0 ? v0 : ~v0;
    if (lane + 32 < n) out[r1] = k1 ? v1 : ~v1;
    kept = k0 + k1;
  } else for (int l = lane; l < n; l += 32) {
    const int v = my[l];
    int r = 0;
    for (int q = 0; q < n; ++q) r += my[q] < v;
    const bool k = keep(v);
    out[r] = k ? v : ~v;
    kept += k;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) kept += __shfl_xor_sync(0xffffffffu, kept, o);
  if (lane == 0) cnt2[i] = kept;
}

// A warp per segment: its kept pairs, in order, at off2[i] of out (rows (i, j); at most cap_out rows).
__global__ void __launch_bounds__(BP_T) k_slots_emit(long long ne, const int32_t* __restrict__ srt,
                                                     const int32_t* __restrict__ cnt, int cap,
                                                     const int32_t* __restrict__ off2, long long cap_out,
                                                     int32_t* __restrict__ out) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ne) return;
  const int i = (int)w;
  const int n = cnt[i] < cap ? cnt[i] : cap;
  const int32_t* const my = srt + (long long)i * cap;
  long long at = off2[i];
  for (int l0 = 0; l0 < n; l0 += 32) {
    const int l = l0 + lane;
    const int v = l < n ? my[l] : -1;
    const unsigned bal = __ballot_sync(0xffffffffu, v >= 0);
    const long long d = at + __popc(bal & ((1u << lane) - 1u));
    if (v >= 0 && d >= 0 && d < cap_out) {
      out[2 * d] = i;
      out[2 * d + 1] = v;
    }
    at += __popc(bal);
  }
}

// ------------------------------------------------------------------------- merge


// The first row of a list sorted by a (read at stride S) whose a >= s: eight-way steps, whose seven loads wait
// together (a binary search's twenty wait in turn).
template <int S>
XK_D int32_t row_start(const int32_t* __restrict__ a, long long n, long long s) {
  long long lo = 0, hi = n;  // rows below lo are < s, rows from hi on are >= s
  while (hi - lo > 8) {
    const long long step = (hi - lo) >> 3;
    int32_t v[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) v[k] = a[S * (lo + (k + 1) * step)];
    int less = 0;
#pragma unroll
    for (int k = 0; k < 7; ++k) less += v[k] < s;
    if (less < 7) hi = lo + (less + 1) * step;
    if (less > 0) lo += less * step + 1;
  }
  int less = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) less += lo + k < hi && a[S * (lo + k)] < s;
  return (int32_t)(lo + less);
}

// Row ranges of the segments, s in [0, ne]: ostart of the table, cstart of the candidate rows.
__global__ void k_seg_starts(const int32_t* __restrict__ old, long long no, const int32_t* __restrict__ cand,
                             long long nc, long long ne, int32_t* __restrict__ ostart, int32_t* __restrict__ cstart) {
  const long long x = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (x <= ne) ostart[x] = row_start<1>(old, no, x);
  else if (x <= 2 * ne + 1) cstart[x - ne - 1] = row_start<2>(cand, nc, x - ne - 1);
}

// A warp per segment: which of its old rows stay as old-only (INACTIVE) pairs (not a candidate, and with DROP not
// pristine either: status INACTIVE, p_n = k_pen = 0, z_t = 0), one bit each, 32 rows a word; cnt = rows of the
// merged segment.  The words of segment w stand from (ostart[w] >> 5) + w on: segments do not share one.
XK_D long long stay_word(long long o0, long long w) { return (o0 >> 5) + w; }

// A segment's list of b, in a warp's shared memory where it fits (a search there is a few dozen clocks a step, in
// global memory a few hundred until its lines have come: k_merge_count 36 -> 30 us, k_merge_order 49 -> 40 us at the
// 1027-wire strand).  rank(key): the entries below key.
constexpr int SEG_LIST = 128;
struct SegList {
  const int32_t* g;  // entry k at g[S k]
  const int* s;      // or at s[k]
  int S, n;
  XK_D int at(int k) const { return s ? s[k] : g[(long long)S * k]; }
  XK_D int rank(int key) const {
    int lo = 0, hi = n;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (at(mid) < key) lo = mid + 1; else hi = mid;
    }
    return lo;
  }
};
XK_D SegList seg_list(const int32_t* g, int S, int n, int* buf, int lane) {
  SegList r{g, n <= SEG_LIST ? buf : nullptr, S, n};
  if (r.s)
    for (int k = lane; k < n; k += 32) buf[k] = g[(long long)S * k];
  return r;
}
template <bool DROP>
__global__ void __launch_bounds__(BP_T) k_merge_count(xk_pairs old, const int32_t* __restrict__ cand,
                                                      const int32_t* __restrict__ ostart,
                                                      const int32_t* __restrict__ cstart, long long ne,
                                                      unsigned* __restrict__ stay, int32_t* __restrict__ cnt) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ne) return;
  __shared__ int buf[BP_T / 32][SEG_LIST];
  const long long o0 = ostart[w], o1 = ostart[w + 1], c0 = cstart[w], c1 = cstart[w + 1];
  int n = (int)(c1 - c0);
  const SegList cl = seg_list(cand + 2 * c0 + 1, 2, n, buf[threadIdx.x >> 5], lane);
  __syncwarp();
  for (long long j = 0; o0 + 32 * j < o1; ++j) {
    const long long o = o0 + 32 * j + lane;
    bool stays = false;
    if (o < o1) {
      const int b = old.eb[o], l = cl.rank(b);
      stays = !(l < cl.n && cl.at(l) == b);
      if (DROP && stays)
        stays = old.status[o] != 0 || old.p_n[o] != 0.0 || old.k_pen[o] != 0.0 || old.z_t[o] != 0.0 ||
                old.z_t[old.cap + o] != 0.0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, stays);
    if (lane == 0) stay[stay_word(o0, w) + j] = m;
    n += __popc(m);
  }
  if (lane == 0) cnt[w] = n;
}

// A warp per segment: ea, eb and source of its merged rows in order of eb.  src: the old row it continues, or
// MERGE_NEW, or MERGE_OLD - o for the old-only row o.
__global__ void __launch_bounds__(BP_T) k_merge_order(xk_pairs old, const int32_t* __restrict__ cand,
                                                      const int32_t* __restrict__ ostart,
                                                      const int32_t* __restrict__ cstart, long long ne,
                                                      const unsigned* __restrict__ stay,
                                                      const int32_t* __restrict__ off, int32_t* __restrict__ ea,
                                                      int32_t* __restrict__ eb, int32_t* __restrict__ src) {
  const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= ne) return;
  const long long o0 = ostart[w], o1 = ostart[w + 1], c0 = cstart[w], c1 = cstart[w + 1], base = off[w];
  const unsigned* const words = stay + stay_word(o0, w);
  __shared__ int buf[BP_T / 32][2][SEG_LIST];
  int(*const mine)[SEG_LIST] = buf[threadIdx.x >> 5];
  const SegList cl = seg_list(cand + 2 * c0 + 1, 2, (int)(c1 - c0), mine[0], lane);
  const SegList ol = seg_list(old.eb + o0, 1, (int)(o1 - o0), mine[1], lane);
  __syncwarp();
  for (int k = lane; k < cl.n; k += 32) {
    const int b = cl.at(k), lo = ol.rank(b);
    long long pos = base + k;
    for (int j = 0; 32 * j < lo; ++j) {  // old-only rows before it
      const int below = lo - 32 * j;
      pos += __popc(words[j] & (below >= 32 ? 0xffffffffu : (1u << below) - 1u));
    }
    ea[pos] = (int)w;
    eb[pos] = b;
    src[pos] = lo < ol.n && ol.at(lo) == b ? (int32_t)(o0 + lo) : MERGE_NEW;
  }
  int before = 0;
  for (int j = 0; 32 * j < ol.n; ++j) {
    const unsigned m = words[j];
    if ((m >> lane) & 1u) {
      const int b = ol.at(32 * j + lane);
      const long long pos = base + before + __popc(m & ((1u << lane) - 1u)) + cl.rank(b);
      ea[pos] = (int)w;
      eb[pos] = b;
      src[pos] = MERGE_OLD - (int32_t)(o0 + 32 * j + lane);
    }
    before += __popc(m);
  }
}

}  // namespace

// slot-list length of the walk: grows to the longest list seen (a power of two), kept for later calls
std::atomic<int> g_slot_cap{32};

extern "C" xk_status xk_broadphase_queued(const xk_mesh* m, const double* u, const xk_bp_params* bp,
                                          int32_t* out_pairs, int64_t cap, int64_t* n_out, int64_t* n_raw,
                                          int64_t* n_prefilter, xk_stream s) {
  if (!m || !bp || !n_out) return xk_set_error(XK_ERR_ARG, "xk_broadphase: null argument");
  cudaStream_t st = (cudaStream_t)s;
  *n_out = 0;
  if (n_raw) *n_raw = 0;
  if (n_prefilter) *n_prefilter = 0;
  const long long ne = m->n_elems;
  if (ne < 2) return XK_OK;
  if (ne > 0x7fffffffLL) return xk_set_error(XK_ERR_OVERFLOW, "xk_broadphase: more than 2^31 segments");
  // the grid has at most cap_cells cells, so the cell arrays are sized without reading it back
  const long long cap_cells = ne * 8 > 4096 ? ne * 8 : 4096;
  int slot_cap = g_slot_cap.load();
  XkScratch S(st);
  if ((double)ne * slot_cap * 8.0 <= 64.0e9)  // one allocation for the usual case: boxes, cells, lists, scans
    XK_TRY(S.reserve((size_t)ne * (48 + 32 + 32 + 32 + 32 + 16 + 8 + 16 + 8 + 8 * (size_t)slot_cap) +
                     (size_t)cap_cells * 9 + (1 << 16)));
  Words* words;
  int32_t *ccnt, *segs, *cstart, *cnt, *raw, *cnt2, *off2, *ecell;
  double *box, *rsum, *part;
  float4 *boxf, *sorted;
  double4_32a* mid;
  MidF* midf;
  int4* range;
  Grid* grid;
  // the words and the cell counts start at zero: they stand together
  char* zero;
  const size_t words_bytes = XkScratch::padded(sizeof(Words)), zero_bytes = words_bytes + sizeof(int32_t) * (cap_cells + 1);
  XK_TRY(S.get(&zero, (long long)zero_bytes));
  words = reinterpret_cast<Words*>(zero);
  ccnt = reinterpret_cast<int32_t*>(zero + words_bytes);
  XK_TRY(S.get(&box, 6 * ne));
  XK_TRY(S.get(&boxf, 2 * ne));
  XK_TRY(S.get(&sorted, 2 * ne));
  XK_TRY(S.get(&mid, ne));
  XK_TRY(S.get(&midf, ne));
  XK_TRY(S.get(&range, ne));
  XK_TRY(S.get(&grid, 1));
  XK_TRY(S.get(&ecell, ne));
  XK_TRY(S.get(&segs, ne));
  XK_TRY(S.get(&cstart, cap_cells + 1));
  XK_TRY(S.get(&cnt, ne + 1));
  XK_TRY(S.get(&raw, ne + 1));
  XK_TRY(S.get(&cnt2, ne + 1));
  XK_TRY(S.get(&off2, ne + 1));
  XK_TRY(S.get(&rsum, ne));
  XK_TRY(S.get(&part, RED_BLOCKS));
  XK_CUDA(cudaMemsetAsync(zero, 0, zero_bytes, st));
  if (ne >= 2LL * xk_sm_count() * 256)
    k_aabb<256><<<xk_blocks(ne, 256), 256, 0, st>>>(*m, u, bp->margin, box, boxf, mid, midf, words, cap_cells,
                                                    bp->cell_size, grid);
  else
    k_aabb<64><<<xk_blocks(ne, 64), 64, 0, st>>>(*m, u, bp->margin, box, boxf, mid, midf, words, cap_cells,
                                                 bp->cell_size, grid);
  // segments sorted by the cell of their lower corner
  k_cell_count<<<xk_blocks(ne, 64), 64, 0, st>>>(box, ne, grid, ecell, ccnt, range);
  XK_CHECK_LAUNCH();
  XK_TRY(xk_exclusive_scan_i32(ccnt, cstart, cap_cells + 1, nullptr, st, &S));
  k_cell_scatter<<<xk_blocks(ne, 256), 256, 0, st>>>(ne, ecell, cstart, ccnt, segs);
  k_cell_boxes<<<xk_blocks(ne, 256), 256, 0, st>>>(ne, segs, ecell, cstart, boxf, sorted);
  XK_CHECK_LAUNCH();
  const int warp_blocks = xk_blocks(ne * 32, BP_T);
  const int excl_layer = (bp->exclude_same_layer && m->layer) ? 1 : 0;
  for (int attempt = 0;; ++attempt) {
    if ((double)ne * slot_cap * 8.0 > 64.0e9)
      return xk_set_error(XK_ERR_OVERFLOW, "xk_broadphase: candidate lists too long for the slot buffers");
    int32_t *slot, *srt;
    XK_TRY(S.get(&slot, ne * slot_cap));
    XK_TRY(S.get(&srt, ne * slot_cap));
    if (attempt > 0) XK_CUDA(cudaMemsetAsync(&words->raw, 0, 4 * sizeof(long long), st));
    k_sweep<<<warp_blocks, BP_T, 0, st>>>(*m, box, boxf, sorted, grid, range, cstart, bp->exclude_shared, excl_layer,
                                          slot_cap, slot, cnt, raw, rsum);
    k_totals<<<RED_BLOCKS, RED_T, 0, st>>>(cnt, raw, rsum, ne, grid, bp->prescreening_margin, part, words);
    k_slots_rank<<<warp_blocks, BP_T, 0, st>>>(*m, mid, midf, slot, cnt, slot_cap, bp->midpoint_prescreening ? 1 : 0,
                                               words, srt, cnt2);
    XK_CHECK_LAUNCH();
    XK_TRY(xk_exclusive_scan_i32(cnt2, off2, ne, reinterpret_cast<int64_t*>(&words->kept), st, &S));
    int64_t h[4];  // raw, pre, longest, kept
    static_assert(offsetof(Words, kept) - offsetof(Words, raw) == 3 * sizeof(int64_t), "four words in a row");
    XK_TRY(xk_read_begin(reinterpret_cast<const int64_t*>(&words->raw), 4, st));
    k_slots_emit<<<warp_blocks, BP_T, 0, st>>>(ne, srt, cnt, slot_cap, off2, cap, out_pairs);
    XK_CHECK_LAUNCH();
    XK_TRY(xk_read_end(h, 4));
    const int longest = (int)h[2];
    if (longest > slot_cap) {  // some lists were cut short: walk again with lists long enough for all
      if (attempt > 0) return xk_set_error(XK_ERR_OVERFLOW, "xk_broadphase: slot lists overflowed twice");
      int c = slot_cap;
      while (c < longest) c *= 2;
      slot_cap = c;
      int prev = g_slot_cap.load();
      while (prev < c && !g_slot_cap.compare_exchange_weak(prev, c)) {
      }
      continue;
    }
    if (h[3] > 0x7fffffffLL) return xk_set_error(XK_ERR_OVERFLOW, "xk_broadphase: more than 2^31 candidates");
    if (n_raw) *n_raw = h[0];
    if (n_prefilter) *n_prefilter = h[1];
    *n_out = h[3];
    if (h[3] > cap) {
      XK_CUDA(cudaStreamSynchronize(st));  // the caller may free the rows
      return xk_set_error(XK_ERR_CAPACITY, "xk_broadphase: output capacity too small");
    }
    return XK_OK;
  }
}

extern "C" xk_status xk_broadphase(const xk_mesh* m, const double* u, const xk_bp_params* bp, int32_t* out_pairs,
                                   int64_t cap, int64_t* n_out, int64_t* n_raw, int64_t* n_prefilter, xk_stream s) {
  const xk_status r = xk_broadphase_queued(m, u, bp, out_pairs, cap, n_out, n_raw, n_prefilter, s);
  if (r == XK_OK) XK_CUDA(cudaStreamSynchronize((cudaStream_t)s));
  return r;
}

// The merged rows' order first (two lists of a few dozen rows per segment), then one kernel moves every row's state
// (pair.cu), with the detection's narrowphase on the way where that is the screened one.
// A thread per old row and one per candidate, as before, took two passes over the whole table, a scan of its rows
// and, in a mixed detection, two more passes for the float state and the narrowphase.
// Measured at the 1027-wire strand (3.2M rows), mixed: 580 us in eight launches -> 310 us in six.
static xk_status merge_impl(const xk_mesh* m, const xk_pairs* old, const int32_t* cands, int64_t n_cands,
                            xk_pairs* out, xk_stream s, bool drop, const MergeScreen* screen = nullptr) {
  if (!m || !old || !out || (n_cands > 0 && !cands)) return xk_set_error(XK_ERR_ARG, "xk_pairs_merge: null argument");
  if ((long long)out->cap < (long long)old->n + n_cands)
    return xk_set_error(XK_ERR_CAPACITY, "xk_pairs_merge: out->cap < old->n + n_cands");
  cudaStream_t st = (cudaStream_t)s;
  XkScratch S(st);
  int32_t *cnt, *off, *ostart, *cstart, *src, *list = nullptr;
  unsigned* stay;
  int64_t* tot;
  const long long ne = m->n_elems, most = (long long)old->n + n_cands, words = old->n / 32 + ne + 1;
  XK_TRY(S.reserve(4 * (size_t)(4 * ne + most * (screen ? 2 : 1) + words) + 16 * (size_t)(ne / 512) + 16384));
  XK_TRY(S.get(&cnt, ne + 1));
  XK_TRY(S.get(&off, ne + 1));
  XK_TRY(S.get(&ostart, ne + 1));
  XK_TRY(S.get(&cstart, ne + 1));
  XK_TRY(S.get(&src, most));
  XK_TRY(S.get(&stay, words));
  XK_TRY(S.get(&tot, 1));
  if (screen) XK_TRY(S.get(&list, most + 1));
  int64_t h = 0;
  if (ne > 0) {
    const int warp_blocks = xk_blocks(ne * 32, BP_T);
    k_seg_starts<<<xk_blocks(2 * ne + 2, 128), 128, 0, st>>>(old->ea, old->n, cands, n_cands, ne, ostart, cstart);
    if (drop)
      k_merge_count<true><<<warp_blocks, BP_T, 0, st>>>(*old, cands, ostart, cstart, ne, stay, cnt);
    else
      k_merge_count<false><<<warp_blocks, BP_T, 0, st>>>(*old, cands, ostart, cstart, ne, stay, cnt);
    XK_CHECK_LAUNCH();
    XK_TRY(xk_exclusive_scan_i32(cnt, off, ne, tot, st, &S));
    XK_TRY(xk_read_begin(tot, 1, st));
    k_merge_order<<<warp_blocks, BP_T, 0, st>>>(*old, cands, ostart, cstart, ne, stay, off, out->ea, out->eb, src);
    XK_CHECK_LAUNCH();
    XK_TRY(xk_merge_rows(m, old, src, tot, most, out, screen, list, st));
    XK_TRY(xk_read_end(&h, 1));
  }
  out->n = (int32_t)h;
  return XK_OK;
}

extern "C" xk_status xk_pairs_merge_queued(const xk_mesh* m, const xk_pairs* old, const int32_t* cands,
                                           int64_t n_cands, xk_pairs* out, int drop, xk_stream s) {
  return merge_impl(m, old, cands, n_cands, out, s, drop != 0);
}

extern "C" xk_status xk_pairs_merge(const xk_mesh* m, const xk_pairs* old, const int32_t* cands, int64_t n_cands,
                                    xk_pairs* out, xk_stream s) {
  XK_TRY(merge_impl(m, old, cands, n_cands, out, s, false));
  XK_CUDA(cudaStreamSynchronize((cudaStream_t)s));
  return XK_OK;
}

extern "C" xk_status xk_pairs_merge_pruned(const xk_mesh* m, const xk_pairs* old, const int32_t* cands,
                                           int64_t n_cands, xk_pairs* out, xk_stream s) {
  XK_TRY(merge_impl(m, old, cands, n_cands, out, s, true));
  XK_CUDA(cudaStreamSynchronize((cudaStream_t)s));
  return XK_OK;
}

extern "C" xk_status xk_pairs_merge_screened(const xk_mesh* m, const xk_pairs* old, const xk_pairs32* old32,
                                             const int32_t* cands, int64_t n_cands, xk_pairs* out, int drop,
                                             const double* u, const float* node32, const xk_contact_params* cp,
                                             int32_t* n_exact, xk_stream s) {
  if (!u || !node32 || !cp || !n_exact) return xk_set_error(XK_ERR_ARG, "xk_pairs_merge_screened: null argument");
  if (m && (m->core_radii || (out && out->coat_cc)))
    return xk_set_error(XK_ERR_ARG, "xk_pairs_merge_screened: not for coated wires");
  if (old32 && (drop || !old32->slot || !old || old32->n != old->n))
    return xk_set_error(XK_ERR_ARG, "xk_pairs_merge_screened: the float table needs its slots and the table's rows, "
                                    "and no pruning");
  if (!old32) {
    XK_TRY(merge_impl(m, old, cands, n_cands, out, s, drop != 0));
    return xk_narrowphase_screened(m, out, u, node32, cp, n_exact, s);
  }
  const MergeScreen q{old32, u, node32, cp, n_exact};
  return merge_impl(m, old, cands, n_cands, out, s, false, &q);
}
