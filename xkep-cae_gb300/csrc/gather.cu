// Per-increment contact pattern and the deterministic, atomic-free reduction of
// pair contributions into nodal forces and 3x3 contact-tangent blocks.
//
// The reference scatters per-pair 12-vectors and 12x12 COO blocks and lets
// np.add.at / scipy sum the duplicates (contact_force/strategy.py:161-167,249-253;
// friction/_assembly.py:85-105,119-157,184-257).  Here the pair kernel reduces
// every contributing pair ("member") to a record (s, t, v, B): its force on
// local node k is c_k v and its tangent block (k, l) is c_k c_l B with
// c = [1-s, s, -(1-t), -t].  Each node sums its incident members and each
// K_c block sums its contributor list, both in a fixed order.
//
// Every contribution to block (v, w) is c_k c_l B and the same member gives
// c_l c_k B to block (w, v): the block at (w, v) equals the block at (v, w)
// (the same 3x3 values, not the transpose; K_c itself is not symmetric once
// friction acts).  So the pattern holds the blocks with row <= column only
// ("upper" blocks), each computed once, and a lower index lists, per node w,
// the stored blocks (v, w) with v < w, for readers that need whole rows.
#include "scan.cuh"

xk_status xk_sumsq_into(const double* x, long long n, double* out, cudaStream_t s);

namespace {

template <typename T>
XK_D T shape_c(T s, T t, int k) {
  switch (k) {
    case 0: return T(1) - s;
    case 1: return s;
    case 2: return -(T(1) - t);
    default: return -t;
  }
}

// In double one subtraction, whatever the lanes' k (a switch issues one for every k that a warp has), and the
// sign moved as a bit: the same values.
template <>
XK_D double shape_c<double>(double s, double t, int k) {
  const double x = (k & 2) ? t : s, om = 1.0 - x, c = (k & 1) ? x : om;
  return __hiloint2double(__double2hiint(c) ^ (int)((unsigned)(k & 2) << 30), __double2loint(c));
}

// A pair contributes in the increment when it is not INACTIVE or still carries a normal force; with
// coated wires every pair does, since the reference evaluates the coating force of every pair.
XK_D bool is_member(const xk_pairs& p, long long i) {
  return (p.status[i] != 0) || (p.p_n[i] > 0.0) || (p.coat_cc != nullptr);
}

// ---------------------------------------------------------------------------------------------------------------
// Contact pattern.  Seven launches whose sizes are bounded by the host's (pairs, nodes, elements), so that the
// host waits once, at the end: a kernel that needs the number of members or blocks reads it on the device, and one
// that would run past a capacity writes nothing.
//   members      scan over the pairs: members, their nodes, the other pairs, members per element
//   elements     scans over the elements (elem_ptr) and the nodes (inc_ptr = its elements' members)
//   sides        member sides of each element, in the order the atomics give
//   k_pat_cols   per node: incidences sorted, distinct neighbours sorted, contributions counted;
//                per element: member sides sorted
//   rows         scans over the nodes (row_ptr with the first contribution; low_ptr)
//   k_pat_rows   per node: columns, contributor lists, term lists and lower index of its row
// The incidences of a node are sorted, so a row that places its contributions in that order emits every block's
// list sorted: no list is sorted after it is filled, and none is filled through atomics.  Before, lists were
// counted, scanned, filled and sorted one after another (30 launches, three waits).  GB300, a detection from the
// same state: 37 wires 630 -> 434 us, 397 wires 1190 -> 885, 1027 wires 2330 -> 1752.
// ---------------------------------------------------------------------------------------------------------------

struct Totals {
  int64_t members, blocks, contribs, low;
};

struct MemberScan {
  xk_mesh m;
  xk_pairs p;
  long long cap;  // members that fit
  long long cap_others;
  int32_t *members, *mnodes, *others, *ecnt;
  Totals* tot;
  bool wide;  // status, p_n and mnodes aligned for vector access
  XK_D long long size(int) const { return p.n; }
  XK_D int64_t one(int, long long i) const { return is_member(p, i) ? 1 : 0; }
  XK_D void eight(int, long long i, int64_t* v) const {
    if (!wide) {
#pragma unroll
      for (int k = 0; k < SCAN_I; ++k) v[k] = one(0, i + k);
      return;
    }
    const uint2 st = *reinterpret_cast<const uint2*>(p.status + i);
    double pn[SCAN_I];
#pragma unroll
    for (int k = 0; k < SCAN_I; k += 2) {
      const double2 x = *reinterpret_cast<const double2*>(p.p_n + i + k);
      pn[k] = x.x;
      pn[k + 1] = x.y;
    }
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k)
      v[k] = ((((k < 4 ? st.x : st.y) >> (8 * (k & 3))) & 0xffu) != 0 || pn[k] > 0.0 || p.coat_cc != nullptr) ? 1 : 0;
  }
  XK_D void store(int, long long i, int n, int64_t prefix, const int64_t* v) const {
    int ea[SCAN_I], eb[SCAN_I];
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k)
      if (k < n && v[k]) {
        ea[k] = p.ea[i + k];
        eb[k] = p.eb[i + k];
      }
    int4 nd[SCAN_I];
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k)
      if (k < n && v[k])
        nd[k] = make_int4(m.conn[2 * ea[k]], m.conn[2 * ea[k] + 1], m.conn[2 * eb[k]], m.conn[2 * eb[k] + 1]);
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
      if (k >= n) continue;
      if (!v[k]) {
        const long long o = i + k - prefix;
        if (o < cap_others) others[o] = (int32_t)(i + k);
        continue;
      }
      if (prefix < cap) {
        members[prefix] = (int32_t)(i + k);
        int32_t* q = mnodes + 4 * prefix;
        if (wide) {
          *reinterpret_cast<int4*>(q) = nd[k];
        } else {
          q[0] = nd[k].x; q[1] = nd[k].y; q[2] = nd[k].z; q[3] = nd[k].w;
        }
        atomicAdd(ecnt + ea[k], 1);
        atomicAdd(ecnt + eb[k], 1);
      }
      ++prefix;
    }
  }
  XK_D void total(int, int64_t s) const { tot->members = s; }
};

// elem_ptr (channel 0) and inc_ptr (channel 1): a node's incidences are its elements' members
struct ElemScan {
  int nn, ne;
  const int32_t *ecnt, *neptr;
  const int2* nelem;
  int32_t *eptr, *iptr;
  XK_D long long size(int c) const { return (c == 0 ? ne : nn) + 1; }
  XK_D int64_t one(int c, long long i) const {
    if (c == 0) return i < ne ? ecnt[i] : 0;
    int64_t s = 0;
    if (i < nn)
      for (int y = neptr[i]; y < neptr[i + 1]; ++y) s += ecnt[nelem[y].x >> 1];
    return s;
  }
  XK_D void eight(int c, long long i, int64_t* v) const {
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) v[k] = one(c, i + k);
  }
  XK_D void store(int c, long long i, int n, int64_t prefix, const int64_t* v) const {
    int32_t* out = c == 0 ? eptr : iptr;
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
      if (k < n) out[i + k] = (int32_t)prefix;
      prefix += v[k];
    }
  }
  XK_D void total(int, int64_t) const {}
};

// row_ptr and the rows' first contributions (channel 0, both counts in one word), low_ptr (channel 1)
struct RowScan {
  int nn;
  const int32_t *rcnt, *ccnt, *lcnt;
  int32_t *rptr, *cbase, *lptr;  // lptr nullable
  Totals* tot;
  XK_D long long size(int) const { return nn + 1; }
  XK_D int64_t one(int c, long long i) const {
    if (i >= nn) return 0;
    return c == 0 ? ((int64_t)ccnt[i] << 32) + rcnt[i] : lcnt[i];
  }
  XK_D void eight(int c, long long i, int64_t* v) const {
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) v[k] = one(c, i + k);
  }
  XK_D void store(int c, long long i, int n, int64_t prefix, const int64_t* v) const {
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
      if (k < n) {
        if (c == 0) {
          rptr[i + k] = (int32_t)prefix;
          cbase[i + k] = (int32_t)(prefix >> 32);
        } else if (lptr) {
          lptr[i + k] = (int32_t)prefix;
        }
      }
      prefix += v[k];
    }
  }
  XK_D void total(int c, int64_t s) const {
    if (c == 0) {
      tot->blocks = s & 0xffffffffLL;
      tot->contribs = s >> 32;
    } else {
      tot->low = s;
    }
  }
};

// Bitonic sort of 32 K values, value 32 r + lane in v[r]: partners less than 32 apart by shuffle, the others in
// the lane's own registers.
template <int K>
XK_D void warp_sort_regs(int (&v)[K], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * K; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int r = 0; r < K; ++r) {
          if (r & (j >> 5)) continue;
          const int q = r | (j >> 5), x = min(v[r], v[q]), y = max(v[r], v[q]);
          v[r] = (r & (k >> 5)) ? y : x;
          v[q] = (r & (k >> 5)) ? x : y;
        }
        continue;
      }
#pragma unroll
      for (int r = 0; r < K; ++r) {
        const int o = __shfl_xor_sync(0xffffffffu, v[r], j);
        const bool up = k >= 32 ? (r & (k >> 5)) == 0 : (lane & k) == 0;
        v[r] = up == ((lane & j) == 0) ? min(v[r], o) : max(v[r], o);
      }
    }
}

template <int K>
XK_D void warp_sort_k(const int* l, int n, int32_t* out, int lane) {
  int v[K];
#pragma unroll
  for (int r = 0; r < K; ++r) v[r] = 32 * r + lane < n ? l[32 * r + lane] : 0x7fffffff;
  __syncwarp();  // out may be l
  warp_sort_regs<K>(v, lane);
#pragma unroll
  for (int r = 0; r < K; ++r)
    if (32 * r + lane < n) out[32 * r + lane] = v[r];
}

// The n <= WS_CAP values of l (shared memory) in ascending order to out.
constexpr int WS_CAP = 256;
__device__ __noinline__ void warp_sort(const int* l, int n, int32_t* out, int lane) {
  if (n <= 32) warp_sort_k<1>(l, n, out, lane);
  else if (n <= 64) warp_sort_k<2>(l, n, out, lane);
  else if (n <= 128) warp_sort_k<4>(l, n, out, lane);
  else warp_sort_k<8>(l, n, out, lane);
}

XK_D void serial_insertion_sort(int32_t* a, int n) {
  for (int x = 1; x < n; ++x) {
    const int key = a[x];
    int y = x - 1;
    while (y >= 0 && a[y] > key) { a[y + 1] = a[y]; --y; }
    a[y + 1] = key;
  }
}

// The member sides of the elements, in the order the atomics give (ecnt counts down to zero).
__global__ void k_pat_sides(xk_pairs p, const int32_t* __restrict__ members, const Totals* __restrict__ tot,
                            long long cap, const int32_t* __restrict__ eptr, int32_t* __restrict__ ecnt,
                            int32_t* __restrict__ raw) {
  const long long mi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nm = tot->members;
  if (nm > cap || mi >= nm) return;
  const int i = members[mi];
  const int ea = p.ea[i], eb = p.eb[i];
  raw[eptr[ea] + atomicSub(&ecnt[ea], 1) - 1] = (int)(mi << 1);
  raw[eptr[eb] + atomicSub(&ecnt[eb], 1) - 1] = (int)(mi << 1) | 1;
}

// A warp per node, then a warp per element.  A node's incidences are its elements' member sides; its neighbours (the
// nodes of every member touching it) are its own elements' nodes and each incidence's partner nodes: up to WS_CAP
// such candidates are sorted in the warp's registers and stand next to their repeats.  The sorted neighbours stay in
// list + 4 inc_ptr[v] for k_pat_rows.  A node with more takes the serial path of one lane; one with more than
// MAX_INC incidences holds at most MAX_COLS columns in its row (err otherwise).
// Bound by the instructions issued.  A hash set in shared memory, its ranking by n comparisons per value and the
// same ranking of the incidences took 1500 instructions a warp and 348 us at 99.6k nodes with 30 incidences and 55
// neighbours each; the register sorts take 107 us.
constexpr int RC_WARPS = 4, MAX_INC = 128, MAX_COLS = 256;
struct PatternArgs {
  int nn, ne;
  long long cap, cap_blocks;
  Totals* tot;
  const int32_t *mnodes, *neptr, *eptr, *iptr, *raw;
  const int2* nelem;
  int32_t *inc, *einc;  // einc nullable
  int32_t *list, *rcnt, *ccnt, *lcnt, *err;
  // k_pat_rows
  const int32_t *rptr, *cbase, *lptr;
  int32_t *col, *brow, *bptr, *contrib, *lblk, *bcodes, *serr;  // lblk, bcodes nullable
};

__global__ void __launch_bounds__(32 * RC_WARPS) k_pat_cols(const __grid_constant__ PatternArgs g) {
  __shared__ int s_inc[RC_WARPS][MAX_INC];
  __shared__ int s_cand[RC_WARPS][WS_CAP];
  if (g.tot->members > g.cap) return;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int* l = s_inc[wid];
  int* cand = s_cand[wid];
  const long long w = (long long)blockIdx.x * RC_WARPS + wid;
  if (w >= g.nn) {  // an element
    const long long e = w - g.nn;
    if (e >= g.ne || !g.einc) return;
    const int o = g.eptr[e], n = g.eptr[e + 1] - o;
    if (n <= WS_CAP) {
      for (int i = lane; i < n; i += 32) cand[i] = g.raw[o + i];
      __syncwarp();
      warp_sort(cand, n, g.einc + o, lane);
    } else if (lane == 0) {
      for (int i = 0; i < n; ++i) g.einc[o + i] = g.raw[o + i];
      serial_insertion_sort(g.einc + o, n);
    }
    return;
  }
  const int v = (int)w;
  const int x0 = g.iptr[v], n = g.iptr[v + 1] - x0;
  if (n == 0) {
    if (lane == 0) g.rcnt[v] = g.ccnt[v] = g.lcnt[v] = 0;
    return;
  }
  const int y0 = g.neptr[v], y1 = g.neptr[v + 1];
  int32_t* inc = g.inc + x0;
  int32_t* out = g.list + 4LL * x0;
  if (n > MAX_INC || 2 * n + (y1 - y0) + 1 > WS_CAP) {
    if (lane != 0) return;
    int q = 0;
    for (int y = y0; y < y1; ++y) {
      const int e = g.nelem[y].x >> 1, p = g.nelem[y].x & 1;
      for (int x = g.eptr[e]; x < g.eptr[e + 1]; ++x)
        inc[q++] = ((g.raw[x] >> 1) << 2) | ((g.raw[x] & 1) << 1) | p;
    }
    serial_insertion_sort(inc, n);
    int nd = 0, nc = 0, low = 0;
    for (int x = 0; x < n; ++x)
      for (int k = 0; k < 4; ++k) {
        const int c = g.mnodes[4LL * (inc[x] >> 2) + k];
        nc += c >= v;
        int y = nd - 1;
        while (y >= 0 && out[y] > c) --y;
        if (y >= 0 && out[y] == c) continue;
        for (int z = nd - 1; z > y; --z) out[z + 1] = out[z];
        out[y + 1] = c;
        ++nd;
        low += c < v;
      }
    if (n > MAX_INC && nd - low > MAX_COLS) atomicOr(g.err, 1);
    g.rcnt[v] = nd - low;
    g.ccnt[v] = nc;
    g.lcnt[v] = low;
    return;
  }
  // incidences: the elements' segments one after the other, then sorted
  int q = 0;
  for (int y = y0; y < y1; ++y) {
    const int2 en = g.nelem[y];
    const int o = g.eptr[en.x >> 1], m = g.eptr[(en.x >> 1) + 1] - o;
    for (int i = lane; i < m; i += 32) {
      const int x = g.raw[o + i];
      l[q + i] = ((x >> 1) << 2) | ((x & 1) << 1) | (en.x & 1);
    }
    q += m;
  }
  __syncwarp();
  int nc = 0;  // contributions to the row: the members' nodes >= v
  for (int i = lane; i < n; i += 32) {
    const int x = l[i];
    const int32_t* nd = g.mnodes + 4LL * (x >> 2) + ((x & 2) ? 0 : 2);
    const int a = nd[0], b = nd[1];
    nc += (a >= v) + (b >= v);
    cand[2 * i] = a;
    cand[2 * i + 1] = b;
  }
  for (int y = y0 + lane; y < y1; y += 32) {
    const int2 en = g.nelem[y];
    const int m = g.eptr[(en.x >> 1) + 1] - g.eptr[en.x >> 1];
    nc += m * (1 + (en.y >= v));
    cand[2 * n + y - y0] = m > 0 ? en.y : v;
  }
  q = 2 * n + (y1 - y0);
  if (lane == 0) cand[q] = v;
  ++q;
  nc = __reduce_add_sync(0xffffffffu, nc);
  __syncwarp();
  warp_sort(l, n, inc, lane);
  warp_sort(cand, q, cand, lane);
  __syncwarp();
  int nd = 0, low = 0;
  for (int i0 = 0; i0 < q; i0 += 32) {
    const int i = i0 + lane;
    const int x = i < q ? cand[i] : 0;
    const bool first = i < q && (i == 0 || cand[i - 1] != x);
    const unsigned bal = __ballot_sync(0xffffffffu, first);
    if (first) out[nd + __popc(bal & below)] = x;
    nd += __popc(bal);
    low += __popc(__ballot_sync(0xffffffffu, first && x < v));
  }
  if (lane == 0) {
    g.rcnt[v] = nd - low;
    g.ccnt[v] = nc;
    g.lcnt[v] = low;
  }
}

// First place in a[0, n) not below c, three probes in flight at a time: a step is one latency of the list's memory.
XK_D int lower_bound4(const int32_t* a, int n, int c) {
  int lo = 0;
  while (n > 0) {
    const int h = n >> 1, q = h >> 1, t = h + 1 + ((n - h - 1) >> 1);  // q <= h < t; t == n at the end of a short range
    const int x = a[lo + q], y = a[lo + h], z = a[lo + (t < n ? t : h)];
    if (y < c) {
      if (t < n && z < c) {
        lo += t + 1;
        n -= t + 1;
      } else {
        lo += h + 1;
        n = t - h - 1;
      }
    } else if (x < c) {
      lo += q + 1;
      n = h - q - 1;
    } else {
      n = q;
    }
  }
  return lo;
}

// Inline term lists of the blocks (variant "sides"): a block's same-side terms are element sums.
constexpr int SIDE_FLAG = (int)0x80000000;
// An element's three sums S^00, S^01, S^11, each as 16 values: the 9 of the
// sum, then 1, 1 in the places of a record's s, t and padding, so that a term
// loads the same values from an element sum as from a combined record (both
// 64-byte aligned) and the weight c_1 c_1 = s s of an element-sum term is 1.
constexpr int SUM_STRIDE = 16;
constexpr int ELEM_SUMS = 3 * SUM_STRIDE;

// code into its place among the n terms of a block (ascending; past four it only counts).
XK_D void add_term(int (&terms)[4], int& n, int code) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {  // no array index at run time
    if (k <= n && (k == n || code < terms[k])) {
      const int t = terms[k];
      terms[k] = code;
      code = t;
    }
  }
  ++n;
}

// The same-side terms of block (v, c) from one of v's elements: its S^pp on the diagonal, S^01 to its other node.
XK_D void side_terms(int2 en, int v, int c, int (&terms)[4], int& n) {
  const int base = SIDE_FLAG | (ELEM_SUMS * (en.x >> 1));
  const bool other = c == en.y;
  if (c == v) {
    add_term(terms, n, base + ((en.x & 1) ? 2 * SUM_STRIDE : 0));
    if (other) add_term(terms, n, base + SUM_STRIDE);
  } else if (other) {
    add_term(terms, n, base + SUM_STRIDE);
  }
}

// A warp per node: its row's columns, each block's contributor and term lists, its lower index.  Contributions are
// taken in the incidences' order, 32 at a time, and each goes behind the ones before it in its block (match over
// the warp, a running position per block in shared memory), so the lists come out sorted.
// Bound by latency: a warp's chain of dependent loads.  So the first 32 incidences, neighbours and elements are asked
// for together, then what hangs on them, before anything is searched; the lower index searches with three probes in
// flight.  282 -> 214 us at 99.6k nodes with 28 blocks a row, against the same kernel without that order and with a
// search per contribution.  A mask of the incidences per block in place of the match took more instructions: 242 us.
constexpr int PR_WARPS = 4, PR_CAP = 512;  // contributions of a row (4 per incidence), columns padded to a power of two
__global__ void __launch_bounds__(32 * PR_WARPS, 8) k_pat_rows(const __grid_constant__ PatternArgs g) {
  __shared__ int s_col[PR_WARPS][PR_CAP];
  __shared__ int s_pos[PR_WARPS][PR_CAP];            // next contribution of a block
  __shared__ int s_inc[PR_WARPS][PR_CAP / 4];
  __shared__ signed char s_cross[PR_WARPS][PR_CAP];  // next cross term
  __shared__ __align__(8) short s_rank[PR_WARPS][PR_CAP];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int v = blockIdx.x * PR_WARPS + wid;
  if (g.tot->members > g.cap || g.tot->blocks > g.cap_blocks || v >= g.nn) return;
  const int o = g.rptr[v], nup = g.rptr[v + 1] - o;
  const int x0 = g.iptr[v], n = g.iptr[v + 1] - x0;
  const int low = g.lcnt[v], cb = g.cbase[v], lo = g.lblk ? g.lptr[v] : 0;
  const int y0 = g.neptr[v], ny = g.neptr[v + 1] - y0;
  if (v == g.nn - 1 && lane == 0) g.bptr[o + nup] = g.cbase[g.nn];
  if (n == 0) return;
  const int nc = 4 * n;
  const int32_t* list = g.list + 4LL * x0;
  const int32_t* inc = g.inc + x0;
  const bool fast = nc <= PR_CAP && nup < PR_CAP;
  // the first of each, then the lower neighbours' rows
  int x = lane < n ? inc[lane] : 0;
  int lc = lane < low ? list[lane] : 0;
  const int up = lane < nup ? list[low + lane] : 0x7fffffff;
  int2 en = lane < ny ? g.nelem[y0 + lane] : make_int2(0, -1);
  const int l0 = g.rptr[lc], l1 = g.rptr[lc + 1], li = g.iptr[lc], ll = g.lcnt[lc];
  if (!fast) {  // a block at a time, its contributions collected from all candidates
    int at = cb;
    for (int r = 0; r < nup; ++r) {
      const int c = list[low + r];
      const int b = o + r;
      if (lane == 0) {
        g.col[b] = c;
        g.brow[b] = v;
        g.bptr[b] = at;
      }
      int n_cross = 0;
      for (int i0 = 0; i0 < nc; i0 += 32) {
        const int i = i0 + lane;
        const int y = i < nc ? inc[i >> 2] : 0;
        const bool hit = i < nc && g.mnodes[4LL * (y >> 2) + (i & 3)] == c;
        const bool cross = hit && ((y >> 1) & 1) != ((i & 3) >> 1);
        const unsigned bh = __ballot_sync(0xffffffffu, hit), bc = __ballot_sync(0xffffffffu, cross);
        if (hit) g.contrib[at + __popc(bh & below)] = (y << 2) | (i & 3);
        const int k = n_cross + __popc(bc & below);
        if (cross && k < 4) s_col[wid][k] = (y << 2) | (i & 3);
        at += __popc(bh);
        n_cross += __popc(bc);
      }
      __syncwarp();
      if (g.bcodes && lane == 0) {
        int terms[4] = {-1, -1, -1, -1}, nt = 0;
        for (int y = 0; y < ny; ++y) side_terms(g.nelem[y0 + y], v, c, terms, nt);
        if (nt + n_cross > 4) atomicOr(g.serr, 1);
        else
          for (int k = 0; k < n_cross; ++k) terms[4 - n_cross + k] = s_col[wid][k];
        *reinterpret_cast<int4*>(g.bcodes + 4LL * b) = make_int4(terms[0], terms[1], terms[2], terms[3]);
      }
      __syncwarp();
    }
  } else {
    int* sc = s_col[wid];
    int* sp = s_pos[wid];
    int* sn = s_inc[wid];
    signed char* sx = s_cross[wid];
    short* rk = s_rank[wid];
    int top = 1;
    while (top <= nup) top <<= 1;  // the columns, padded to a power of two above their number
    for (int r = lane; r < top; r += 32) {
      sc[r] = r < 32 ? up : (r < nup ? list[low + r] : 0x7fffffff);
      sp[r] = 0;
    }
    __syncwarp();
    // the block of each contribution and the counts per block, cross ones in the upper half; v is column 0
    for (int j = lane; j < n; j += 32) {
      if (j >= 32) x = inc[j];
      sn[j] = x;
      const int k = x & 3;
      const int32_t* nd = g.mnodes + 4LL * (x >> 2);
      const int c[3] = {nd[k ^ 1], nd[(k & 2) ^ 2], nd[(k & 2) ^ 3]};
      int r[3] = {0, 0, 0};
      for (int st = top >> 1; st > 0; st >>= 1)
#pragma unroll
        for (int q = 0; q < 3; ++q)
          if (sc[r[q] + st - 1] < c[q]) r[q] += st;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        if (c[q] < v) r[q] = -1;
        else atomicAdd(&sp[r[q]], q > 0 ? 0x10001 : 1);
      }
      // in the order of the local nodes
      const int own0 = (k & 1) ? r[0] : 0, own1 = (k & 1) ? 0 : r[0];
      const bool a = (k & 2) == 0;
      *reinterpret_cast<short4*>(rk + 4 * j) =
          make_short4(a ? own0 : r[1], a ? own1 : r[2], a ? r[1] : own0, a ? r[2] : own1);
    }
    if (lane == 0) atomicAdd(&sp[0], n);
    __syncwarp();
    int at = cb;
    for (int r0 = 0; r0 < nup; r0 += 32) {
      const int r = r0 + lane;
      const int c = r < nup ? sp[r] : 0, w = r < nup ? sc[r] : -1;
      int f = c & 0xffff;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, f, d);
        if (lane >= d) f += y;
      }
      const int b = o + r;
      if (g.bcodes) {
        int terms[4] = {-1, -1, -1, -1}, nt = 0;
        for (int y = 0; y < ny; ++y) {
          const int2 ey = y < 32 ? make_int2(__shfl_sync(0xffffffffu, en.x, y & 31), __shfl_sync(0xffffffffu, en.y, y & 31))
                                 : g.nelem[y0 + y];
          side_terms(ey, v, w, terms, nt);
        }
        if (r < nup) {
          const int n_cross = c >> 16;
          if (nt + n_cross > 4) atomicOr(g.serr, 1);
          sx[r] = nt + n_cross > 4 ? 4 : 4 - n_cross;
          *reinterpret_cast<int4*>(g.bcodes + 4LL * b) = make_int4(terms[0], terms[1], terms[2], terms[3]);
        }
      }
      if (r < nup) {
        const int first = at + f - (c & 0xffff);
        g.col[b] = w;
        g.brow[b] = v;
        g.bptr[b] = first;
        sp[r] = first;
      }
      at += __shfl_sync(0xffffffffu, f, 31);
    }
    __syncwarp();
    for (int i0 = 0; i0 < nc; i0 += 32) {
      const int i = i0 + lane;
      const int r = i < nc ? rk[i] : -1;
      const int y = i < nc ? sn[i >> 2] : 0;
      const int code = (y << 2) | (i & 3);
      const bool cross = r >= 0 && ((y >> 1) & 1) != ((i & 3) >> 1);
      const unsigned same = __match_any_sync(0xffffffffu, r);
      const unsigned crosses = __ballot_sync(0xffffffffu, cross) & same;
      int k = 4;
      if (r >= 0) {
        g.contrib[sp[r] + __popc(same & below)] = code;
        if (cross && g.bcodes) k = sx[r] + __popc(crosses & below);
      }
      if (k < 4) g.bcodes[4LL * (o + r) + k] = code;
      __syncwarp();
      if (r >= 0 && (same & below) == 0) {  // the first of its block moves the block on
        sp[r] += __popc(same);
        if (g.bcodes) sx[r] = min(sx[r] + __popc(crosses), 4);  // 4: full (a count would overrun its 8 bits)
      }
      __syncwarp();
    }
  }
  if (!g.lblk) return;
  if (lane < low) g.lblk[lo + lane] = l0 + lower_bound4(g.list + 4LL * li + ll, l1 - l0, v);
  for (int i = lane + 32; i < low; i += 32) {
    lc = list[i];
    const int rc = g.rptr[lc];
    g.lblk[lo + i] = rc + lower_bound4(g.list + 4LL * g.iptr[lc] + g.lcnt[lc], g.rptr[lc + 1] - rc, v);
  }
}

// Mesh node -> (element, local index, other node) lists, and member sides per element.
__global__ void k_node_elem_count(xk_mesh m, int32_t* __restrict__ cnt) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.n_elems) return;
  atomicAdd(&cnt[m.conn[2 * e]], 1);
  atomicAdd(&cnt[m.conn[2 * e + 1]], 1);
}

__global__ void k_node_elem_fill(xk_mesh m, const int32_t* __restrict__ ptr, int32_t* __restrict__ fill,
                                 int2* __restrict__ ne) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m.n_elems) return;
  for (int p = 0; p < 2; ++p) {
    const int v = m.conn[2 * e + p];
    ne[ptr[v] + atomicAdd(&fill[v], 1)] = make_int2((e << 1) | p, m.conn[2 * e + 1 - p]);
  }
}

__global__ void k_segment_sort_pairs(const int32_t* __restrict__ ptr, long long nseg, int2* __restrict__ a) {
  long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nseg) return;
  const int lo = ptr[v], hi = ptr[v + 1];
  for (int x = lo + 1; x < hi; ++x) {
    const int2 key = a[x];
    int y = x - 1;
    while (y >= lo && a[y].x > key.x) { a[y + 1] = a[y]; --y; }
    a[y + 1] = key;
  }
}

// One member record (16 values for combined records) through vector loads.
template <typename T, int N>
XK_D void load_rec(const T* __restrict__ r, T* out);
template <>
XK_D void load_rec<float, 16>(const float* __restrict__ r, float* out) {
  const float4* p = reinterpret_cast<const float4*>(r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = __ldg(p + i);
    out[4 * i] = v.x; out[4 * i + 1] = v.y; out[4 * i + 2] = v.z; out[4 * i + 3] = v.w;
  }
}
template <>
XK_D void load_rec<double, 16>(const double* __restrict__ r, double* out) {
  const double2* p = reinterpret_cast<const double2*>(r);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double2 v = __ldg(p + i);
    out[2 * i] = v.x; out[2 * i + 1] = v.y;
  }
}

// Eight lanes per node: lane l of the group takes incidences l, l+8, ...; the
// group's partial sums are combined by a fixed shuffle tree, so the result does
// not depend on timing.  Sums run in the record precision T (the mixed path
// accumulates in float) and are converted once per degree of freedom.
constexpr int GF_LANES = 8;
template <typename T>
__global__ void k_gather_force(int n_nodes, const int32_t* __restrict__ ptr, const int32_t* __restrict__ inc,
                               const T* __restrict__ rec, int rs, int stc, int vcol, int vcol2,
                               const double* __restrict__ base, double scale, const double* __restrict__ f_ext,
                               const uint8_t* __restrict__ fixed, double* __restrict__ out) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = gid / GF_LANES, lane = gid % GF_LANES;
  const bool live = v < n_nodes;
  T acc[3] = {T(0), T(0), T(0)};
  if (live && ptr)
    for (int x = ptr[v] + lane; x < ptr[v + 1]; x += GF_LANES) {
      const int code = inc[x], k = code & 3;
      const T* r = rec + (long long)(code >> 2) * rs;
      const T c = shape_c<T>(r[stc], r[stc + 1], k);
      for (int d = 0; d < 3; ++d) {
        T w = r[vcol + d];
        if (vcol2 >= 0) w += r[vcol2 + d];
        acc[d] += c * w;
      }
    }
#pragma unroll
  for (int o = GF_LANES / 2; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) acc[d] += __shfl_down_sync(0xffffffffu, acc[d], o, GF_LANES);
#pragma unroll
  for (int d = 0; d < 3; ++d) acc[d] = __shfl_sync(0xffffffffu, acc[d], 0, GF_LANES);
  if (live && lane < 6) {
    const int d = lane;
    const long long dof = 6LL * v + d;
    double r = base ? base[dof] : 0.0;
    if (d < 3) r += scale * (double)(d == 0 ? acc[0] : (d == 1 ? acc[1] : acc[2]));
    if (f_ext) r -= f_ext[dof];
    if (fixed && fixed[dof]) r = 0.0;
    out[dof] = r;
  }
}

// The block sums of a residual kernel's squares go to `part`; the last block to finish (`count`, zero between
// launches, finds it) adds them in block order into *norm2: a fixed order whatever the timing.  b: this
// block's sum, in thread 0; T threads, all of which call it.
template <int T>
XK_D void norm2_of_blocks(double b, double* __restrict__ part, unsigned int* __restrict__ count,
                          double* __restrict__ norm2) {
  __shared__ double red[T / 32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (gridDim.x == 1) {  // nothing to wait for
    if (threadIdx.x == 0) *norm2 = b;
    return;
  }
  if (threadIdx.x == 0) {
    part[blockIdx.x] = b;
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0;
  for (int k = threadIdx.x; k < (int)gridDim.x; k += T) a += __ldcg(part + k);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
  if (lane == 0) red[warp] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < T / 32; ++w) t += red[w];
    *norm2 = t;
    *count = 0u;  // ready for the next launch
  }
}
// the counter of both residual kernels, the last word of norm_scratch: beyond the block sums of either
unsigned int* norm_count(double* part, int n_nodes) {
  return part ? reinterpret_cast<unsigned int*>(part + (6LL * n_nodes + 255) / 256) : nullptr;
}

XK_D double to_f64(float x) { return xk_f2d(x); }  // the conversion in integer arithmetic (the FP64 pipe is slow)
XK_D double to_f64(double x) { return x; }

// s, t and v of a combined record
XK_D void load_stv(const float* __restrict__ r, float* o) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(r) + 2), b = __ldg(reinterpret_cast<const float4*>(r) + 3);
  o[0] = a.y; o[1] = a.z; o[2] = a.w; o[3] = b.x; o[4] = b.y;
}
XK_D void load_stv(const double* __restrict__ r, double* o) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(r) + 4), b = __ldg(reinterpret_cast<const double2*>(r) + 5),
                c = __ldg(reinterpret_cast<const double2*>(r) + 6);
  o[0] = a.y; o[1] = b.x; o[2] = b.y; o[3] = c.x; o[4] = c.y;
}

// The assembly's form of k_gather_force: combined records, the squared norm fused.  The same sums in the same
// order; what it saves is latency: a record's five values come by two (three in double) vector loads, two
// incidences' loads are in flight together, and the norm takes no further launches.
// GFN_NODES a CTA, so that the block sums fit norm_scratch.
// Measured with both norm launches: 37-wire strand in double (4,773 nodes) 18 -> 11 us, its eager assembly 75 -> 67 us;
// 64 small strands in float 26 -> 22 us, 93 -> 89 us.
constexpr int GFN_NODES = 48, GFN_T = GFN_NODES * GF_LANES;
static_assert(6 * GFN_NODES % 32 == 0, "whole warps of squares");
template <typename T>
__global__ void __launch_bounds__(GFN_T) k_gather_force_norm(int n_nodes, const int32_t* __restrict__ ptr,
                                                             const int32_t* __restrict__ inc,
                                                             const T* __restrict__ rec,
                                                             const double* __restrict__ base, double scale,
                                                             const double* __restrict__ f_ext,
                                                             const uint8_t* __restrict__ fixed,
                                                             double* __restrict__ out, double* __restrict__ part,
                                                             unsigned int* __restrict__ count,
                                                             double* __restrict__ norm2) {
  static_assert(XK_REC_S == 9 && XK_REC_V == 11, "combined record layout");
  __shared__ T s_acc[3 * GFN_NODES];
  __shared__ double s_sq[6 * GFN_NODES];
  const int local = threadIdx.x / GF_LANES, lane = threadIdx.x % GF_LANES, v0 = blockIdx.x * GFN_NODES;
  const bool live = v0 + local < n_nodes;
  // the DOFs of the CTA's nodes, one a thread, on their way while the records are gathered
  const long long dof = 6LL * v0 + threadIdx.x;
  const bool mine = threadIdx.x < 6 * GFN_NODES && dof < 6LL * n_nodes;
  double r = 0.0, f = 0.0;
  bool fix = false;
  if (mine) {
    if (base) r = base[dof];
    if (f_ext) f = f_ext[dof];
    if (fixed) fix = fixed[dof] != 0;
  }
  T acc[3] = {T(0), T(0), T(0)};
  if (live && ptr) {
    const int x0 = ptr[v0 + local], x1 = ptr[v0 + local + 1];
    for (int x = x0 + lane; x < x1; x += 2 * GF_LANES) {
      const bool two = x + GF_LANES < x1;
      const int c0 = inc[x], c1 = two ? inc[x + GF_LANES] : c0;
      T q[2][5];
      load_stv(rec + (long long)(c0 >> 2) * XK_REC_STRIDE_COMBINED, q[0]);
      if (two) load_stv(rec + (long long)(c1 >> 2) * XK_REC_STRIDE_COMBINED, q[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (j == 1 && !two) break;
        const T c = shape_c<T>(q[j][0], q[j][1], (j == 0 ? c0 : c1) & 3);
#pragma unroll
        for (int d = 0; d < 3; ++d) acc[d] += c * q[j][2 + d];
      }
    }
  }
#pragma unroll
  for (int o = GF_LANES / 2; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) acc[d] += __shfl_down_sync(0xffffffffu, acc[d], o, GF_LANES);
  if (lane == 0)
#pragma unroll
    for (int d = 0; d < 3; ++d) s_acc[3 * local + d] = acc[d];
  __syncthreads();
  if (threadIdx.x < 6 * GFN_NODES) {
    if (mine) {
      const int d = threadIdx.x % 6;
      if (d < 3) r += scale * to_f64(s_acc[3 * (threadIdx.x / 6) + d]);
      if (f_ext) r -= f;
      if (fix) r = 0.0;
      out[dof] = r;
    }
    s_sq[threadIdx.x] = r * r;
  }
  if (!norm2) return;  // uniform over the launch
  __syncthreads();
  double b = 0.0;
  if (threadIdx.x < 32) {  // the FP64 pipe takes a warp's addition for as long as a thread's: one warp adds
#pragma unroll
    for (int k = 0; k < 6 * GFN_NODES / 32; ++k) b += s_sq[threadIdx.x + 32 * k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) b += __shfl_down_sync(0xffffffffu, b, o);
  }
  norm2_of_blocks<GFN_T>(b, part, count, norm2);
}

// Column of s (then t) in a record of RS values: combined records put B first.
template <int RS>
__host__ __device__ constexpr int rec_st() { return RS == XK_REC_STRIDE_COMBINED ? XK_REC_S : 0; }

template <typename T, int RS, int BCOL>
XK_D void add_contrib(const T* __restrict__ rec, int code, T* acc) {
  constexpr int ST = rec_st<RS>();
  const int k = (code >> 2) & 3, l = code & 3;
  T r[RS];
  if (RS == 16) {
    load_rec<T, 16>(rec + (long long)(code >> 4) * RS, r);
  } else {
#pragma unroll
    for (int q = 0; q < RS; ++q) r[q] = rec[(long long)(code >> 4) * RS + q];
  }
  const T w = shape_c<T>(r[ST], r[ST + 1], k) * shape_c<T>(r[ST], r[ST + 1], l);
#pragma unroll
  for (int q = 0; q < 9; ++q) acc[q] += w * r[BCOL + q];
}

// Variant "sides", step 1: S_e^00, S_e^01, S_e^11 (9 values each) of every
// element from its members, one thread per (element, B component); the weights
// are the products c_p c_q of the member's side: (1-s)^2, (1-s)s, s^2 on side A
// and the same in t on side B (the signs of c_2, c_3 cancel).
//
// With combined records the same pass also forms the element's force sums
// F_e^0 = sum c_p v and F_e^1 = sum c_q v over its members (p, q the element's
// first and second local node on the member's side: c = 1-s, s on side A and
// -(1-t), -t on side B), 8 values per element after the 36 * ne tangent sums;
// a node's contact force is then the sum of F over its incident elements
// (k_gather_force_elem).
constexpr int ELEM_FORCE = 8;

template <typename T, int RS, int BCOL>
__global__ void k_elem_sums(int ne, const int32_t* __restrict__ eptr, const int32_t* __restrict__ einc,
                            const T* __restrict__ rec, T* __restrict__ S) {
  constexpr int ST = rec_st<RS>();
  constexpr bool FORCE = RS == XK_REC_STRIDE_COMBINED;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 9LL * ne) return;
  const int e = (int)(t / 9), q = (int)(t % 9);
  T s00 = T(0), s01 = T(0), s11 = T(0), f0 = T(0), f1 = T(0);
  const int x1 = eptr[e + 1];
#pragma unroll 4
  for (int x = eptr[e]; x < x1; ++x) {
    const int code = einc[x];
    const T* r = rec + (long long)(code >> 1) * RS;
    const T a = r[ST + (code & 1)];
    const T b = r[BCOL + q];
    const T om = T(1) - a;
    s00 += (om * om) * b;
    s01 += (om * a) * b;
    s11 += (a * a) * b;
    if (FORCE && q < 3) {
      const T v = (code & 1) ? -r[XK_REC_V + q] : r[XK_REC_V + q];
      f0 += om * v;
      f1 += a * v;
    }
  }
  T* o = S + (long long)ELEM_SUMS * e;
  o[q] = s00;
  o[SUM_STRIDE + q] = s01;
  o[2 * SUM_STRIDE + q] = s11;
  if (q < 3) {  // padding of sum q: (s, t) = (1, 1)
    o[q * SUM_STRIDE + 9] = T(1);
    o[q * SUM_STRIDE + 10] = T(1);
    if (FORCE) {
      T* f = S + (long long)ELEM_SUMS * ne + (long long)ELEM_FORCE * e;
      f[q] = f0;
      f[3 + q] = f1;
      if (q < 2) f[6 + q] = T(0);
    }
  }
}

// The same sums for combined records, four lanes per element: lane q sums the incidences
// q, q + 4, q + 8, ... of the element (each one record read as two 256-bit loads for float),
// and the four partial sums are combined by a fixed shuffle tree ((q + q^2) + (q^1 + q^3)), so the
// result does not depend on timing.  It differs from k_elem_sums' single running sum by
// rounding only.
template <typename T>
XK_D void load16(const T* __restrict__ p, T* v);
template <>
XK_D void load16<float>(const float* __restrict__ p, float* v) {  // p 32-byte aligned
  ldg8(p, v);
  ldg8(p + 8, v + 8);
}
template <>
XK_D void load16<double>(const double* __restrict__ p, double* v) {
  const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double2 x = __ldg(q + i);
    v[2 * i] = x.x; v[2 * i + 1] = x.y;
  }
}

template <typename T>
XK_D void store4(T* p, T a, T b, T c, T d);
template <>
XK_D void store4<float>(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
template <>
XK_D void store4<double>(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 7 : 4) k_elem_sums_rec(int ne, const int32_t* __restrict__ eptr,
                                                       const int32_t* __restrict__ einc, const T* __restrict__ rec,
                                                       T* __restrict__ S) {
  static_assert(XK_REC_B == 0 && XK_REC_S == 9 && XK_REC_V == 11, "combined record layout");
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int e = (int)(gid >> 2), q = (int)(gid & 3);
  const bool live = e < ne;  // a quad is all live or all dead (4 | 128)
  T s00[9], s01[9], s11[9], f0[3], f1[3];
#pragma unroll
  for (int c = 0; c < 9; ++c) { s00[c] = T(0); s01[c] = T(0); s11[c] = T(0); }
#pragma unroll
  for (int c = 0; c < 3; ++c) { f0[c] = T(0); f1[c] = T(0); }
  const int x0 = live ? eptr[e] : 0, x1 = live ? eptr[e + 1] : 0;
  // two incidences per round (x and x + 4), both records loaded before either is summed; the
  // sums still take the lane's incidences in order
  for (int x = x0 + q; x < x1; x += 8) {
    const bool two = x + 4 < x1;
    const int code0 = einc[x];
    const int code1 = two ? einc[x + 4] : code0;
    T r[2][16];
    load16<T>(rec + (long long)(code0 >> 1) * XK_REC_STRIDE_COMBINED, r[0]);
    if (two) load16<T>(rec + (long long)(code1 >> 1) * XK_REC_STRIDE_COMBINED, r[1]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (j == 1 && !two) break;
      const int code = j == 0 ? code0 : code1;
      const T a = (code & 1) ? r[j][XK_REC_S + 1] : r[j][XK_REC_S];
      const T om = T(1) - a;
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        s00[c] += (om * om) * r[j][c];
        s01[c] += (om * a) * r[j][c];
        s11[c] += (a * a) * r[j][c];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const T v = (code & 1) ? -r[j][XK_REC_V + c] : r[j][XK_REC_V + c];
        f0[c] += om * v;
        f1[c] += a * v;
      }
    }
  }
  // Reduce-scatter over the quad: the 33 sums (S^00, S^01, S^11, F^0, F^1, padded to 36) split in
  // halves between lanes q and q ^ 2, then in quarters between q and q ^ 1, so that lane q ends with
  // the nine values it stores (lane 0 S^00, 1 S^01, 2 S^11, 3 F^0 F^1) as (l_q + l_q^2) +
  // (l_q^1 + l_q^3): a fixed tree of 27 shuffles per lane.
  T v[36];
#pragma unroll
  for (int c = 0; c < 9; ++c) { v[c] = s00[c]; v[9 + c] = s01[c]; v[18 + c] = s11[c]; }
#pragma unroll
  for (int c = 0; c < 3; ++c) { v[27 + c] = f0[c]; v[30 + c] = f1[c]; v[33 + c] = T(0); }
  const bool hi = (q >> 1) & 1, odd = q & 1;
#pragma unroll
  for (int c = 0; c < 18; ++c) {  // lane q keeps half hi, receives it from q ^ 2
    const T y = __shfl_xor_sync(0xffffffffu, hi ? v[c] : v[18 + c], 2);
    if (hi) v[18 + c] += y; else v[c] += y;
  }
  T w[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) {  // within the kept half, quarter odd, received from q ^ 1
    const T a = hi ? v[18 + c] : v[c], b = hi ? v[27 + c] : v[9 + c];
    const T y = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
    w[c] = (odd ? b : a) + y;
  }
  if (!live) return;
  // vector stores: lanes 0-2 write sum S^00, S^01, S^11 (its 9 values, then (s, t) = (1, 1) and a
  // zero; the last 4 values of a sum are not read), lane 3 the force sums
  if (q < 3) {
    T* o = S + (long long)ELEM_SUMS * e + q * SUM_STRIDE;
    store4<T>(o, w[0], w[1], w[2], w[3]);
    store4<T>(o + 4, w[4], w[5], w[6], w[7]);
    store4<T>(o + 8, w[8], T(1), T(1), T(0));
  } else {
    T* f = S + (long long)ELEM_SUMS * ne + (long long)ELEM_FORCE * e;
    store4<T>(f, w[0], w[1], w[2], w[3]);
    store4<T>(f + 4, w[4], w[5], T(0), T(0));
  }
}

// R[dof] = base[dof] + scale * (contact force at the node) - f_ext[dof], zero where fixed, from
// the element force sums of the last element-side tangent gather: one thread per node, its
// incident elements in their list order.  The block partial sums of R^2 (each thread's six
// squares in order, then a fixed shuffle tree over the warp and over the block's warps) go to
// `part`, and the last block to finish adds them in block order into *norm2 (a fixed order
// whatever the timing); `count` (zero between launches) finds the last block.  VEC: base,
// f_ext and out are 16-byte aligned and moved as double2.
constexpr int GFE_T = 256;

template <typename T, bool VEC>
__global__ void __launch_bounds__(GFE_T) k_gather_force_elem(int n_nodes, int ne, const int32_t* __restrict__ neptr,
                                                             const int2* __restrict__ nelem, const T* __restrict__ S,
                                                             const double* __restrict__ base, double scale,
                                                             const double* __restrict__ f_ext,
                                                             const uint8_t* __restrict__ fixed,
                                                             double* __restrict__ out, double* __restrict__ part,
                                                             unsigned int* __restrict__ count,
                                                             double* __restrict__ norm2) {
  const int v = blockIdx.x * GFE_T + threadIdx.x;
  double sq = 0.0;
  if (v < n_nodes) {
    double r[6];
    if (base) {
      if (VEC) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double2 x = __ldg(reinterpret_cast<const double2*>(base + 6LL * v) + i);
          r[2 * i] = x.x;
          r[2 * i + 1] = x.y;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 6; ++c) r[c] = base[6LL * v + c];
      }
    } else {
#pragma unroll
      for (int c = 0; c < 6; ++c) r[c] = 0.0;
    }
    const T* F = S + (long long)ELEM_SUMS * ne;
    T acc[3] = {T(0), T(0), T(0)};
    for (int y = neptr[v]; y < neptr[v + 1]; ++y) {
      const int ex = nelem[y].x;  // (element << 1) | local index of v in it
      const T* f = F + (long long)ELEM_FORCE * (ex >> 1) + 3 * (ex & 1);
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] += f[c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) r[c] += scale * to_f64(acc[c]);
    if (f_ext) {
      if (VEC) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double2 x = __ldg(reinterpret_cast<const double2*>(f_ext + 6LL * v) + i);
          r[2 * i] -= x.x;
          r[2 * i + 1] -= x.y;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 6; ++c) r[c] -= f_ext[6LL * v + c];
      }
    }
    if (fixed) {
#pragma unroll
      for (int c = 0; c < 6; ++c)
        if (fixed[6LL * v + c]) r[c] = 0.0;
    }
    if (VEC) {
#pragma unroll
      for (int i = 0; i < 3; ++i) reinterpret_cast<double2*>(out + 6LL * v)[i] = make_double2(r[2 * i], r[2 * i + 1]);
    } else {
#pragma unroll
      for (int c = 0; c < 6; ++c) out[6LL * v + c] = r[c];
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) sq = fma(r[c], r[c], sq);
  }
  if (!norm2) return;  // uniform over the launch
  __shared__ double red[GFE_T / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  double b = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < GFE_T / 32; ++w) b += red[w];
  norm2_of_blocks<GFE_T>(b, part, count, norm2);
}

template <typename T>
XK_D void load12(const T* __restrict__ p, T* v);
template <>
XK_D void load12<float>(const float* __restrict__ p, float* v) {  // p 32-byte aligned
  ldg8(p, v);
  const float4 x = __ldg(reinterpret_cast<const float4*>(p) + 2);
  v[8] = x.x; v[9] = x.y; v[10] = x.z; v[11] = x.w;
}
template <>
XK_D void load12<double>(const double* __restrict__ p, double* v) {
  const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const double2 x = __ldg(q + i);
    v[2 * i] = x.x; v[2 * i + 1] = x.y;
  }
}

// acc += one term of a block (-1: none): B and (s, t) of an element sum (s = t = 1) or of a member record
template <typename T>
XK_D void sides_term(const T* __restrict__ S, const T* __restrict__ rec, int c, T* acc) {
  if (c == -1) return;
  T v[12];
  load12<T>(c < 0 ? S + (c & 0x7fffffff) : rec + (long long)(c >> 4) * XK_REC_STRIDE_COMBINED, v);
  const int k = c < 0 ? 1 : (c >> 2) & 3, l = c < 0 ? 1 : c & 3;
  const T w = shape_c<T>(v[9], v[10], k) * shape_c<T>(v[9], v[10], l);
#pragma unroll
  for (int q = 0; q < 9; ++q) acc[q] += w * v[q];
}

// Variant "sides", step 2: one thread per block over its (at most four) inline
// terms in their sorted order: element sums, then cross contributions; the
// block values go out through shared memory so that the stores are coalesced.
constexpr int GS_T = 128;

template <typename T, int RS, int BCOL>
XK_D void add_term(const T* __restrict__ S, const T* __restrict__ rec, int code, T* acc) {
  if (code == -1) return;
  if (code < 0) {
    const T* s = S + (code & 0x7fffffff);
#pragma unroll
    for (int q = 0; q < 9; ++q) acc[q] += s[q];
  } else {
    add_contrib<T, RS, BCOL>(rec, code, acc);
  }
}

// The grid is persistent (as many CTAs per SM as are resident, each taking every gridDim.x-th tile of
// GS_T blocks): a thread loads its code of the CTA's next tile before it gathers the terms of the
// current one, so the code load's latency hides behind the term loads.
XK_D int4 sides_code(const int4* __restrict__ codes, long long nnzb, long long tile) {
  const long long b = tile * GS_T + threadIdx.x;
  return b < nnzb ? __ldcs(codes + b) : make_int4(-1, -1, -1, -1);
}

// The blocks of a tile in descending order of their numbers of terms (stable): thread t gets the codes of the
// t-th in c; returns which block of the tile that is.  Most blocks have one term and some have up to four, so a
// warp of consecutive blocks issues its slowest lane's three to four terms; the FP64 pipe, which bounds the
// double gather, takes a full issue for every one.  Sorted, one warp of four has the long blocks.  Every block's
// sum is its own thread's, in the order of its codes.
// Measured at the 1027-wire strand (2.79M blocks, 3.3M terms): 251 us -> 175 us.  In float, where the loads bound it,
// the blocks stay in order.
struct TermOrder {
  int4 code[GS_T];
  int idx[GS_T];
  int cnt[GS_T / 32][4];  // blocks of a warp with 4, 3, 2, 1 terms
};
XK_D int order_by_terms(int4& c, TermOrder& s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = (c.x != -1) + (c.y != -1) + (c.z != -1) + (c.w != -1);
  const unsigned below = (1u << lane) - 1u;
  int before = 0;  // blocks of this warp with more terms, or as many and a lower lane
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned m = __ballot_sync(0xffffffffu, n == 4 - k);
    if (lane == k) s.cnt[warp][k] = __popc(m);
    if (n == 4 - k) before = __popc(m & below);
  }
  const unsigned none = __ballot_sync(0xffffffffu, n == 0);
  __syncthreads();
  int rank = before;
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int w = 0; w < GS_T / 32; ++w)
      if (n < 4 - k || (n == 4 - k && w < warp)) rank += s.cnt[w][k];
  if (n == 0) {  // after all others: the warps' empty blocks in turn
    rank += __popc(none & below);
    for (int w = 0; w < warp; ++w) rank += 32 - (s.cnt[w][0] + s.cnt[w][1] + s.cnt[w][2] + s.cnt[w][3]);
  }
  s.code[rank] = c;
  s.idx[rank] = threadIdx.x;
  __syncthreads();
  c = s.code[threadIdx.x];
  return s.idx[threadIdx.x];
}

template <typename T, int RS, int BCOL>
__global__ void __launch_bounds__(GS_T, sizeof(T) == 4 ? 16 : 8) k_gather_tangent_sides(long long nnzb, const int4* __restrict__ codes,
                                                               const T* __restrict__ S, const T* __restrict__ rec,
                                                               T* __restrict__ K) {
  __shared__ __align__(16) T stage[GS_T * 9];
  __shared__ TermOrder order;
  const long long ntiles = (nnzb + GS_T - 1) / GS_T;
  long long tile = blockIdx.x;
  int4 cn = tile < ntiles ? sides_code(codes, nnzb, tile) : make_int4(-1, -1, -1, -1);
  for (; tile < ntiles; tile += gridDim.x) {
    const long long b0 = tile * GS_T;
    int4 c = cn;
    int at = threadIdx.x;  // this thread's block of the tile
    if (tile + gridDim.x < ntiles) cn = sides_code(codes, nnzb, tile + gridDim.x);
    if (sizeof(T) == 8) at = order_by_terms(c, order);
    T acc[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) acc[q] = T(0);
    if (RS == XK_REC_STRIDE_COMBINED) {
      // each term is the first twelve values of its element sum or member record
      sides_term<T>(S, rec, c.x, acc);
      sides_term<T>(S, rec, c.y, acc);
      sides_term<T>(S, rec, c.z, acc);
      sides_term<T>(S, rec, c.w, acc);
    } else {
      add_term<T, RS, BCOL>(S, rec, c.x, acc);
      add_term<T, RS, BCOL>(S, rec, c.y, acc);
      add_term<T, RS, BCOL>(S, rec, c.z, acc);
      add_term<T, RS, BCOL>(S, rec, c.w, acc);
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) stage[at * 9 + q] = acc[q];
    __syncthreads();
    const long long rem = nnzb - b0;
    const int nv = 9 * (int)(rem < GS_T ? rem : GS_T);
    T* out = K + 9 * b0;
    if (sizeof(T) == 4 && ((uintptr_t)out & 15) == 0) {
      // 16-byte stores of the staged values (a CTA's 128 blocks are 4608 bytes)
      const int n4 = nv / 4;
      for (int v = threadIdx.x; v < n4; v += GS_T)
        reinterpret_cast<float4*>(out)[v] = reinterpret_cast<const float4*>(stage)[v];
      for (int v = 4 * n4 + threadIdx.x; v < nv; v += GS_T) out[v] = stage[v];
    } else {
      for (int v = threadIdx.x; v < nv; v += GS_T) out[v] = stage[v];
    }
    __syncthreads();  // the stage is read out before the next tile overwrites it
  }
}

// persistent grid of the sides gather: every SM's share of CTAs, or one CTA per tile when fewer
int sides_grid(long long nnzb, int per_sm) {
  const int sms = xk_sm_count();
  const long long tiles = (nnzb + GS_T - 1) / GS_T;
  const long long cap = (long long)sms * per_sm;
  return (int)(tiles < cap ? (tiles > 0 ? tiles : 1) : cap);
}


// Variant "lanes": a warp owns 32 consecutive blocks and spreads their
// contributors one per lane (32 per round); a segmented inclusive scan over
// the lanes (fixed shuffle tree, segments = blocks) sums each block's run in
// the round and the run's last lane adds it to the block's shared-memory
// accumulator.  Fewer serial steps per lane than the chunked variant below,
// more shuffles per contributor.
template <typename T, int RS, int BCOL>
__global__ void __launch_bounds__(128) k_gather_tangent_lanes(long long nnzb, const int32_t* __restrict__ bptr,
                                                             const int32_t* __restrict__ contrib,
                                                             const T* __restrict__ rec, T* __restrict__ K) {
  __shared__ T acc[4][32 * 9];
  __shared__ int ptr_s[4][33];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long b0 = ((long long)blockIdx.x * 4 + wl) * 32;
  if (b0 >= nnzb) return;  // whole warp
  const int nblk = (int)((nnzb - b0) < 32 ? (nnzb - b0) : 32);
  T* A = acc[wl];
  int* P = ptr_s[wl];
#pragma unroll
  for (int q = 0; q < 9; ++q) A[q * 32 + lane] = T(0);
  P[lane] = bptr[b0 + (lane < nblk ? lane : nblk)];
  if (lane == 0) P[32] = bptr[b0 + nblk];
  __syncwarp();
  const int x0 = P[0], x1 = P[nblk];
  for (int base = x0; base < x1; base += 32) {
    const int x = base + lane;
    const bool valid = x < x1;
    int slot = 0;
    if (valid) {
      int lo = 0, hi = nblk - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P[mid] <= x) lo = mid; else hi = mid - 1;
      }
      slot = lo;
    }
    T v[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) v[q] = T(0);
    if (valid) add_contrib<T, RS, BCOL>(rec, contrib[x], v);
    const int prev_slot = __shfl_up_sync(0xffffffffu, slot, 1);
    const bool head = valid && (lane == 0 || prev_slot != slot);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int seg_start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const T y = __shfl_up_sync(0xffffffffu, v[q], d);
        if (lane - d >= seg_start) v[q] += y;
      }
    }
    const int next_slot = __shfl_down_sync(0xffffffffu, slot, 1);
    const bool next_valid = __shfl_down_sync(0xffffffffu, (int)valid, 1) != 0;
    const bool tail = valid && (lane == 31 || !next_valid || next_slot != slot);
    if (tail) {
#pragma unroll
      for (int q = 0; q < 9; ++q) A[slot * 9 + q] += v[q];
    }
    __syncwarp();
  }
  for (int i = lane; i < 9 * nblk; i += 32) K[9 * b0 + i] = A[i];
}

// Variant "chunks" (default for double): Contributor counts are very uneven: 61% of the blocks of a strand have one
// contributor, a node's diagonal block up to ~36.  A warp owns 32 consecutive
// blocks and cuts their contributor list into chunks of GT_CH, one per lane
// (a round covers 32 * GT_CH contributors).  A lane sums its chunk serially;
// a block whose contributors end inside the chunk is added to the block's
// shared-memory accumulator by that lane, with the partial sums of the lanes
// before it (a segmented inclusive scan of the lanes' last partial sums over
// a fixed shuffle tree).  After the last round the warp stores its 32 x 9
// values contiguously.  Every sum is taken in a fixed order.
constexpr int GT_WARPS = 4;
constexpr int GT_CH = 4;

template <typename T, int RS, int BCOL>
__global__ void __launch_bounds__(32 * GT_WARPS) k_gather_tangent(long long nnzb, const int32_t* __restrict__ bptr,
                                                                 const int32_t* __restrict__ contrib,
                                                                 const T* __restrict__ rec, T* __restrict__ K) {
  __shared__ T acc[GT_WARPS][32 * 9];
  __shared__ int ptr_s[GT_WARPS][33];
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long b0 = ((long long)blockIdx.x * GT_WARPS + wl) * 32;
  if (b0 >= nnzb) return;  // whole warp
  const int nblk = (int)((nnzb - b0) < 32 ? (nnzb - b0) : 32);
  T* A = acc[wl];
  int* P = ptr_s[wl];
#pragma unroll
  for (int q = 0; q < 9; ++q) A[q * 32 + lane] = T(0);
  P[lane] = bptr[b0 + (lane < nblk ? lane : nblk)];
  if (lane == 0) P[32] = bptr[b0 + nblk];
  __syncwarp();
  const int x0 = P[0], x1 = P[nblk];
  for (int base = x0; base < x1; base += 32 * GT_CH) {
    const int c0 = base + lane * GT_CH;
    const int c1 = min(c0 + GT_CH, x1);
    const bool has = c0 < c1;
    // slot of the chunk's first contributor: last slot whose start <= c0
    int slot = 0;
    if (has) {
      int lo = 0, hi = nblk - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P[mid] <= c0) lo = mid; else hi = mid - 1;
      }
      slot = lo;
    }
    const int first_slot = slot;
    const bool first_open = has && P[slot] < c0;  // first block began before this chunk
    T part[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) part[q] = T(0);
    T head[9];  // sum over the first block's contributors in this chunk, once it is closed
    bool head_closed = false;
    for (int x = c0; x < c1; ++x) {
      while (x >= P[slot + 1]) {  // the current block ends before x: close it
        if (slot == first_slot && first_open) {
#pragma unroll
          for (int q = 0; q < 9; ++q) head[q] = part[q];
          head_closed = true;
        } else {
#pragma unroll
          for (int q = 0; q < 9; ++q) A[slot * 9 + q] += part[q];
        }
#pragma unroll
        for (int q = 0; q < 9; ++q) part[q] = T(0);
        ++slot;
      }
      add_contrib<T, RS, BCOL>(rec, contrib[x], part);
    }
    const int last_slot = slot;
    // lanes whose last block is open at the end of the chunk pass its partial on
    // (lane 31 closes at the end of the round; the next round adds the rest)
    const bool tail_open = has && lane < 31 && c1 < P[last_slot + 1] && c1 < x1;
    // segmented inclusive scan over lanes of the last partials; a lane starts a
    // segment unless its first block continues the previous lane's last block
    const int prev_last = __shfl_up_sync(0xffffffffu, last_slot, 1);
    const bool prev_open = __shfl_up_sync(0xffffffffu, (int)tail_open, 1) != 0;
    const bool cont = lane > 0 && has && prev_open && prev_last == first_slot;
    // value entering the scan: the lane's last partial when its last block is the
    // continued first block, else its last partial alone (a new segment)
    T v[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) v[q] = part[q];
    const bool seg_head = !(cont && last_slot == first_slot && !head_closed);
    const unsigned heads = __ballot_sync(0xffffffffu, seg_head);
    const int seg_start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const T y = __shfl_up_sync(0xffffffffu, v[q], d);
        if (lane - d >= seg_start) v[q] += y;
      }
    }
    // carry into this lane's first block = the previous lane's scanned value
    T carry[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const T y = __shfl_up_sync(0xffffffffu, v[q], 1);
      carry[q] = cont ? y : T(0);
    }
    if (has) {
      if (head_closed) {  // the first block ended inside this chunk
#pragma unroll
        for (int q = 0; q < 9; ++q) A[first_slot * 9 + q] += carry[q] + head[q];
      }
      if (!tail_open) {  // the last block ends here (or the round ends)
        if (last_slot == first_slot && !head_closed) {
#pragma unroll
          for (int q = 0; q < 9; ++q) A[last_slot * 9 + q] += v[q];  // scanned: carry + own
        } else {
#pragma unroll
          for (int q = 0; q < 9; ++q) A[last_slot * 9 + q] += part[q];
        }
      }
    }
    __syncwarp();
  }
  for (int i = lane; i < 9 * nblk; i += 32) K[9 * b0 + i] = A[i];
}

}  // namespace

extern "C" xk_status xk_contact_pattern_build(const xk_mesh* m, const xk_pairs* p, xk_contact_pattern* pat,
                                              xk_stream s) {
  if (!m || !p || !pat) return xk_set_error(XK_ERR_ARG, "xk_contact_pattern_build: null argument");
  if (!pat->inc_ptr || !pat->row_ptr) return xk_set_error(XK_ERR_ARG, "xk_contact_pattern_build: row arrays missing");
  cudaStream_t st = (cudaStream_t)s;
  const int nn = m->n_nodes, ne = m->n_elems;
  const long long np = p->n;
  pat->n_nodes = nn;
  pat->n_elems = ne;
  pat->sides_ok = 0;
  const bool sides = pat->node_elem_ptr && pat->node_elem && pat->elem_ptr && pat->elem_inc && pat->bcodes;
  const bool lower = pat->low_ptr && pat->low_blk;
  const long long nmx = np < pat->cap_members ? np : pat->cap_members;  // members this build can hold
  const long long longest = (ne > nn ? ne : nn) + 1;
  // one piece that starts at zero: the counts and the scans' words
  const long long w_mem = scan_words(np, 1), w_el = scan_words(longest, 2), w_row = scan_words(nn + 1, 2);
  const long long n_sums = scan_sums(np, 1) + scan_sums(longest, 2) + scan_sums(nn + 1, 2);
  const size_t zero = sizeof(Totals) + sizeof(int32_t) * (size_t)(2 + w_mem + w_el + w_row + ne + 1);
  XkScratch S(st);
  XK_TRY(S.reserve(zero + 4 * ((size_t)(sides ? 0 : 2 * (nn + 1) + 4 * (size_t)ne + ne + 1) + 18 * (size_t)nmx +
                               4 * ((size_t)nn + 1) + 2 * (size_t)n_sums) + (1 << 14)));
  char* z;
  int64_t* sums;
  PatternArgs g = {};
  XK_TRY(S.get(&z, (long long)zero));
  XK_TRY(S.get(&sums, n_sums));
  int32_t *raw, *cbase;
  XK_TRY(S.get(&raw, 2 * nmx));
  XK_TRY(S.get(&g.list, 16 * nmx));
  XK_TRY(S.get(&g.rcnt, nn));
  XK_TRY(S.get(&g.ccnt, nn));
  XK_TRY(S.get(&g.lcnt, nn));
  XK_TRY(S.get(&cbase, nn + 1));
  int32_t *neptr = pat->node_elem_ptr, *nelem = pat->node_elem, *eptr = pat->elem_ptr;
  if (!sides) {  // the mesh topology of this call only
    XK_TRY(S.get(&neptr, nn + 1));
    XK_TRY(S.get(&nelem, 4 * (long long)ne));
    XK_TRY(S.get(&eptr, ne + 1));
  }
  XK_CUDA(cudaMemsetAsync(z, 0, zero, st));
  Totals* tot = reinterpret_cast<Totals*>(z);
  int32_t* err = reinterpret_cast<int32_t*>(z + sizeof(Totals));  // err, then serr
  int* words = err + 2;
  int32_t* ecnt = words + w_mem + w_el + w_row;
  // mesh node -> elements (mesh topology: built once per pattern and mesh)
  if (!sides || !pat->node_elem_ready) {
    int32_t *cnt, *fill;
    XK_TRY(S.get(&cnt, nn + 1));
    XK_TRY(S.get(&fill, nn + 1));
    XK_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (nn + 1), st));
    XK_CUDA(cudaMemsetAsync(fill, 0, sizeof(int32_t) * (nn + 1), st));
    if (ne > 0) k_node_elem_count<<<xk_blocks(ne, 256), 256, 0, st>>>(*m, cnt);
    XK_CHECK_LAUNCH();
    XK_TRY(xk_exclusive_scan_i32(cnt, neptr, nn + 1, nullptr, st, &S));
    if (ne > 0) k_node_elem_fill<<<xk_blocks(ne, 256), 256, 0, st>>>(*m, neptr, fill, reinterpret_cast<int2*>(nelem));
    k_segment_sort_pairs<<<xk_blocks(nn, 128), 128, 0, st>>>(neptr, nn, reinterpret_cast<int2*>(nelem));
    XK_CHECK_LAUNCH();
  }
  const int2* node_elem = reinterpret_cast<const int2*>(nelem);
  // members and others
  if (np > 0) {
    auto on = [](const void* q, uintptr_t bytes) { return ((uintptr_t)q & (bytes - 1)) == 0; };
    const MemberScan op = {*m, *p, pat->cap_members, pat->cap_others, pat->members, pat->member_nodes, pat->others,
                           ecnt, tot, on(p->status, 8) && on(p->p_n, 16) && on(pat->member_nodes, 16)};
    XK_TRY(scan_launch(op, np, 1, sums, words, st));
  }
  // member sides per element, incidences per node
  XK_TRY(scan_launch(ElemScan{nn, ne, ecnt, neptr, node_elem, eptr, pat->inc_ptr}, longest, 2,
                     sums + scan_sums(np, 1), words + w_mem, st));
  if (nmx > 0) k_pat_sides<<<xk_blocks(nmx, 256), 256, 0, st>>>(*p, pat->members, tot, pat->cap_members, eptr, ecnt, raw);
  XK_CHECK_LAUNCH();
  g.nn = nn;
  g.ne = ne;
  g.cap = pat->cap_members;
  g.cap_blocks = pat->cap_blocks;
  g.tot = tot;
  g.mnodes = pat->member_nodes;
  g.neptr = neptr;
  g.eptr = eptr;
  g.iptr = pat->inc_ptr;
  g.raw = raw;
  g.nelem = node_elem;
  g.inc = pat->inc;
  g.einc = sides ? pat->elem_inc : nullptr;
  g.err = err;
  g.serr = err + 1;
  g.rptr = pat->row_ptr;
  g.cbase = cbase;
  g.lptr = lower ? pat->low_ptr : nullptr;
  g.col = pat->col;
  g.brow = pat->blk_row;
  g.bptr = pat->blk_ptr;
  g.contrib = pat->contrib;
  g.lblk = lower ? pat->low_blk : nullptr;
  g.bcodes = sides ? pat->bcodes : nullptr;
  const long long warps = (long long)nn + (sides ? ne : 0);
  if (warps > 0) k_pat_cols<<<xk_blocks(warps, RC_WARPS), 32 * RC_WARPS, 0, st>>>(g);
  XK_CHECK_LAUNCH();
  // rows
  XK_TRY(scan_launch(RowScan{nn, g.rcnt, g.ccnt, g.lcnt, pat->row_ptr, cbase, lower ? pat->low_ptr : nullptr, tot},
                     nn + 1, 2, sums + scan_sums(np, 1) + scan_sums(longest, 2), words + w_mem + w_el, st));
  if (nn > 0) k_pat_rows<<<xk_blocks(nn, PR_WARPS), 32 * PR_WARPS, 0, st>>>(g);
  else XK_CUDA(cudaMemsetAsync(pat->blk_ptr, 0, sizeof(int32_t), st));
  XK_CHECK_LAUNCH();
  struct {
    Totals t;
    int32_t err, serr;
  } h;
  XK_CUDA(cudaMemcpyAsync(&h, z, sizeof(h), cudaMemcpyDeviceToHost, st));
  XK_CUDA(cudaStreamSynchronize(st));
  pat->n_members = (int32_t)h.t.members;
  pat->n_others = (int32_t)(np - h.t.members);
  if (sides) pat->node_elem_ready = 1;
  if (h.t.members > pat->cap_members || np - h.t.members > pat->cap_others)
    return xk_set_error(XK_ERR_CAPACITY, "xk_contact_pattern_build: member / other-pair capacity too small");
  if (h.err) return xk_set_error(XK_ERR_OVERFLOW, "xk_contact_pattern_build: a node touches more than 256 contact nodes");
  pat->nnzb = h.t.blocks;
  if (h.t.blocks > pat->cap_blocks)
    return xk_set_error(XK_ERR_CAPACITY, "xk_contact_pattern_build: block capacity too small");
  pat->n_contrib = h.t.contribs;
  pat->nnzb_full = h.t.blocks + (lower ? h.t.low : 0);
  pat->sides_ok = sides && !h.serr ? 1 : 0;
  return XK_OK;
}

static bool aligned32(const void* p) { return ((uintptr_t)p & 31) == 0; }

static xk_status rec_columns(int out_mode, int which, bool tangent, int* c1, int* c2) {
  *c2 = -1;
  if (out_mode == XK_OUT_COMBINED) {
    if (which != XK_WHICH_COMBINED) return xk_set_error(XK_ERR_ARG, "combined records hold only combined values");
    *c1 = tangent ? XK_REC_B : XK_REC_V;
    return XK_OK;
  }
  if (out_mode != XK_OUT_SPLIT) return xk_set_error(XK_ERR_ARG, "out_mode");
  if (tangent) {
    if (which == XK_WHICH_NORMAL) *c1 = 8;
    else if (which == XK_WHICH_FRICTION) *c1 = 17;
    else return xk_set_error(XK_ERR_ARG, "split tangent records need which = normal or friction");
  } else {
    if (which == XK_WHICH_NORMAL) *c1 = 2;
    else if (which == XK_WHICH_FRICTION) *c1 = 5;
    else { *c1 = 2; *c2 = 5; }
  }
  return XK_OK;
}

extern "C" xk_status xk_contact_gather_force(const xk_contact_pattern* pat, const void* rec, int precision,
                                             int out_mode, int which, const double* base, double scale,
                                             const double* f_ext, const uint8_t* fixed, double* out, double* norm2,
                                             xk_stream s) {
  if (!pat || !out) return xk_set_error(XK_ERR_ARG, "xk_contact_gather_force: null argument");
  int c1, c2;
  XK_TRY(rec_columns(out_mode, which, false, &c1, &c2));
  const int rs = out_mode == XK_OUT_COMBINED ? XK_REC_STRIDE_COMBINED : XK_REC_STRIDE_SPLIT;
  const int stc = out_mode == XK_OUT_COMBINED ? XK_REC_S : 0;
  const bool use = pat->n_members > 0 && rec;
  const int32_t* ptr = use ? pat->inc_ptr : nullptr;
  const int32_t* inc = use ? pat->inc : nullptr;
  cudaStream_t st = (cudaStream_t)s;
  const int nn = pat->n_nodes;
  if (nn > 0) {
    if (precision == XK_FP64)
      k_gather_force<double><<<xk_blocks((long long)GF_LANES * nn, 128), 128, 0, st>>>(nn, ptr, inc, (const double*)rec, rs, stc, c1, c2,
                                                                         base, scale, f_ext, fixed, out);
    else if (precision == XK_MIXED)
      k_gather_force<float><<<xk_blocks((long long)GF_LANES * nn, 128), 128, 0, st>>>(nn, ptr, inc, (const float*)rec, rs, stc, c1, c2,
                                                                        base, scale, f_ext, fixed, out);
    else
      return xk_set_error(XK_ERR_ARG, "xk_contact_gather_force: precision");
    XK_CHECK_LAUNCH();
  }
  if (norm2) return xk_sumsq_into(out, 6LL * nn, norm2, st);
  return XK_OK;
}

// xk_contact_gather_force from combined records with the norm fused, for a caller that owns the pattern's
// norm_scratch (calls that overlap on one pattern would race on it).
xk_status xk_contact_gather_force_norm(const xk_contact_pattern* pat, const void* rec, int precision,
                                       const double* base, double scale, const double* f_ext, const uint8_t* fixed,
                                       double* out, double* norm2, xk_stream s) {
  const int nn = pat->n_nodes;
  if (nn <= 0 || !out || !pat->norm_scratch || ((uintptr_t)rec & 15) != 0)
    return xk_contact_gather_force(pat, rec, precision, XK_OUT_COMBINED, XK_WHICH_COMBINED, base, scale, f_ext, fixed,
                                   out, norm2, s);
  const bool use = pat->n_members > 0 && rec;
  const int32_t* ptr = use ? pat->inc_ptr : nullptr;
  const int nb = xk_blocks((long long)GF_LANES * nn, GFN_T);
  unsigned int* count = norm_count(pat->norm_scratch, nn);
  cudaStream_t st = (cudaStream_t)s;
  if (precision == XK_FP64)
    k_gather_force_norm<double><<<nb, GFN_T, 0, st>>>(nn, ptr, pat->inc, (const double*)rec, base, scale, f_ext, fixed,
                                                      out, pat->norm_scratch, count, norm2);
  else
    k_gather_force_norm<float><<<nb, GFN_T, 0, st>>>(nn, ptr, pat->inc, (const float*)rec, base, scale, f_ext, fixed,
                                                     out, pat->norm_scratch, count, norm2);
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_contact_gather_force_elem(const xk_contact_pattern* pat, int precision, const double* base,
                                                  double scale, const double* f_ext, const uint8_t* fixed,
                                                  double* out, double* norm2, xk_stream s) {
  if (!pat || !out) return xk_set_error(XK_ERR_ARG, "xk_contact_gather_force_elem: null argument");
  if (!pat->node_elem_ptr || !pat->node_elem || !pat->elem_sums || (norm2 && !pat->norm_scratch))
    return xk_set_error(XK_ERR_ARG, "xk_contact_gather_force_elem: the element-side pattern was not built");
  if (precision != XK_FP64 && precision != XK_MIXED)
    return xk_set_error(XK_ERR_ARG, "xk_contact_gather_force_elem: precision");
  const int nn = pat->n_nodes, ne = (int)pat->n_elems;
  if (nn <= 0) {
    if (norm2) XK_CUDA(cudaMemsetAsync(norm2, 0, sizeof(double), (cudaStream_t)s));
    return XK_OK;
  }
  const int nb = xk_blocks(nn, GFE_T);  // at most (6 n_nodes + 255) / 256 block sums fit norm_scratch
  double* part = pat->norm_scratch;
  unsigned int* count = norm_count(part, nn);
  const int2* nelem = reinterpret_cast<const int2*>(pat->node_elem);
  const bool vec = ((uintptr_t)base & 15) == 0 && ((uintptr_t)f_ext & 15) == 0 && ((uintptr_t)out & 15) == 0;
  cudaStream_t st = (cudaStream_t)s;
#define XK_GFE(TT, VV)                                                                                           \
  k_gather_force_elem<TT, VV><<<nb, GFE_T, 0, st>>>(nn, ne, pat->node_elem_ptr, nelem, (const TT*)pat->elem_sums, \
                                                    base, scale, f_ext, fixed, out, part, count, norm2)
  if (precision == XK_FP64) {
    if (vec) XK_GFE(double, true); else XK_GFE(double, false);
  } else {
    if (vec) XK_GFE(float, true); else XK_GFE(float, false);
  }
#undef XK_GFE
  XK_CHECK_LAUNCH();
  return XK_OK;
}

extern "C" xk_status xk_contact_gather_tangent(const xk_contact_pattern* pat, const void* rec, int precision,
                                               int out_mode, int which, int variant, void* Kc_vals, xk_stream s) {
  if (!pat || !rec || !Kc_vals) return xk_set_error(XK_ERR_ARG, "xk_contact_gather_tangent: null argument");
  int c1, c2;
  XK_TRY(rec_columns(out_mode, which, true, &c1, &c2));
  if (variant < 0 || variant > XK_GATHER_SIDES_BLOCKS)
    return xk_set_error(XK_ERR_ARG, "xk_contact_gather_tangent: variant");
  const bool sides = variant >= XK_GATHER_SIDES;
  const bool sums = variant != XK_GATHER_SIDES_BLOCKS, blocks = variant != XK_GATHER_SIDES_SUMS;
  if (sides && out_mode == XK_OUT_COMBINED && !(aligned32(rec) && aligned32(pat->elem_sums)))
    return xk_set_error(XK_ERR_ARG, "xk_contact_gather_tangent: rec and elem_sums must be 32-byte aligned");
  if (sides && !(pat->elem_ptr && pat->elem_inc && pat->bcodes && pat->elem_sums && pat->sides_ok == 1))
    return xk_set_error(XK_ERR_ARG, "xk_contact_gather_tangent: the element-side pattern was not built");
  if (pat->nnzb == 0) return XK_OK;
  cudaStream_t st = (cudaStream_t)s;
  const int nb = xk_blocks((pat->nnzb + 31) / 32, GT_WARPS);
  const bool comb = out_mode == XK_OUT_COMBINED;
  // variant: 0 default (chunks for double, lanes for float), 1 lanes, 2 chunks, 3 element sides
  const bool chunks = variant == 2 || (variant == 0 && precision == XK_FP64);
  const int ne = (int)pat->n_elems;
#define XK_GT(TT, RSV, BC)                                                                                   \
  do {                                                                                                      \
    if (sides) {                                                                                            \
      if (sums && ne > 0 && RSV == XK_REC_STRIDE_COMBINED)                                                  \
        k_elem_sums_rec<TT><<<xk_blocks(4LL * ne, 128), 128, 0, st>>>(ne, pat->elem_ptr, pat->elem_inc,     \
                                                                (const TT*)rec, (TT*)pat->elem_sums);       \
      else if (sums && ne > 0)                                                                              \
        k_elem_sums<TT, RSV, BC><<<xk_blocks(9LL * ne, 256), 256, 0, st>>>(ne, pat->elem_ptr, pat->elem_inc,   \
                                                                           (const TT*)rec, (TT*)pat->elem_sums); \
      if (blocks)                                                                                           \
        k_gather_tangent_sides<TT, RSV, BC><<<sides_grid(pat->nnzb, pat->sides_per_sm > 0 ? pat->sides_per_sm : (sizeof(TT) == 4 ? 16 : 8)), GS_T, 0, st>>>( \
            pat->nnzb, reinterpret_cast<const int4*>(pat->bcodes), (const TT*)pat->elem_sums, (const TT*)rec,  \
            (TT*)Kc_vals);                                                                                  \
    } else if (chunks)                                                                                      \
      k_gather_tangent<TT, RSV, BC><<<nb, 32 * GT_WARPS, 0, st>>>(pat->nnzb, pat->blk_ptr, pat->contrib,     \
                                                                  (const TT*)rec, (TT*)Kc_vals);            \
    else                                                                                                    \
      k_gather_tangent_lanes<TT, RSV, BC><<<xk_blocks((pat->nnzb + 31) / 32, 4), 128, 0, st>>>(             \
          pat->nnzb, pat->blk_ptr, pat->contrib, (const TT*)rec, (TT*)Kc_vals);                             \
  } while (0)
  if (precision == XK_FP64) {
    if (comb) XK_GT(double, 16, XK_REC_B);
    else if (c1 == 8) XK_GT(double, 32, 8);
    else XK_GT(double, 32, 17);
  } else if (precision == XK_MIXED) {
    if (comb) XK_GT(float, 16, XK_REC_B);
    else if (c1 == 8) XK_GT(float, 32, 8);
    else XK_GT(float, 32, 17);
  } else {
    return xk_set_error(XK_ERR_ARG, "xk_contact_gather_tangent: precision");
  }
#undef XK_GT
  XK_CHECK_LAUNCH();
  return XK_OK;
}
