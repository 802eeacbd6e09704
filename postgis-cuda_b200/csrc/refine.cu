// Exact refinement of candidate pairs: ST_Intersects, intersection area (Green's theorem over the boundary
// pieces inside the other polygon, product-rule weights on shared boundaries) and DE-9IM evidence, one warp per
// pair. Restates the decisions of the reference's k_refine / edge_contrib_loc (engine/engine.cuh:333-636) with
// its lane ownership kept (lane l owns local edges l, l+32, ...; A's then B's; shfl_down tree 16..1), so the
// FP64 area and boundary-length sums have one fixed rounding order: bit-identical to the CPU oracle.
//
// Pairs whose local edge lists fit CAP run from shared memory, a warp each; larger pairs are queued and re-run by
// k_refine_block (filtered: a block each) and, beyond its lists, k_refine_scratch (per-warp lists in global scratch); the
// filtered bin's pairs with an edge of many split points by k_refine_split.
//
// Two variants with the same decisions and the same FP64 values:
//  - plain (F = false): the reference's sweeps, FP64 box tests (refine_pair_t<false>).
//  - filtered (F = true): candidate edge pairs first, then only the work they need (refine_pair_m in the shared-memory
//    bins, refine_pair_t<true, FLAT> in the scratch bin). Box rejection tests are plain comparisons (max(a, b) < x  <=>
//    a < x && b < x for finite values) instead of FP64 min/max, which on sm_100a issue on the XU pipe. Containment probes
//    are tested by the whole warp (crossing parity is order-free).
#include <type_traits>
#include "engine.h"
#include "pairkit.cuh"

namespace gsj {

constexpr int CAP = 128;                         // plain: local edges per polygon per warp in shared memory
constexpr int RB_WARPS = 4;                      // warps per block
constexpr size_t EDGE_BYTES = 4 * sizeof(double) + sizeof(uint32_t);
constexpr size_t LIST_BYTES = CAP * EDGE_BYTES;  // one list
constexpr size_t RB_SMEM = (size_t)RB_WARPS * 2 * LIST_BYTES;
constexpr int U_GLOBAL = 2;   // edges a step of the sweeps over lists in global memory
constexpr int CAP_F = 128;                       // filtered: local edges per polygon per warp (a multiple of 32, below 256)
constexpr size_t EDGE_BYTES_8 = 4 * sizeof(double) + 1;   // filtered shared-memory bins: flags in a byte

struct PairGeo { Box ov; double tol, eps_par, snap, cx, cy; };

// Candidate edge pairs of the filtered variant: every (i, j) of A's and B's local edges whose boxes come within
// 2 tol of each other - a superset of the pairs any box test of the pair routine keeps (those use tol or no pad).
// Built by one lane-balanced sweep over the na x nb grid (ballot compaction keeps (i, j) order); per-edge
// ranges: A edge i owns cp[sa[i] .. sa[i+1]), B edge j owns pj[(j ? sb[j-1] : 0) .. sb[j]) (entries in i order).
// Large grids are searched by buckets instead: NBK slabs along the overlap box's longer side, B's edges listed per
// slab (bl, boff), each lane scanning only its A edge's slabs and reporting a pair once, in the first slab both
// edges reach; the lane sorts its few candidates (at most LCAP) so the list keeps (i, j) order.
// Only the oversized pairs of the scratch kernel use the buckets: for the shared-memory bins the grid is faster.
constexpr int NBK = 16, LCAP = 32;
constexpr int GRID_MAX = 2048;   // scratch kernel: na x nb up to this: the grid sweep
// cap: entries of cp / pj; rec: a self pair's recorded contributions, one per A edge (the scratch kernel's B list)
struct FlatBuf { uint32_t* cp; uint16_t* pj; uint32_t* sa; uint32_t* sb; uint32_t* bl; uint32_t* boff; int cap, blcap; double* rec; };

__device__ __forceinline__ void warp_exscan(uint32_t* a, int n, int lane) {   // in place over a[0 .. n)
  uint32_t run = 0;
  for (int base = 0; base < n; base += 32) {
    const int t = base + lane;
    const uint32_t v = t < n ? a[t] : 0u;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (t < n) a[t] = run + x - v;
    run += __shfl_sync(0xffffffffu, x, 31);
  }
  __syncwarp();
}

// Bucketed search (large grids): fills cp in (i, j) order with the per-edge counts in sa / sb and returns the
// number of candidates, or -1 when a bucket list or a lane's candidate buffer would overflow.
__device__ int bucket_candidates(const EList& LA, int na, const EList& LB, int nb, double pad, const Box& ov, const FlatBuf& fb, int lane) {
  const bool ax = (ov.x1 - ov.x0) >= (ov.y1 - ov.y0);
  const double o0 = ax ? ov.x0 : ov.y0, len = ax ? ov.x1 - ov.x0 : ov.y1 - ov.y0;
  const double inv = len > 0 ? NBK / len : 0.0;
  auto bk = [&](double v) {   // monotone in v
    const double t = (v - o0) * inv;
    return t < 1.0 ? 0 : (t >= (double)(NBK - 1) ? NBK - 1 : (int)t);
  };
  const unsigned lt = (1u << lane) - 1;
  if (lane <= NBK) fb.boff[lane] = 0;
  __syncwarp();
  for (int j = lane; j < nb; j += 32) {   // slab span of each B edge (kept in pj until the scatter)
    const double c0 = ax ? LB.x0[j] : LB.y0[j], c1 = ax ? LB.x1[j] : LB.y1[j];
    const int s0 = bk(c0 < c1 ? c0 : c1), s1 = bk(c0 < c1 ? c1 : c0);
    fb.pj[j] = (uint16_t)(s0 | (s1 << 8));
    for (int b2 = s0; b2 <= s1; b2++) atomicAdd(&fb.boff[b2], 1u);
  }
  __syncwarp();
  warp_exscan(fb.boff, NBK + 1, lane);
  if ((int)fb.boff[NBK] > fb.blcap) return -1;
  for (int b2 = 0; b2 < NBK; b2++) {   // stable lists: B edges of slab b2 in increasing j
    int run = 0;
    for (int j0 = 0; j0 < nb; j0 += 32) {
      const int j = j0 + lane;
      int s0 = 0;
      bool cov = false;
      if (j < nb) { const uint32_t sp = fb.pj[j]; s0 = (int)(sp & 0xFFu); cov = s0 <= b2 && b2 <= (int)(sp >> 8); }
      const unsigned m = __ballot_sync(0xffffffffu, cov);
      if (cov) fb.bl[fb.boff[b2] + run + __popc(m & lt)] = (uint32_t)j | ((uint32_t)s0 << 16);
      run += __popc(m);
    }
  }
  __syncwarp();
  int cnt = 0;
  for (int t0 = 0; t0 < na; t0 += 32) {
    const int i = t0 + lane;
    int ni = 0;
    uint16_t lc[LCAP];
    if (i < na) {
      const double px = LA.x0[i], py = LA.y0[i], qx = LA.x1[i], qy = LA.y1[i];
      const double ax0 = (px < qx ? px : qx) - pad, ax1 = (px < qx ? qx : px) + pad;
      const double ay0 = (py < qy ? py : qy) - pad, ay1 = (py < qy ? qy : py) + pad;
      const int s0 = bk(ax ? ax0 : ay0), s1 = bk(ax ? ax1 : ay1);
      for (int b2 = s0; b2 <= s1; b2++)
        for (uint32_t e = fb.boff[b2]; e < fb.boff[b2 + 1]; e++) {
          const uint32_t v = fb.bl[e];
          const int j = (int)(v & 0xFFFFu), sj = (int)(v >> 16);
          if ((sj > s0 ? sj : s0) != b2) continue;   // the pair belongs to the first slab both edges reach
          if (out_cmp(LB.x0[j], LB.y0[j], LB.x1[j], LB.y1[j], ax0, ay0, ax1, ay1)) continue;
          if (ni < LCAP) lc[ni] = (uint16_t)j;
          ni++;
        }
      if (ni <= LCAP)
        for (int u = 1; u < ni; u++) {
          const uint16_t v = lc[u];
          int w = u - 1;
          while (w >= 0 && lc[w] > v) { lc[w + 1] = lc[w]; w--; }
          lc[w + 1] = v;
        }
    }
    if (__any_sync(0xffffffffu, ni > LCAP)) return -1;
    int x = ni;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int off = cnt + x - ni;
    if (i < na) {
      fb.sa[i] = (uint32_t)ni;
      for (int k = 0; k < ni; k++) {
        if (off + k < fb.cap) fb.cp[off + k] = (uint32_t)i | ((uint32_t)lc[k] << 16);
        atomicAdd(&fb.sb[lc[k]], 1u);
      }
    }
    cnt += __shfl_sync(0xffffffffu, x, 31);
  }
  __syncwarp();
  return cnt;
}

// returns the number of candidate pairs (> fb.cap: the lists were not kept)
template <bool BUCKETS>
__device__ int flat_candidates(const EList& LA, int na, const EList& LB, int nb, double pad, const Box& ov, const FlatBuf& fb, int lane) {
  for (int t = lane; t <= na; t += 32) fb.sa[t] = 0;
  for (int t = lane; t <= nb; t += 32) fb.sb[t] = 0;
  __syncwarp();
  if (na == 0 || nb == 0) return 0;
  const unsigned lt = (1u << lane) - 1;
  const int total = na * nb;
  int cnt = -1;
  if (BUCKETS && total > GRID_MAX) {
    cnt = bucket_candidates(LA, na, LB, nb, pad, ov, fb, lane);
    if (cnt < 0) {   // overflowed: count afresh with the grid
      for (int t = lane; t <= na; t += 32) fb.sa[t] = 0;
      for (int t = lane; t <= nb; t += 32) fb.sb[t] = 0;
      __syncwarp();
    }
  }
  if (cnt < 0) {
  const int qi = 32 / nb, qj = 32 % nb;
  int i = lane / nb, j = lane % nb;
  cnt = 0;
  for (int base = 0; base < total; base += 32) {
    bool keep = false;
    if (base + lane < total) {
      const double px = LA.x0[i], py = LA.y0[i], qx = LA.x1[i], qy = LA.y1[i];
      const double ax0 = (px < qx ? px : qx) - pad, ax1 = (px < qx ? qx : px) + pad;
      const double ay0 = (py < qy ? py : qy) - pad, ay1 = (py < qy ? qy : py) + pad;
      keep = !out_cmp(LB.x0[j], LB.y0[j], LB.x1[j], LB.y1[j], ax0, ay0, ax1, ay1);
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    const int pos = cnt + __popc(m & lt);
    if (keep && pos < fb.cap) {
      fb.cp[pos] = (uint32_t)i | ((uint32_t)j << 16);
      atomicAdd(&fb.sa[i], 1u);
      atomicAdd(&fb.sb[j], 1u);
    }
    cnt += __popc(m);
    i += qi; j += qj;
    if (j >= nb) { j -= nb; i++; }
  }
  }
  if (cnt > fb.cap) return cnt;
  __syncwarp();
  warp_exscan(fb.sa, na + 1, lane);
  warp_exscan(fb.sb, nb + 1, lane);
  // stable scatter by j: entries of one B edge keep their (increasing i) order
  for (int base = 0; base < cnt; base += 32) {
    const int e = base + lane;
    const bool v = e < cnt;
    const uint32_t jj = v ? (fb.cp[e] >> 16) : 0xFFFFFu;
    const unsigned peers = __match_any_sync(0xffffffffu, jj);
    if (v) fb.pj[fb.sb[jj] + __popc(peers & lt)] = (uint16_t)e;
    __syncwarp();
    if (v && (peers & lt) == 0) fb.sb[jj] += __popc(peers);
    __syncwarp();
  }
  return cnt;
}

// Green's-theorem contribution of edge p->q within the other polygon + relate lengths (engine.cuh:416-515), in three
// steps: the edge's cuts (split points and coincident intervals against the other polygon's edges), its segments
// between consecutive split points, each segment's value.
struct EdgeRef { double px, py, qx, qy, dx, dy, len2, len; uint32_t fl; };   // len: where lengths are wanted
struct EdgeCuts {
  double ts[MAXS]; int ns;
  double ol0[MAXO], ol1[MAXO]; bool osame[MAXO]; int oidx[MAXO]; int no;
};
struct Segment { double t0, t1, mx, my; int net, first, net_real, n_real; bool valid, need; };

template <class EL>
__device__ __forceinline__ EdgeRef edge_ref(const EL& L, int i, bool rel) {
  EdgeRef e;
  e.px = L.x0[i]; e.py = L.y0[i]; e.qx = L.x1[i]; e.qy = L.y1[i]; e.fl = L.fl[i];
  e.dx = e.qx - e.px; e.dy = e.qy - e.py;
  e.len2 = e.dx * e.dx + e.dy * e.dy;
  e.len = rel ? sqrt(e.len2) : 0.0;
  return e;
}

// the cuts that edge k of the other polygon makes
template <bool F, class EL>
__device__ __forceinline__ void edge_visit(EdgeCuts& C, const EdgeRef& e, const EL& L, int k, const PairGeo& G) {
  const double px = e.px, py = e.py, qx = e.qx, qy = e.qy, dx = e.dx, dy = e.dy, len2 = e.len2, tol = G.tol;
  const double ex0 = L.x0[k], ey0 = L.y0[k], ex1 = L.x1[k], ey1 = L.y1[k];
  const double bx0 = fmin(px, qx) - tol, bx1 = fmax(px, qx) + tol, by0 = fmin(py, qy) - tol, by1 = fmax(py, qy) + tol;
  if (F ? out_cmp(ex0, ey0, ex1, ey1, bx0, by0, bx1, by1)
        : (fmax(ex0, ex1) < bx0 || fmin(ex0, ex1) > bx1 || fmax(ey0, ey1) < by0 || fmin(ey0, ey1) > by1)) return;
  const double tol2len2 = tol * tol * len2, eps2 = G.eps_par * G.eps_par, snap2 = G.snap * G.snap;
  const uint32_t efl = L.fl[k], cut = e.fl;
  const double fx = ex1 - ex0, fy = ey1 - ey0;
  const double r = dx * fy - dy * fx;
  const double flen2 = fx * fx + fy * fy;
  const double c0 = orient(px, py, qx, qy, ex0, ey0), c1 = orient(px, py, qx, qy, ex1, ey1);
  bool col = (c0 * c0 <= snap2 * len2 || ((efl & 2u) && c0 * c0 <= tol2len2)) && (c1 * c1 <= snap2 * len2 || ((efl & 4u) && c1 * c1 <= tol2len2));
  if (!col && flen2 > 0) {
    const double g0 = orient(ex0, ey0, ex1, ey1, px, py), g1 = orient(ex0, ey0, ex1, ey1, qx, qy), tf = tol * tol * flen2;
    col = (g0 * g0 <= snap2 * flen2 || ((cut & 2u) && g0 * g0 <= tf)) && (g1 * g1 <= snap2 * flen2 || ((cut & 4u) && g1 * g1 <= tf));
  }
  // the ends of a coincident interval, or the parameters of a crossing on both edges: n1 / d and n2 / d
  const double wx = ex0 - px, wy = ey0 - py;
  double n1, n2, d;
  if (col) {
    d = len2; n1 = wx * dx + wy * dy; n2 = (ex1 - px) * dx + (ey1 - py) * dy;
  } else {
    if (!(r * r > eps2 * len2 * flen2)) return;
    d = r; n1 = wx * fy - wy * fx;
    if (r > 0 ? (n1 <= 0 || n1 >= r) : (n1 >= 0 || n1 <= r)) return;
    n2 = wx * dy - wy * dx;
  }
  // n / d is n for n = +-0 (up to the zero's sign, which no test reads) and exactly 1 for n = d: a coincident edge's ends need no division
  n1 = n1 == 0.0 ? 0.0 : (n1 == d ? 1.0 : n1 / d);
  n2 = n2 == 0.0 ? 0.0 : (n2 == d ? 1.0 : n2 / d);
  if (col) {
    const double lo = fmax((double)0, fmin(n1, n2)), hi = fmin((double)1, fmax(n1, n2));
    if (hi > lo) {
      if (lo > 0 && C.ns < MAXS) C.ts[C.ns++] = lo;
      if (hi < 1 && C.ns < MAXS) C.ts[C.ns++] = hi;
      if (C.no < MAXO) { C.ol0[C.no] = lo; C.ol1[C.no] = hi; C.osame[C.no] = (dx * fx + dy * fy) > 0; C.oidx[C.no] = k; C.no++; }
    }
  } else {
    bool in = n2 >= 0 && n2 <= 1;
    if (!in) {
      const double du = tol / (flen2 > 0 ? sqrt(flen2) : (double)1);
      in = n2 >= -du && n2 <= 1 + du;
    }
    if (in && C.ns < MAXS) C.ts[C.ns++] = n1;
  }
}
__device__ __forceinline__ void edge_cuts_begin(EdgeCuts& C) { C.ts[0] = 0; C.ts[1] = 1; C.ns = 2; C.no = 0; }
__device__ __forceinline__ void edge_cuts_sort(EdgeCuts& C) {
#pragma unroll 1
  for (int a = 1; a < C.ns; a++) {
    const double v = C.ts[a];
    int b = a - 1;
#pragma unroll 1
    while (b >= 0 && C.ts[b] > v) { C.ts[b + 1] = C.ts[b]; b--; }
    C.ts[b + 1] = v;
  }
}

// segment k of the edge: its midpoint, the coincident intervals over it, and whether the inside test of the midpoint
// is read by its value (lens: lengths are wanted and the edge is real; AREA: the area term is wanted)
template <bool AREA = true, class EL>
__device__ __forceinline__ Segment edge_segment(const EdgeCuts& C, const EdgeRef& e, const EL& L, int k, const PairGeo& G, bool lens) {
  Segment s;
  s.t0 = C.ts[k]; s.t1 = C.ts[k + 1];
  s.valid = s.t1 > s.t0;
  const double tm = (double)0.5 * (s.t0 + s.t1);
  s.mx = e.px + e.dx * tm; s.my = e.py + e.dy * tm;
  s.net = 0; s.first = -1; s.net_real = 0; s.n_real = 0;
#pragma unroll 1
  for (int o = 0; o < C.no; o++)
    if (tm > C.ol0[o] && tm < C.ol1[o]) {
      const int sgn = C.osame[o] ? 1 : -1;
      s.net += sgn; if (s.first < 0) s.first = o;
      if (!(L.fl[C.oidx[o]] & 1u)) { s.net_real += sgn; s.n_real++; }
    }
  const bool half = s.net == 1 || s.net == -1;
  const bool in_ov = s.mx >= G.ov.x0 && s.mx <= G.ov.x1 && s.my >= G.ov.y0 && s.my <= G.ov.y1;
  s.need = s.valid && in_ov && ((AREA && (s.first < 0 || !half)) || (lens && s.net_real == 0 && !(s.n_real == 0 && half)));
  return s;
}
// adds the segment's length to l_in / l_on and its term to acc (AREA); vin: the midpoint is inside (false where not needed)
template <bool AREA = true, class EL>
__device__ __forceinline__ void edge_segment_add(const Segment& s, const EdgeCuts& C, const EdgeRef& e, const EL& L, const PairGeo& G, bool lens, int vin,
                                                 double& acc, double& l_in, double& l_on, uint32_t& bits) {
  const int net = s.net;
  if (lens) {
    const double seg = e.len * (s.t1 - s.t0);
    if (s.net_real != 0) { l_on += seg; bits |= (s.net_real > 0 ? REL_COIN_SAME : REL_COIN_OPP) | REL_TOUCH; }
    else if (s.n_real == 0 && (net == 1 || net == -1)) l_in += 0.5 * seg;
    else if (vin) l_in += seg;
  }
  if constexpr (!AREA) return;
  double w;
  if (s.first < 0) w = vin ? 1.0 : 0.0;
  else if (net == 1 || net == -1) w = 0.5;
  else if (net == 0) w = vin ? 1.0 : 0.0;
  else {
    const int fo = C.oidx[s.first];
    const bool sb = left_of(L.x0[fo], L.y0[fo], L.x1[fo], L.y1[fo], s.mx, s.my);
    const bool m_left = C.osame[s.first] ? sb : !sb;
    int other = m_left ? vin - net : vin + net;
    other = other < 0 ? 0 : (other > 1 ? 1 : other);
    w = 0.5 * (vin + other);
  }
  if (w != 0.0) {
    const double ax = e.px + e.dx * s.t0 - G.cx, ay = e.py + e.dy * s.t0 - G.cy, bx = e.px + e.dx * s.t1 - G.cx, by = e.py + e.dy * s.t1 - G.cy;
    acc += w * (double)(ax * by - ay * bx);
  }
}

// One edge by one lane. each_k(visit) calls visit(k) for the other polygon's local edges k in increasing order: all of
// them, or only those of a candidate list that holds every k passing the box test (the same visits, the same results).
template <bool F, int U, class EL, class EachK>
__device__ double edge_contrib_k(const EL& LS, int i, const EL& L, int cnt, bool in_c, const PairGeo& G, bool rel, double& l_in, double& l_on, uint32_t& bits,
                                 EachK&& each_k) {
  const EdgeRef e = edge_ref(LS, i, rel);
  if (e.len2 == 0) return 0.0;
  const bool lens = rel && !(e.fl & 1u);
  EdgeCuts C;
  edge_cuts_begin(C);
  each_k([&](int k) { edge_visit<F>(C, e, L, k, G); });
  edge_cuts_sort(C);
  double acc = 0.0;
#pragma unroll 1
  for (int k = 0; k + 1 < C.ns; k++) {
    const Segment s = edge_segment(C, e, L, k, G, lens);
    if (!s.valid) continue;
    const int vin = s.need && inside_from_c<F, U>(L, cnt, G.cx, G.cy, in_c, s.mx, s.my) ? 1 : 0;
    edge_segment_add(s, C, e, L, G, lens, vin, acc, l_in, l_on, bits);
  }
  return acc;
}
template <bool F, int U, class EL>
__device__ __forceinline__ double edge_contrib(const EL& LS, int i, const EL& L, int cnt, bool in_c, const PairGeo& G, bool rel, double& l_in, double& l_on,
                                               uint32_t& bits) {
  return edge_contrib_k<F, U>(LS, i, L, cnt, in_c, G, rel, l_in, l_on, bits, [&](auto&& visit) {
#pragma unroll U
    for (int k = 0; k < cnt; k++) visit(k);
  });
}

__device__ __forceinline__ double pair_snap(double2 oa, double2 ea) {   // engine.cuh:524-527
  const double m = fmax(fmax(fabs(oa.x), fabs(oa.x + ea.x)), fmax(fabs(oa.y), fabs(oa.y + ea.y)));
  return 0.5 * (__longlong_as_double(__double_as_longlong(m) + 1) - m);   // the next double up: m >= 0
}

// a lane's share of a pair's sums: twice the signed area, lengths of A inside / on B and of B inside / on A
struct PairSums { double s2 = 0.0, ai = 0.0, ao = 0.0, bi = 0.0, bo = 0.0; };
template <bool AREA = true, bool REL = true>
__device__ __forceinline__ void pair_result(const PairSums& S, bool sums, bool hit, bool rtouch, uint32_t bits, uint8_t& o_flag, double& o_area, double4& o_ev,
                                            uint32_t& o_evb) {
  double ar = 0.0; double4 e4 = make_double4(0, 0, 0, 0); uint32_t eb4 = rtouch ? REL_TOUCH : 0;
  if (sums) {
    double s2 = S.s2;
    if (REL) e4 = make_double4(S.ai, S.ao, S.bi, S.bo);
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {   // warp_sum of the five, side by side
      if (AREA) s2 += __shfl_down_sync(0xffffffffu, s2, o);
      if (REL) {
        e4.x += __shfl_down_sync(0xffffffffu, e4.x, o); e4.y += __shfl_down_sync(0xffffffffu, e4.y, o);
        e4.z += __shfl_down_sync(0xffffffffu, e4.z, o); e4.w += __shfl_down_sync(0xffffffffu, e4.w, o);
      }
    }
    ar = 0.5 * s2;
    eb4 = __reduce_or_sync(0xffffffffu, bits);
  }
  const bool ev_any = e4.x != 0 || e4.y != 0 || e4.z != 0 || e4.w != 0;
  o_flag = hit ? 1 : ((ar != 0.0 || ev_any) ? 2 : 0);
  o_area = ar; o_ev = e4; o_evb = eb4;
}

// geometry of a pair in the frame of A's origin: overlap box, tolerances, the probe point c
__device__ __forceinline__ PairGeo pair_geo(const DLayer& P, const DLayer& R, uint32_t a, uint32_t b, const RefineArgs& rp, Frame& A, Frame& B) {
  const double2 oa = P.origin[a], ob = R.origin[b], ea = P.ext[a], eb = R.ext[b];
  const double sx = ob.x - oa.x, sy = ob.y - oa.y;
  const double pad = 4.0 * fmax(rp.tol_abs, (double)rp.tol_rel * fmax(fmax(ea.x, ea.y), fmax(eb.x, eb.y)));
  PairGeo G;
  G.ov = Box{fmax(0.0, sx) - pad, fmax(0.0, sy) - pad, fmin(ea.x, sx + eb.x) + pad, fmin(ea.y, sy + eb.y) + pad};
  A = frame_of(P, a, oa.x, oa.y); B = frame_of(R, b, oa.x, oa.y);
  G.tol = fmax(rp.tol_abs, (double)rp.tol_rel * fmax(G.ov.x1 - G.ov.x0, G.ov.y1 - G.ov.y0));
  G.eps_par = rp.eps_par;
  G.snap = rp.snap_half_ulp ? pair_snap(oa, ea) : 0.0;
  G.cx = (double)(G.ov.x0 + 0.381966 * (G.ov.x1 - G.ov.x0));
  G.cy = (double)(G.ov.y0 + 0.414213 * (G.ov.y1 - G.ov.y0));
  return G;
}

// One pair, whole warp. Returns false when a local list exceeded cap (nothing written).
// FLAT (the filtered scratch kernel): candidate lists in global scratch; a pair whose list would exceed fb->cap is
// handed back (false) and runs with the full sweeps.
// SELF (FLAT only): the pair is a geometry with itself in one layer; the caller passes one list as both LA and LB.
// B's gather and B's contribution pass would repeat A's exactly (the same edges in the same frame, the same candidates
// in the same order, so the same values): A's pass runs once and each lane adds its recorded values a second time, in
// the same order, which is the sum the two passes make.
// U: edges a step of the sweeps. Lists in shared memory are swept one by one (code size), lists in global memory two at a time, so
// that their loads overlap. Refinement, 1 / 2 / 4 at a time: plain relate self-join of 5k parcels 4.08 / 3.26 / 3.29 ms, of
// 100k 21.7 / 20.4 / 23.2; pairs of 2000-8000 edges, filtered, 115.5 / 105.6 / 101.0; allocation-free call, 20k parcels, 13.9 / 11.1 / 19.5.
template <bool F, int U, bool FLAT = false, bool BUCKETS = false, bool SELF = false>
__device__ bool refine_pair_t(const DLayer& P, const DLayer& R, uint32_t a, uint32_t b, const RefineArgs& rp, EList LA, EList LB, int cap,
                              int lane, uint8_t& o_flag, double& o_area, double4& o_ev, uint32_t& o_evb, const FlatBuf* fb = nullptr,
                              unsigned long long* ep = nullptr) {
  Frame A, B;
  const PairGeo G = pair_geo(P, R, a, b, rp, A, B);
  int na = 0, nb = 0;
#pragma unroll 1
  for (int side = 0; side < (SELF ? 1 : 2); side++) {   // one inlined copy of the gather
    const int n = collect<F>(side ? B : A, G.ov, side ? LB : LA, cap, lane);
    if (side) nb = n; else na = n;
  }
  if constexpr (SELF) nb = na;
  if (na > cap || nb > cap) return false;
  __syncwarp();
  int ncp = -1;   // candidate edge pairs (FLAT); -1: sweep every edge pair
  if constexpr (FLAT) {
    ncp = flat_candidates<BUCKETS>(LA, na, LB, nb, 2.0 * G.tol, G.ov, *fb, lane);
    if (ncp > fb->cap) return false;
  }
  // boundary contact
  bool hit = false, hit_any = false;
  if constexpr (FLAT) {
    // one candidate per lane; the warp stops at the first real contact (hit_any is then implied)
#pragma unroll 1
    for (int base = 0; base < ncp; base += 32) {
      const int e = base + lane;
      if (e < ncp) {
        const uint32_t c = fb->cp[e];
        const int i = (int)(c & 0xFFFFu), j = (int)(c >> 16);
        const double px0 = LA.x0[i], py0 = LA.y0[i], px1 = LA.x1[i], py1 = LA.y1[i];
        const double qx0 = LB.x0[j], qy0 = LB.y0[j], qx1 = LB.x1[j], qy1 = LB.y1[j];
        const double ax0 = px0 < px1 ? px0 : px1, ax1 = px0 < px1 ? px1 : px0, ay0 = py0 < py1 ? py0 : py1, ay1 = py0 < py1 ? py1 : py0;
        if (!out_cmp(qx0, qy0, qx1, qy1, ax0, ay0, ax1, ay1) && seg_isect(px0, py0, px1, py1, qx0, qy0, qx1, qy1)) {
          hit_any = true;
          if (!((LA.fl[i] | LB.fl[j]) & 1u)) hit = true;
        }
      }
      if (__any_sync(0xffffffffu, hit)) { hit = true; break; }
    }
  } else {
    auto seg_loop = [&](int i) {
      const double px0 = LA.x0[i], py0 = LA.y0[i], px1 = LA.x1[i], py1 = LA.y1[i];
      const uint32_t fa = LA.fl[i];
      const double ax0 = fmin(px0, px1), ax1 = fmax(px0, px1), ay0 = fmin(py0, py1), ay1 = fmax(py0, py1);
      auto test = [&](int j) {
        const double qx0 = LB.x0[j], qy0 = LB.y0[j], qx1 = LB.x1[j], qy1 = LB.y1[j];
        if (F ? out_cmp(qx0, qy0, qx1, qy1, ax0, ay0, ax1, ay1)
              : (fmax(qx0, qx1) < ax0 || fmin(qx0, qx1) > ax1 || fmax(qy0, qy1) < ay0 || fmin(qy0, qy1) > ay1)) return false;
        if (seg_isect(px0, py0, px1, py1, qx0, qy0, qx1, qy1)) {
          hit_any = true;
          if (!((fa | LB.fl[j]) & 1u)) { hit = true; return true; }
        }
        return false;
      };
#pragma unroll U
      for (int j = 0; j < nb; j++) if (test(j)) break;
    };
#pragma unroll 1
    for (int i = lane; i < na && !hit; i += 32) seg_loop(i);
  }
  hit = __any_sync(0xffffffffu, hit);
  hit_any = __any_sync(0xffffffffu, hit_any || hit);
  const bool rtouch = hit;
  bool inB_c = false, inA_c = false;
  if (!hit || rp.want_area || rp.want_relate)
#pragma unroll 1
    for (int side = 0; side < 2; side++) {
      const bool in = pip_full_warp(side ? A : B, G.cx, G.cy, lane);
      if (side) inA_c = in; else inB_c = in;
    }
  bool contain_any = false;
  if (!hit) {
    if constexpr (F) {
      hit = contains_warp<false>(A, B, LA, na, LB, nb, inA_c, inB_c, G.ov, G.cx, G.cy, lane, contain_any);
    } else {   // no real boundary contact: intersects iff a real-edge vertex of one lies inside the other (engine.cuh:577-594)
      bool h = false, ha = false;
#pragma unroll 1
      for (uint32_t r = A.r0 + lane; r < A.r1 && !h; r += 32) {
        double x, y; const bool real = probe_vertex(A, r, x, y);
        if (!real) A.v(P.rvo[r], x, y);
        if (x >= G.ov.x0 && x <= G.ov.x1 && y >= G.ov.y0 && y <= G.ov.y1 && inside_from_c<F, U>(LB, nb, G.cx, G.cy, inB_c, x, y)) { ha = true; h = real; }
      }
#pragma unroll 1
      for (uint32_t r = B.r0 + lane; r < B.r1 && !h; r += 32) {
        double x, y; const bool real = probe_vertex(B, r, x, y);
        if (!real) B.v(R.rvo[r], x, y);
        if (x >= G.ov.x0 && x <= G.ov.x1 && y >= G.ov.y0 && y <= G.ov.y1 && inside_from_c<F, U>(LA, na, G.cx, G.cy, inA_c, x, y)) { ha = true; h = real; }
      }
      hit = __any_sync(0xffffffffu, h);
      contain_any = __any_sync(0xffffffffu, ha);
    }
  }
  PairSums S;
  uint32_t bits = rtouch ? REL_TOUCH : 0;
  const bool sums = (hit || hit_any || contain_any) && (rp.want_area || rp.want_relate);
  if (sums) {
    const bool rel = rp.want_relate != 0;
    if constexpr (FLAT && SELF) {   // the self pair's A pass, recorded per edge, then added again in order
      const uint32_t* cp = fb->cp;
#pragma unroll 1
      for (int i = lane; i < na; i += 32) {
        const int r0 = (int)fb->sa[i], r1 = (int)fb->sa[i + 1];
        const double v = edge_contrib_k<F, U>(LA, i, LB, nb, inB_c, G, rel, S.ai, S.ao, bits, [&](auto&& visit) {
#pragma unroll 1
          for (int e = r0; e < r1; e++) visit((int)(cp[e] >> 16));
        });
        fb->rec[i] = v;
        S.s2 += v;
      }
#pragma unroll 1
      for (int i = lane; i < na; i += 32) S.s2 += fb->rec[i];
      S.bi = S.ai; S.bo = S.ao;
    } else if constexpr (FLAT) {   // visit only each edge's candidates, in the same increasing order; one call site for both passes
      const uint32_t* cp = fb->cp;
      const uint16_t* pj = fb->pj;
#pragma unroll 1
      for (int pass = 0; pass < 2; pass++) {
        const EList& LS = pass ? LB : LA;
        const EList& LO = pass ? LA : LB;
        const int nself = pass ? nb : na, nother = pass ? na : nb;
        const bool inc = pass ? inA_c : inB_c;
        double lin = 0.0, lon = 0.0;   // this pass's lengths (each starts from 0, so the sums are the same)
#pragma unroll 1
        for (int i = lane; i < nself; i += 32) {
          const int r0 = pass ? (i ? (int)fb->sb[i - 1] : 0) : (int)fb->sa[i];
          const int r1 = pass ? (int)fb->sb[i] : (int)fb->sa[i + 1];
          S.s2 += edge_contrib_k<F, U>(LS, i, LO, nother, inc, G, rel, lin, lon, bits, [&](auto&& visit) {
#pragma unroll 1
            for (int e = r0; e < r1; e++) visit(pass ? (int)(cp[pj[e]] & 0xFFFFu) : (int)(cp[e] >> 16));
          });
        }
        if (pass) { S.bi = lin; S.bo = lon; } else { S.ai = lin; S.ao = lon; }
      }
    } else {
#pragma unroll 1
      for (int i = lane; i < na; i += 32) S.s2 += edge_contrib<F, U>(LA, i, LB, nb, inB_c, G, rel, S.ai, S.ao, bits);
#pragma unroll 1
      for (int i = lane; i < nb; i += 32) S.s2 += edge_contrib<F, U>(LB, i, LA, na, inA_c, G, rel, S.bi, S.bo, bits);
    }
  }
  pair_result(S, sums, hit, rtouch, bits, o_flag, o_area, o_ev, o_evb);
  if (ep && lane == 0) *ep += (unsigned long long)na * (unsigned long long)nb;   // local edge pairs: the refinement's work unit
  return true;
}

// the plain routine, callable from other translation units (the allocation-free entry point)
__device__ bool refine_pair(const DLayer& P, const DLayer& R, uint32_t a, uint32_t b, const RefineArgs& rp, EList LA, EList LB, int cap, int lane,
                            uint8_t& o_flag, double& o_area, double4& o_ev, uint32_t& o_evb) {
  return refine_pair_t<false, U_GLOBAL>(P, R, a, b, rp, LA, LB, cap, lane, o_flag, o_area, o_ev, o_evb);
}

// ---- the shared-memory bins' pair routine (filtered variants) -----------------------------------------------------------
// Per warp: the two edge lists, the boxes of B's edges on a 15-bit grid over the overlap box (qb), a queue of candidate edge
// pairs (q) and the cuts of both polygons' edges as linked lists (head of each edge, nodes val / nxt): a split point's
// parameter, or an edge of the other polygon that coincides with part of the edge. cand: bit i of A (then bit j of B) set
// when any edge of the other polygon comes within 2 tol of the edge.
// The routine is bound by instruction issue, dependent latency (16 warps per SM) and instruction fetch, so the work is laid out to keep
// lanes busy side by side and the code small: edge pairs whose boxes come within 2 tol are queued and classified 32 at a
// time, one per lane, from the four orientations of the pair, which decide the contact and every cut the two edges make in each
// other. The contribution passes are left with the coincident pairs, one per shared edge. The inside tests of a
// pass's segments are taken one at a time by the whole warp, and edges that follow one another with no edge of the
// other polygon within 2 tol share one test (edge_pass).
// Loops are kept rolled on purpose: the kernel runs nearly straight through its code, and above about 48 KB of it the
// warps wait for instructions (100k parcels, this kernel: 71 KB 5.66 ms, 54 KB 3.82 ms, 49 KB 2.86 ms, with the
// instruction-fetch stall at 8.6, 4.3 and 0.9 cycles an instruction).
// Cuts as linked lists instead of masks and a pool of split points: 500k-parcel relate self-join 21.2 -> 20.4 ms.
// 100k-parcel relate self-join, against lanes that each visited their own edge's candidates: this bin 3.45 -> 2.86 ms, the
// self bin 1.44 -> 0.76 ms; two 60k layers, area: 4.35 -> 3.16 ms (14.5 -> 20.5 lanes active per instruction).
constexpr int NIL = 0x7FFF, COVER = 0x8000;   // nxt: end of list; bit 15: the node names a coincident edge
template <class Q>
struct CutLists { uint2* qb; double* val; uint32_t* headA; uint32_t* headB; uint32_t* cand; uint16_t* nxt; Q* q; uint32_t* count; int cap; };
struct Nodes { int n; bool full; };   // nodes in use (a warp's own lists; a block counts in *count); full: some did not fit

// Classifies one candidate edge pair (i of A, j of B) per lane: real / any contact (seg_isect on the four orientations
// of the pair, behind the same box test), and for either edge what edge_visit finds for it: coincidence (a node that
// names the edge) or a split point. The two edges' conditions are the same but for their box tests, the order of a product and
// the end tolerances; r, tn and un change sign together when the edges swap roles, so un / r is B's parameter.
// S32: the contact's signs through the FP32 filter where the contact is all that is wanted; cuts need the orientations' values.
template <bool S32, bool SELF, bool CUTS, int SH, class Q, class EL>
__device__ __forceinline__ void classify_pairs(const EL& LA, const EL& LB, const PairGeo& G, const CutLists<Q>& cl, uint32_t e, bool act, int lane, Nodes& nd,
                                               bool& hit, bool& hit_any) {
  const int i = (int)(e >> SH), j = (int)(e & ((1u << SH) - 1u));
  bool sa = false, sb = false, va = false, vb = false;   // split point of A's / B's edge; coincident part of A's / B's edge
  double t = 0, u = 0;
  if (act) {
    const double px = LA.x0[i], py = LA.y0[i], qx = LA.x1[i], qy = LA.y1[i];
    const double ex0 = LB.x0[j], ey0 = LB.y0[j], ex1 = LB.x1[j], ey1 = LB.y1[j];
    const uint32_t fa = LA.fl[i], fb = LB.fl[j];
    const double c0 = orient(px, py, qx, qy, ex0, ey0), c1 = orient(px, py, qx, qy, ex1, ey1);
    const double g0 = orient(ex0, ey0, ex1, ey1, px, py), g1 = orient(ex0, ey0, ex1, ey1, qx, qy);
    const double ax0 = px < qx ? px : qx, ax1 = px < qx ? qx : px, ay0 = py < qy ? py : qy, ay1 = py < qy ? qy : py;
    const double bx0 = ex0 < ex1 ? ex0 : ex1, bx1 = ex0 < ex1 ? ex1 : ex0, by0 = ey0 < ey1 ? ey0 : ey1, by1 = ey0 < ey1 ? ey1 : ey0;
    const bool near = !(bx1 < ax0 || bx0 > ax1 || by1 < ay0 || by0 > ay1);
    if (S32 && !CUTS) {
      if (near && seg_isect32(px, py, qx, qy, ex0, ey0, ex1, ey1)) { hit_any = true; if (!((fa | fb) & 1u)) hit = true; }
    } else if (!SELF && near) {
      bool is = ((g0 > 0 && g1 < 0) || (g0 < 0 && g1 > 0)) && ((c0 > 0 && c1 < 0) || (c0 < 0 && c1 > 0));
      is = is || (g0 == 0 && px >= bx0 && px <= bx1 && py >= by0 && py <= by1) || (g1 == 0 && qx >= bx0 && qx <= bx1 && qy >= by0 && qy <= by1) ||
           (c0 == 0 && ex0 >= ax0 && ex0 <= ax1 && ey0 >= ay0 && ey0 <= ay1) || (c1 == 0 && ex1 >= ax0 && ex1 <= ax1 && ey1 >= ay0 && ey1 <= ay1);
      if (is) { hit_any = true; if (!((fa | fb) & 1u)) hit = true; }
    }
    if constexpr (CUTS) {
      const double tol = G.tol;
      bool ka = near, kb = near;   // the box tests of the two edges, padded by tol
      if (!near) {
        ka = !(bx1 < ax0 - tol || bx0 > ax1 + tol || by1 < ay0 - tol || by0 > ay1 + tol);
        kb = !(ax1 < bx0 - tol || ax0 > bx1 + tol || ay1 < by0 - tol || ay0 > by1 + tol);
      }
      const double dx = qx - px, dy = qy - py, fx = ex1 - ex0, fy = ey1 - ey0;
      const double len2 = dx * dx + dy * dy, flen2 = fx * fx + fy * fy, snap2 = G.snap * G.snap, eps2 = G.eps_par * G.eps_par;
      // an end's distance passes within the snap distance, a cut point's within tol as well
      const double ca = snap2 * len2, cat = fmax(ca, tol * tol * len2), cb = snap2 * flen2, cbt = fmax(cb, tol * tol * flen2);
      const bool onA = c0 * c0 <= ((fb & 2u) ? cat : ca) && c1 * c1 <= ((fb & 4u) ? cat : ca);
      const bool onB = g0 * g0 <= ((fa & 2u) ? cbt : cb) && g1 * g1 <= ((fa & 4u) ? cbt : cb);
      ka = ka && len2 != 0; kb = kb && flen2 != 0;
      va = ka && (onA || (onB && flen2 > 0));
      vb = kb && (onB || (onA && len2 > 0));
      const double r = dx * fy - dy * fx, wx = ex0 - px, wy = ey0 - py, tn = wx * fy - wy * fx, un = wx * dy - wy * dx;
      sa = ka && !va && r * r > eps2 * len2 * flen2 && (r > 0 ? (tn > 0 && tn < r) : (tn < 0 && tn > r));
      sb = kb && !vb && r * r > eps2 * flen2 * len2 && (r > 0 ? (un > 0 && un < r) : (un < 0 && un > r));
      if (sa || sb) {
#pragma unroll 1
        for (int z = 0; z < 2; z++) {   // one site for the division and the square root: t, then u; beyond an end: within its tolerance?
          const double q = (z ? un : tn) / r, f2 = z ? flen2 : len2;
          bool in = q >= 0 && q <= 1;
          if (!in) { const double d = tol / (f2 > 0 ? sqrt(f2) : (double)1); in = q >= -d && q <= 1 + d; }
          if (z) { u = q; sa = sa && in; } else { t = q; sb = sb && in; }
        }
      }
    }
  }
  if constexpr (!CUTS) return;
  const unsigned ma = __ballot_sync(0xffffffffu, sa || va), mB = __ballot_sync(0xffffffffu, sb || vb);
  if (ma | mB) {
    const unsigned lt = (1u << lane) - 1;
    const int total = __popc(ma) + __popc(mB);
    int at = nd.n;
    if (cl.count) {
      if (lane == 0) at = (int)atomicAdd(cl.count, (uint32_t)total);
      at = __shfl_sync(0xffffffffu, at, 0);
    } else {
      nd.n += total;
    }
    if (at + total > cl.cap) nd.full = true;
    else {
      if (sa || va) {
        const int k = at + __popc(ma & lt);
        cl.val[k] = va ? (double)j : t;
        cl.nxt[k] = (uint16_t)(atomicExch(&cl.headA[i], (uint32_t)k) | (va ? COVER : 0));
      }
      if (sb || vb) {
        const int k = at + __popc(ma) + __popc(mB & lt);
        cl.val[k] = vb ? (double)i : u;
        cl.nxt[k] = (uint16_t)(atomicExch(SELF ? &cl.headA[j] : &cl.headB[j], (uint32_t)k) | (vb ? COVER : 0));
      }
    }
  }
}

// the interval that edge k of the other polygon, coincident with part of edge e, covers of it (edge_visit's arithmetic)
template <class EL>
__device__ __forceinline__ void edge_cover(EdgeCuts& C, const EdgeRef& e, const EL& L, int k) {
  double tc = 0, te = 0;
#pragma unroll 1
  for (int z = 0; z < 2; z++) {   // one site for the division; exact twins, the shared edges of a tiling, need none
    const double n = ((z ? L.x1 : L.x0)[k] - e.px) * e.dx + ((z ? L.y1 : L.y0)[k] - e.py) * e.dy;
    tc = te;
    te = n == 0.0 ? 0.0 : (n == e.len2 ? 1.0 : n / e.len2);
  }
  const double lo = fmax((double)0, fmin(tc, te)), hi = fmin((double)1, fmax(tc, te));
  if (!(hi > lo)) return;
  if (lo > 0 && C.ns < MAXS) C.ts[C.ns++] = lo;
  if (hi < 1 && C.ns < MAXS) C.ts[C.ns++] = hi;
  if (C.no < MAXO) {
    C.ol0[C.no] = lo; C.ol1[C.no] = hi; C.oidx[C.no] = k;
    C.osame[C.no] = (e.dx * (L.x1[k] - L.x0[k]) + e.dy * (L.y1[k] - L.y0[k])) > 0;
    C.no++;
  }
}

// Candidate edge pairs (boxes within 2 tol of each other, or a little more on the grid) found and classified; CUTS: the cuts
// are wanted, else the contact alone (the search then ends at the first real one). SELF: only j > i is searched (an edge
// always coincides with itself); self: a geometry with itself searched in full, less each edge with itself. One warp takes the 32 A edges from ic0 on, then those from ic0 + step on, ...
template <bool S32, int MS, bool SELF, bool CUTS, int SH, class Q, class EL>
__device__ Nodes find_pairs(const EL& LA, int na, const EL& LB, int nb, const PairGeo& G, const CutLists<Q>& cl, int ic0, int step, int lane, bool& hit,
                            bool& hit_any, bool self = false) {
  Nodes nd{0, false};
  uint32_t any = 0;
  scan_edge_pairs<SELF, SH>(
      LA, na, LB, nb, G.ov, 2.0 * G.tol, 2.0 * G.tol, cl.qb, cl.q, ic0, step, lane,
      [&](int w, uint32_t bits) {
        if constexpr (!SELF && CUTS) {
          any |= bits;
          const uint32_t ob = __reduce_or_sync(0xffffffffu, bits);
          if (lane == 0 && ob) atomicOr(&cl.cand[MS / 32 + w], ob);
        }
      },
      [&](int ic) {
        if constexpr (!SELF && CUTS) {
          const unsigned c = __ballot_sync(0xffffffffu, any != 0);
          if (lane == 0) cl.cand[ic >> 5] = c;
          any = 0;
        }
      },
      [&](uint32_t e, bool act) {
        classify_pairs<S32, SELF, CUTS, SH>(LA, LB, G, cl, e, act && !(self && (e >> SH) == (e & ((1u << SH) - 1u))), lane, nd, hit, hit_any);
        return !CUTS && __any_sync(0xffffffffu, hit);
      });
  return nd;
}
// the grid boxes of B's edges and, where cuts are wanted, empty lists; t of nt: the calling thread among those that share them
template <int MS, bool SELF, bool CUTS, class Q, class EL>
__device__ __forceinline__ void begin_pairs(const EL& LB, int na, int nb, const PairGeo& G, const CutLists<Q>& cl, int t, int nt) {
  fill_boxes(LB, nb, qgrid(G.ov), cl.qb, t, nt);
  if constexpr (CUTS) {
#pragma unroll 1
    for (int i = t; i < na; i += nt) cl.headA[i] = NIL;
    if (!SELF) {
#pragma unroll 1
      for (int j = t; j < nb; j += nt) cl.headB[j] = NIL;
      if (t < 2 * (MS / 32)) cl.cand[t] = 0u;
    }
  }
}

// The cuts that all edges of the other polygon make, met in increasing order: the reference's own sweep, for an edge with more
// split points than are kept (which are kept depends on the order) and for pairs with more cuts than the lists hold.
template <class EL>
__device__ __forceinline__ void edge_sweep(EdgeCuts& C, const EdgeRef& e, const EL& L, int cnt, const PairGeo& G) {
  edge_cuts_begin(C);
#pragma unroll 1
  for (int k = 0; k < cnt; k++) edge_visit<true>(C, e, L, k, G);
  edge_cuts_sort(C);
}

// Lane's edge i with its cuts: split points in any order (they are sorted), coincident edges in increasing order.
// C.ns == MAXS: the split points reached the number that is kept (which are kept depends on the order they are met in).
// self: the lists are one geometry's, whose edges each coincide with themselves (no node says so). SWEEP: such an edge's
// cuts, and all edges' where the lists are not whole (sweep), are found by sweeping the other polygon's nother edges.
template <bool REL, bool SWEEP, class Q, class EL>
__device__ __forceinline__ void edge_cuts(EdgeRef& e, EdgeCuts& C, const EL& LS, int i, bool valid, const EL& LO, int nother, const CutLists<Q>& cl,
                                          const uint32_t* head, bool self, bool sweep, const PairGeo& G) {
  edge_cuts_begin(C);
  e.px = e.py = e.qx = e.qy = e.dx = e.dy = e.len2 = e.len = 0.0; e.fl = 0;
  if (!valid) return;
  e = edge_ref(LS, i, REL);
  if (!SWEEP || !sweep) {
    int nc = self ? 1 : 0, k = self ? i : 0x7FFFFFFF;   // coincident edges, the first of them
#pragma unroll 1
    for (uint32_t n = head[i]; n != NIL;) {
      const uint32_t w = cl.nxt[n];
      const double v = cl.val[n];
      if (w & COVER) { nc++; k = min(k, (int)v); }
      else if (C.ns < MAXS) C.ts[C.ns++] = v;
      n = w & NIL;
    }
#pragma unroll 1
    while (nc > 0) {
      edge_cover(C, e, LO, k);
      if (--nc == 0) break;
      int next = self && i > k ? i : 0x7FFFFFFF;
#pragma unroll 1
      for (uint32_t n = head[i]; n != NIL;) {
        const uint32_t w = cl.nxt[n];
        const int c = (w & COVER) ? (int)cl.val[n] : 0x7FFFFFFF;
        if (c > k) next = min(next, c);
        n = w & NIL;
      }
      k = next;
    }
  }
  if (SWEEP && (sweep || C.ns == MAXS)) edge_sweep(C, e, LO, nother, G);
  else edge_cuts_sort(C);
}

// The inside tests of 32 lanes' points (need, mx, my) against the polygon LO, one test at a time by the whole warp; lanes
// linked to their predecessor (bit l of link: points l - 1 and l lie on the same side of LO) take its answer.
template <bool S32, class EL>
__device__ __forceinline__ bool inside_lanes(bool need, double mx, double my, unsigned link, const EL& LO, int nother, bool inc, const PairGeo& G, int lane) {
  const unsigned needm = __ballot_sync(0xffffffffu, need), le = (2u << lane) - 1u;
  if (!needm) return false;
  // this lane's run of linked points: [start, end); its first that needs the test takes it for all
  const unsigned heads = ~link;
  const int start = 31 - __clz(heads & le);
  const unsigned after = heads & ~le;
  const unsigned run = (after ? (after & (0u - after)) - 1u : 0xffffffffu) & ~((1u << start) - 1u);
  const int tester = __ffs(needm & run) - 1;
  unsigned in = 0;
#pragma unroll 1
  for (unsigned m = __ballot_sync(0xffffffffu, need && tester == lane); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const double x = __shfl_sync(0xffffffffu, mx, src), y = __shfl_sync(0xffffffffu, my, src);
    if (inside_from_c_warp<S32>(LO, nother, G.cx, G.cy, inc, x, y, lane)) in |= 1u << src;
  }
  return need && ((in >> tester) & 1u);
}
// links of a chunk of edges, a bit each (see edge_pass): fr = edges without candidates
__device__ __forceinline__ unsigned edge_links(const EdgeRef& e, bool valid, unsigned fr, int lane) {
  const double prx = __shfl_up_sync(0xffffffffu, e.qx, 1), pry = __shfl_up_sync(0xffffffffu, e.qy, 1);
  return __ballot_sync(0xffffffffu, valid && lane > 0 && prx == e.px && pry == e.py) & fr & (fr << 1);
}

// One polygon's contribution pass: lane l owns edges l, l + 32, ... and adds its values in that order. Each lane collects its
// edge's split points and coincident intervals; the segments are then taken in step, the k-th of every edge at once,
// and their inside tests by the whole warp, one after the other. Returns false when an edge's split points reach the
// number that is kept (SWEEP: never; the edge is swept).
// Edges with no edge of the other polygon within 2 tol have one segment and no cut. Two of them that share an end
// point are connected by a path that keeps at least 2 tol away from the other polygon, so their midpoints lie on the same side of it: a run
// of such edges takes one test. (The crossing-parity test returns the true side for points this far from the boundary:
// its orientation signs can only be wrong for points within rounding, ~1e-7 of tol, of an edge's line.) tol below
// 1e-12 of the overlap box (a caller's own tolerances) turns the sharing off.
template <bool S32, bool SELF, bool AREA, bool REL, bool SWEEP, class Q, class EL>
__device__ __forceinline__ bool edge_pass(const EL& LS, int nself, const EL& LO, int nother, const CutLists<Q>& cl, const uint32_t* head, const uint32_t* cand,
                                          bool inc, const PairGeo& G, bool share, int lane, double& s2, double& lin, double& lon, uint32_t& bits,
                                          double* rec) {
#pragma unroll 1
  for (int ic = 0, c = 0; ic < nself; ic += 32, c++) {
    const int i = ic + lane;
    EdgeRef e;
    EdgeCuts C;
    edge_cuts<REL, SWEEP>(e, C, LS, i, i < nself, LO, nother, cl, head, SELF, false, G);
    if (!SWEEP && __any_sync(0xffffffffu, C.ns == MAXS)) return false;
    if (e.len2 == 0) C.ns = 0;
    const bool lens = REL && !(e.fl & 1u);
    unsigned link = 0;
    if constexpr (!SELF) link = edge_links(e, i < nself, share ? ~cand[c] : 0u, lane);
    double acc = 0.0;
#pragma unroll 1
    for (int k = 0; __any_sync(0xffffffffu, k + 1 < C.ns); k++) {
      Segment s;
      s.valid = s.need = false;
      s.mx = s.my = 0;
      if (k + 1 < C.ns) s = edge_segment<AREA>(C, e, LO, k, G, lens);
      const bool vin = inside_lanes<S32>(s.need, s.mx, s.my, k ? 0u : link, LO, nother, inc, G, lane);
      if (s.valid) edge_segment_add<AREA>(s, C, e, LO, G, lens, vin ? 1 : 0, acc, lin, lon, bits);
    }
    if (AREA) s2 += acc;
    if (AREA && rec) rec[c] = acc;
  }
  return true;
}

// What a pair's refinement has to give: the flag alone; the area; the DE-9IM evidence of intersecting pairs (flag 1; the others are
// not told apart); everything. Each is compiled by itself: what is not wanted costs neither instructions nor
// instruction-cache room.
enum Want { W_FLAG = 0, W_AREA = 1, W_REL = 2, W_ALL = 3 };

// One pair by one warp from shared memory. DONE, or, with nothing written, LONG: a local list exceeded cap or the cuts the
// room kept for them; SPLIT (not with SWEEP): an edge has more split points than are kept.
// SELF (> 0): the pair is a geometry with itself in one layer; the caller passes one list of up to SELF edges as both LA and LB. B's
// gather and B's contribution pass would repeat A's exactly (the same edges in the same frame, the same cuts in the same
// order, so the same values): A's pass runs once and each lane adds its recorded values a second time, in the same
// order, which is the sum the two passes make. Every edge meets itself, so the contact needs no test.
enum Done { LONG = 0, DONE = 1, SPLIT = 2 };
template <bool S32, int SELF, int W, bool SWEEP = false>
__device__ Done refine_pair_m(const DLayer& P, const DLayer& R, uint32_t a, uint32_t b, const RefineArgs& rp, EList8 LA, EList8 LB, int cap, int lane,
                              uint8_t& o_flag, double& o_area, double4& o_ev, uint32_t& o_evb, const CutLists<uint16_t>& cl, unsigned long long* ep) {
  constexpr int MS = SELF ? SELF : CAP_F;   // edges a side; B's bits of cand follow A's
  constexpr bool AREA = W == W_AREA || W == W_ALL, REL = W >= W_REL;
  Frame A, B;
  const PairGeo G = pair_geo(P, R, a, b, rp, A, B);
  int na = 0, nb = 0;
  bool inB_c = false, inA_c = false;
#pragma unroll 1
  for (int side = 0; side < (SELF ? 1 : 2); side++) {   // one inlined copy of the gather; it also takes the parity of the probe point c
    bool in = false;
    const int n = collect<true, true, S32>(side ? B : A, G.ov, side ? LB : LA, cap, lane, G.cx, G.cy, &in);
    if (side) { nb = n; inB_c = in; } else { na = n; inA_c = in; }
  }
  if constexpr (SELF > 0) { nb = na; inB_c = inA_c; }
  if (na > cap || nb > cap) return LONG;
  __syncwarp();
  bool hit = false, hit_any = false;
  Nodes nd{0, false};
  if constexpr (SELF == 0 || W != W_FLAG) {
    begin_pairs<MS, (SELF > 0), W != W_FLAG>(LB, na, nb, G, cl, lane, 32);
    __syncwarp();
    nd = find_pairs<S32, MS, (SELF > 0), W != W_FLAG, 8>(LA, na, LB, nb, G, cl, 0, 32, lane, hit, hit_any);
  }
  if constexpr (SELF > 0) {
#pragma unroll 1
    for (int i = lane; i < na; i += 32) { hit_any = true; if (!(LA.fl[i] & 1u)) hit = true; }
  }
  if (nd.full) return LONG;
  hit = __any_sync(0xffffffffu, hit);
  hit_any = __any_sync(0xffffffffu, hit_any || hit);
  const bool rtouch = hit;
  if (!hit) hit = contains_warp<S32>(A, B, LA, na, LB, nb, inA_c, inB_c, G.ov, G.cx, G.cy, lane, hit_any);
  PairSums S;
  uint32_t bits = rtouch ? REL_TOUCH : 0;
  const bool sums = W != W_FLAG && (hit || (W != W_REL && hit_any));
  if constexpr (W != W_FLAG)
    if (sums) {
      const bool share = G.tol >= 1e-12 * fmax(G.ov.x1 - G.ov.x0, G.ov.y1 - G.ov.y0);
      if constexpr (SELF > 0) {
        double rec[SELF / 32];
        if (!edge_pass<S32, true, AREA, REL, false>(LA, na, LB, nb, cl, cl.headA, cl.cand, inB_c, G, false, lane, S.s2, S.ai, S.ao, bits, rec)) return LONG;
#pragma unroll 1
        for (int c = 0; AREA && c * 32 < na; c++) S.s2 += rec[c];
        S.bi = S.ai; S.bo = S.ao;
      } else {
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {   // one inlined copy of the pass
          double lin = 0.0, lon = 0.0;   // this pass's lengths (each starts from 0, so the sums are the same)
          if (!edge_pass<S32, false, AREA, REL, SWEEP>(pass ? LB : LA, pass ? nb : na, pass ? LA : LB, pass ? na : nb, cl, pass ? cl.headB : cl.headA,
                                                       cl.cand + (pass ? MS / 32 : 0), pass ? inA_c : inB_c, G, share, lane, S.s2, lin, lon, bits, nullptr))
            return SPLIT;
          if (pass) { S.bi = lin; S.bo = lon; } else { S.ai = lin; S.ao = lon; }
        }
      }
    }
  pair_result<AREA, REL>(S, sums, hit, rtouch, bits, o_flag, o_area, o_ev, o_evb);
  if (lane == 0) *ep += (unsigned long long)na * (unsigned long long)nb;   // local edge pairs: the refinement's work unit
  return DONE;
}

// shared memory of one warp of the filtered bins: lists (one for self pairs), grid boxes, node values, heads, cand, node
// links, queue, flags
// split points and coincident edges of both polygons (about 45 for parcel neighbours); of a self pair, beside each edge itself
constexpr int NODES = 304, NODES_SELF = 160;
// (the flag alone: lists, grid boxes, queue, flags)
__host__ __device__ constexpr size_t warp_bytes(int cap, bool self, bool cuts = true) {
  const size_t sides = self ? 1 : 2;
  if (!cuts) return sides * cap * EDGE_BYTES_8 + (size_t)cap * 8 + QCAP * 2;
  const size_t nodes = self ? NODES_SELF : NODES;
  return sides * cap * EDGE_BYTES_8 + (size_t)cap * 8 + nodes * 8 + sides * cap * 4 + 2 * (cap / 32) * 4 + nodes * 2 + QCAP * 2;
}
static_assert(warp_bytes(128, false) % 16 == 0 && warp_bytes(256, true) % 16 == 0, "a warp's part starts on 16 bytes");
template <int MS, bool SELF, bool CUTS>
__device__ __forceinline__ void carve_warp(unsigned char* base, EList8& LA, EList8& LB, CutLists<uint16_t>& cl) {
  constexpr int nodes = SELF ? NODES_SELF : NODES;
  double* d = reinterpret_cast<double*>(base);
  auto doubles = [&](EList8& L) { L.x0 = d; L.y0 = d + MS; L.x1 = d + 2 * MS; L.y1 = d + 3 * MS; d += 4 * MS; };
  doubles(LA);
  if (!SELF) doubles(LB);
  cl.qb = reinterpret_cast<uint2*>(d);
  cl.val = d + MS;
  cl.headA = reinterpret_cast<uint32_t*>(cl.val + (CUTS ? nodes : 0));
  cl.headB = SELF ? cl.headA : cl.headA + MS;
  cl.cand = cl.headB + MS;
  cl.nxt = reinterpret_cast<uint16_t*>(cl.cand + 2 * (MS / 32));
  cl.q = CUTS ? cl.nxt + nodes : reinterpret_cast<uint16_t*>(cl.val);
  cl.count = nullptr;
  cl.cap = nodes;
  LA.fl = reinterpret_cast<uint8_t*>(cl.q + QCAP);
  if (SELF) LB = LA; else LB.fl = LA.fl + MS;
}
template <bool F, int W> struct Cfg;
template <int W> struct Cfg<false, W> { static constexpr int cap = CAP; static constexpr size_t smem = RB_SMEM, warp = 0; static constexpr int minb = 3; };
template <int W> struct Cfg<true, W> {   // the flag alone needs no room for cuts and fewer registers: 5 blocks per SM
  static constexpr int cap = CAP_F;
  static constexpr size_t warp = warp_bytes(CAP_F, false, W != W_FLAG), smem = RB_WARPS * warp;
  static constexpr int minb = W == W_FLAG ? 5 : 4;
};

constexpr int NSPLIT = 12;   // counter of k_refine_split's pairs, behind nheavy

// S32 (filtered only): the orientation signs of the gather's parity, of the inside tests and, for the flag alone, of the contact test
// through the certified FP32 filter
template <bool F, bool S32 = false, int W = W_ALL>
__global__ void __launch_bounds__(RB_WARPS * 32, Cfg<F, W>::minb) k_refine(DLayer P, DLayer R, const uint2* __restrict__ pairs, uint64_t np,
                                                                        RefineArgs rp, uint8_t* flag, double* area, double4* ev, uint32_t* evb,
                                                                        uint32_t* heavy, unsigned long long* nheavy, unsigned long long* next,
                                                                        unsigned long long* epairs, int run, int runs, int bin_cap,
                                                                        int skip_self) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_ep[RB_WARPS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (lane == 0) s_ep[wib] = 0;
  __syncwarp();
  EList LA, LB;
  EList8 MA, MB;
  CutLists<uint16_t> mbuf;
  if constexpr (F) {
    carve_warp<CAP_F, false, W != W_FLAG>(smem + (size_t)wib * Cfg<F, W>::warp, MA, MB, mbuf);
  } else {
    LA = carve(smem + (size_t)wib * 2 * LIST_BYTES, CAP);
    LB = carve(smem + (size_t)wib * 2 * LIST_BYTES + LIST_BYTES, CAP);
  }
  auto one = [&](uint64_t p) {
    const uint2 pr = pairs[p];
    if (skip_self && pr.x == pr.y) return;   // a geometry with itself: the self bin's
    uint8_t f; double ar; double4 e4; uint32_t b4;
    Done d;
    if constexpr (F) d = refine_pair_m<S32, 0, W>(P, R, pr.x, pr.y, rp, MA, MB, bin_cap, lane, f, ar, e4, b4, mbuf, &s_ep[wib]);
    else d = refine_pair_t<false, 1>(P, R, pr.x, pr.y, rp, LA, LB, bin_cap, lane, f, ar, e4, b4, nullptr, &s_ep[wib]) ? DONE : LONG;
    if (lane == 0) {
      if (d != DONE) {   // the list's front, or its back for k_refine_split
        heavy[d == LONG ? atomicAdd(nheavy, 1ull) : np - 1 - atomicAdd(nheavy + NSPLIT, 1ull)] = (uint32_t)p;
        flag[p] = 0;
      }
      else {
        flag[p] = f;
        if (area) area[p] = ar;
        if (ev) { ev[p] = e4; evb[p] = b4; }
      }
    }
    __syncwarp();
  };
  if constexpr (F) {
    // warps take runs of `run` consecutive pairs (shared probe geometry) from a counter, at most `runs` runs each:
    // the grid is sized to cover every pair that way, and bounded block lifetimes let the kernels of other
    // streams (higher-priority requests) take SMs as blocks retire
    for (int k = 0; k < runs; k++) {
      unsigned long long p0 = 0;
      if (lane == 0) p0 = atomicAdd(next, (unsigned long long)run);
      p0 = __shfl_sync(0xffffffffu, p0, 0);
      if (p0 >= np) break;
      const uint64_t p1 = p0 + run < np ? p0 + run : np;
      for (uint64_t p = p0; p < p1; p++) one(p);
    }
  } else {
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < np; p += nw) one(p);
  }
  __syncwarp();
  if (lane == 0 && s_ep[wib]) atomicAdd(epairs, s_ep[wib]);
}

// The pairs of the shared-memory bin with an edge of more split points than are kept (a straight edge across a stair-stepped or
// finely divided outline): the same routine, which sweeps such an edge. By itself, because the sweep's code in the bin cost every pair
// more than it saved these (400k-parcel relate self-join, refinement 14.7 -> 15.3-16.3 ms in six forms: instruction fetch). 20k strips
// across outlines of 96 edges, 24 cuts on an edge, area, whole call: 20.1 ms when the scratch bin took them, 4.3 ms by the block bin,
// 2.15 ms here. 20k strips across 600 edges with 150 cuts (the block bins sweep too): 118.9 -> 11.1 ms.
template <bool S32, int W>
__global__ void __launch_bounds__(RB_WARPS * 32, Cfg<true, W>::minb) k_refine_split(DLayer P, DLayer R, const uint2* __restrict__ pairs, uint64_t np, RefineArgs rp,
                                                                                   uint8_t* flag, double* area, double4* ev, uint32_t* evb,
                                                                                   const uint32_t* list, const unsigned long long* nlist,
                                                                                   unsigned long long* next, unsigned long long* epairs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_ep[RB_WARPS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (lane == 0) s_ep[wib] = 0;
  __syncwarp();
  EList8 LA, LB;
  CutLists<uint16_t> cl;
  carve_warp<CAP_F, false, W != W_FLAG>(smem + (size_t)wib * Cfg<true, W>::warp, LA, LB, cl);
  const uint64_t n = *nlist;   // written by k_refine, launched before this kernel
  for (;;) {
    unsigned long long h = 0;
    if (lane == 0) h = atomicAdd(next, 1ull);
    h = __shfl_sync(0xffffffffu, h, 0);
    if (h >= n) break;
    const uint32_t p = list[np - 1 - h];
    const uint2 pr = pairs[p];
    uint8_t f; double ar; double4 e4; uint32_t b4;
    refine_pair_m<S32, 0, W, true>(P, R, pr.x, pr.y, rp, LA, LB, CAP_F, lane, f, ar, e4, b4, cl, &s_ep[wib]);   // DONE: its lists fitted before
    if (lane == 0) {
      flag[p] = f;
      if (area) area[p] = ar;
      if (ev) { ev[p] = e4; evb[p] = b4; }
    }
    __syncwarp();
  }
  if (lane == 0 && s_ep[wib]) atomicAdd(epairs, s_ep[wib]);
}

// Self bin (filtered variants, a layer joined with itself): the pairs of a geometry with itself, 24 % of a parcel
// self-join's pairs and the costliest (every edge is local). One list of up to 256 edges per warp (the largest that the
// queue's bytes index and that keeps 4 blocks of 4 warps per SM), A's gather and contribution pass only (refine_pair_m SELF).
constexpr int CAP_SELF = 256;
constexpr size_t SELF_SMEM = RB_WARPS * warp_bytes(CAP_SELF, true);
constexpr int SELF_MINB = 4;   // blocks per SM: 4 x 53 KB of shared memory

// positions of the self pairs (a == b) among the candidate pairs, warp-aggregated (order free: outputs go by position)
__global__ void k_self_index(const uint2* __restrict__ pairs, uint64_t np, uint32_t* sidx, unsigned long long* nself) {
  const int lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < np; base += stride) {   // warp-uniform
    const uint64_t p = base + lane;
    bool is = false;
    if (p < np) { const uint2 pr = pairs[p]; is = pr.x == pr.y; }
    const unsigned m = __ballot_sync(0xffffffffu, is);
    unsigned long long at = 0;
    if (lane == 0 && m) at = atomicAdd(nself, (unsigned long long)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (is) sidx[at + __popc(m & ((1u << lane) - 1))] = (uint32_t)p;
  }
}

template <bool S32, int W>
__global__ void __launch_bounds__(RB_WARPS * 32, SELF_MINB) k_refine_self(DLayer P, const uint2* __restrict__ pairs, const uint32_t* __restrict__ sidx,
                                                                          const unsigned long long* nself, RefineArgs rp, uint8_t* flag, double* area,
                                                                          double4* ev, uint32_t* evb, uint32_t* heavy, unsigned long long* nheavy,
                                                                          unsigned long long* next, unsigned long long* epairs, int run, int runs,
                                                                          int self_cap) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_ep[RB_WARPS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  if (lane == 0) s_ep[wib] = 0;
  __syncwarp();
  EList8 L, L2;
  CutLists<uint16_t> mbuf;
  carve_warp<CAP_SELF, true, true>(smem + (size_t)wib * warp_bytes(CAP_SELF, true), L, L2, mbuf);
  const uint64_t n = *nself;   // written by k_self_index, launched before this kernel
  for (int k = 0; k < runs; k++) {
    unsigned long long h0 = 0;
    if (lane == 0) h0 = atomicAdd(next, (unsigned long long)run);
    h0 = __shfl_sync(0xffffffffu, h0, 0);
    if (h0 >= n) break;
    const uint64_t h1 = h0 + run < n ? h0 + run : n;
    for (uint64_t h = h0; h < h1; h++) {
      const uint32_t p = sidx[h];
      const uint2 pr = pairs[p];
      uint8_t f; double ar; double4 e4; uint32_t b4;
      const Done d = refine_pair_m<S32, CAP_SELF, W>(P, P, pr.x, pr.y, rp, L, L, self_cap, lane, f, ar, e4, b4, mbuf, &s_ep[wib]);
      if (lane == 0) {
        if (d != DONE) { heavy[atomicAdd(nheavy, 1ull)] = p; flag[p] = 0; }
        else {
          flag[p] = f;
          if (area) area[p] = ar;
          if (ev) { ev[p] = e4; evb[p] = b4; }
        }
      }
      __syncwarp();
    }
  }
  __syncwarp();
  if (lane == 0 && s_ep[wib]) atomicAdd(epairs, s_ep[wib]);
}

// Block bin (filtered variants): the pairs the shared-memory bins hand on, a block of 4 warps per pair, lists of up to 512
// edges a side in shared memory (54 KB a block, 4 blocks per SM). The routine is refine_pair_m's with the edges of the
// gather, the search and the passes dealt out to the warps in chunks of 32; the sums keep their order: a lane's running sums
// pass through shared memory from the warp of one chunk to that of the next. Larger pairs go on to a second form with 1024
// edges a side and 8 warps (108 KB, 2 blocks per SM), and from there to the scratch bin: a pair of 700 edges took 0.4 ms by
// itself in the scratch bin.
// Against the scratch bin's warp per pair with lists in global memory (10 % of the warps an SM holds, 37k instructions a
// pair), whole refinement: two 120k layers with areas (7k such pairs) 7.82 -> 6.47 ms, 20k queries relate (3.9k) 1.70 ->
// 1.32 ms, 100 queries (29: the latency of one pair) 0.27 -> 0.15 ms.
constexpr int CAP_BIG = 512, CAP_BIG2 = 1024;
constexpr int block_warps(int cap) { return cap / 128; }
constexpr size_t block_smem(size_t cap) {   // lists, grid boxes, 2 cap nodes, heads, cand, sums, queues
  return 2 * cap * EDGE_BYTES_8 + cap * 8 + 2 * cap * 8 + 2 * cap * 4 + 2 * (cap / 32) * 4 + 5 * 32 * 8 + (cap / 128) * QCAP * 4 + 2 * cap * 2;
}

// the edges of A meeting the box, by the whole block, compacted in ring order; inside: the parity of (mx, my). cnt: one
// word per warp and a spare set (the rounds alternate, so one barrier a round is enough)
template <bool S32, int NW>
__device__ int collect_block(const Frame& A, const Box& ov, const EList8& L, int cap, uint32_t* cnt, double mx, double my, bool& inside) {
  const DLayer& S = *A.L;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  bool par = false;
  int have = 0, flip = 0;
#pragma unroll 1
  for (uint32_t ra = A.r0; ra < A.r1; ra++) {
    const uint64_t s = S.rvo[ra];
    const uint32_t n = (uint32_t)(S.rvo[ra + 1] - s);
#pragma unroll 1
    for (uint32_t base = 0; base + 1 < n; base += NW * 32, flip ^= NW) {
      const uint32_t i = base + threadIdx.x;
      double2 p = make_double2(0, 0), q = p;
      if (i + 1 < n) { p = S.xy[s + i]; q = S.xy[s + i + 1]; }
      const GatherEdge e = gather_edge<true, true, S32>(A, ov, s, n, i, p, q, mx, my, par);
      const unsigned m = __ballot_sync(0xffffffffu, e.in);
      if (lane == 0) cnt[flip + wid] = __popc(m);
      __syncthreads();
      int pos = have + __popc(m & ((1u << lane) - 1));
      for (int w = 0; w < NW; w++) {
        const int c = cnt[flip + w];
        if (w < wid) pos += c;
        have += c;
      }
      if (e.in && pos < cap) { L.x0[pos] = e.x0; L.y0[pos] = e.y0; L.x1[pos] = e.x1; L.y1[pos] = e.y1; L.fl[pos] = e.fl; }
    }
  }
  inside = (__syncthreads_count(par) & 1) != 0;
  return have;
}

template <bool S32, int W, int CAP>
__global__ void __launch_bounds__(block_warps(CAP) * 32, 16 / block_warps(CAP)) k_refine_block(DLayer P, DLayer R, const uint2* __restrict__ pairs, const uint32_t* __restrict__ list,
                                                                   const unsigned long long* nlist, RefineArgs rp, uint8_t* flag, double* area, double4* ev,
                                                                   uint32_t* evb, uint32_t* heavy, unsigned long long* nheavy, unsigned long long* next,
                                                                   unsigned long long* epairs, int same_layer) {
  constexpr int NW = block_warps(CAP), NODES_BLOCK = 2 * CAP;
  constexpr bool AREA = W == W_AREA || W == W_ALL, REL = W >= W_REL;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ unsigned long long s_h;
  __shared__ uint32_t s_cnt[2 * NW], s_nodes, s_bits;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t n = *nlist;   // written by the bins launched before this kernel
  EList8 LA, LB;
  CutLists<uint32_t> cl;
  double* sums;   // s2, lin, lon of each lane (the pass that runs), then A's lin and lon
  {
    double* d = reinterpret_cast<double*>(smem);
    auto doubles = [&](EList8& L) { L.x0 = d; L.y0 = d + CAP; L.x1 = d + 2 * CAP; L.y1 = d + 3 * CAP; d += 4 * CAP; };
    doubles(LA);
    doubles(LB);
    cl.qb = reinterpret_cast<uint2*>(d);
    cl.val = d + CAP;
    sums = cl.val + NODES_BLOCK;
    cl.headA = reinterpret_cast<uint32_t*>(sums + 5 * 32);
    cl.headB = cl.headA + CAP;
    cl.cand = cl.headB + CAP;
    cl.q = cl.cand + 2 * (CAP / 32) + wid * QCAP;
    cl.nxt = reinterpret_cast<uint16_t*>(cl.cand + 2 * (CAP / 32) + NW * QCAP);
    cl.count = &s_nodes;
    cl.cap = NODES_BLOCK;
    LA.fl = reinterpret_cast<uint8_t*>(cl.nxt + NODES_BLOCK);
    LB.fl = LA.fl + CAP;
  }
  for (;;) {
    __syncthreads();   // the previous pair's shared memory is no longer read
    if (threadIdx.x == 0) { s_h = atomicAdd(next, 1ull); s_nodes = 0; s_bits = 0; }
    __syncthreads();
    if (s_h >= n) break;
    const uint32_t p = list[s_h];
    const uint2 pr = pairs[p];
    Frame A, B;
    const bool self = same_layer && pr.x == pr.y;
    const PairGeo G = pair_geo(P, R, pr.x, pr.y, rp, A, B);
    int na = 0, nb = 0;
    bool inA_c = false, inB_c = false;
#pragma unroll 1
    for (int side = 0; side < 2; side++) {
      bool in = false;
      const int c = collect_block<S32, NW>(side ? B : A, G.ov, side ? LB : LA, CAP, s_cnt, G.cx, G.cy, in);
      if (side) { nb = c; inB_c = in; } else { na = c; inA_c = in; }
    }
    const bool over = na > CAP || nb > CAP;   // the same in every thread, as sweep
    bool hit = false, hit_any = false, sweep = false;
    if (!over) {
      begin_pairs<CAP, false, W != W_FLAG>(LB, na, nb, G, cl, threadIdx.x, NW * 32);
      __syncthreads();
      const Nodes nd = find_pairs<S32, CAP, false, W != W_FLAG, 16>(LA, na, LB, nb, G, cl, wid * 32, NW * 32, lane, hit, hit_any, self);
      if (self)
        for (int i = threadIdx.x; i < na; i += NW * 32) { hit_any = true; if (!(LA.fl[i] & 1u)) hit = true; }
      hit = __syncthreads_or(hit);
      hit_any = __syncthreads_or(hit_any || hit);
      sweep = __syncthreads_or(nd.full);
    }
    const bool rtouch = hit;
    if (!over && !hit) {   // every warp for itself, the same answer
      hit = contains_warp<S32>(A, B, LA, na, LB, nb, inA_c, inB_c, G.ov, G.cx, G.cy, lane, hit_any);
    }
    const bool want = !over && W != W_FLAG && (hit || (W != W_REL && hit_any));
    PairSums S;
    uint32_t bits = rtouch ? REL_TOUCH : 0;
    if constexpr (W != W_FLAG)
      if (want) {
        const bool share = G.tol >= 1e-12 * fmax(G.ov.x1 - G.ov.x0, G.ov.y1 - G.ov.y0);
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {
          const EList8& LS = pass ? LB : LA;
          const EList8& LO = pass ? LA : LB;
          const int nself = pass ? nb : na, nother = pass ? na : nb;
          const uint32_t* head = pass ? cl.headB : cl.headA;
          const uint32_t* cand = cl.cand + (pass ? CAP / 32 : 0);
          const bool inc = pass ? inA_c : inB_c;
          if (wid == 0) {   // a lane's sums: s2 runs on, each pass's lengths start from 0
            if (pass) { sums[96 + lane] = sums[32 + lane]; sums[128 + lane] = sums[64 + lane]; } else sums[lane] = 0.0;
            sums[32 + lane] = 0.0; sums[64 + lane] = 0.0;
          }
          __syncthreads();
#pragma unroll 1
          for (int c0 = 0; c0 * 32 < nself; c0 += NW) {
            const int c = c0 + wid, i = c * 32 + lane;
            EdgeRef e;
            EdgeCuts C;
            edge_cuts<REL, true>(e, C, LS, i, i < nself, LO, nother, cl, head, self, sweep, G);
            if (e.len2 == 0) C.ns = 0;
            const bool lens = REL && !(e.fl & 1u);
            const unsigned link = edge_links(e, i < nself, share && c * 32 < nself ? ~cand[c] : 0u, lane);
            uint32_t vin = 0;   // bit k: segment k's midpoint is inside (fewer than MAXS segments)
#pragma unroll 1
            for (int k = 0; __any_sync(0xffffffffu, k + 1 < C.ns); k++) {
              bool need = false;
              double mx = 0, my = 0;
              if (k + 1 < C.ns) {
                const Segment s = edge_segment<AREA>(C, e, LO, k, G, lens);
                need = s.need; mx = s.mx; my = s.my;
              }
              if (inside_lanes<S32>(need, mx, my, k ? 0u : link, LO, nother, inc, G, lane)) vin |= 1u << k;
            }
#pragma unroll 1
            for (int w = 0; w < NW; w++) {   // the chunks' terms in their order
              if (w == wid && c * 32 < nself) {
                double acc = 0.0, lin = sums[32 + lane], lon = sums[64 + lane];
#pragma unroll 1
                for (int k = 0; k + 1 < C.ns; k++) {
                  const Segment s = edge_segment<AREA>(C, e, LO, k, G, lens);
                  if (s.valid) edge_segment_add<AREA>(s, C, e, LO, G, lens, (vin >> k) & 1u ? 1 : 0, acc, lin, lon, bits);
                }
                __syncwarp();
                if (i < nself) sums[lane] += acc;
                sums[32 + lane] = lin; sums[64 + lane] = lon;
              }
              __syncthreads();
            }
          }
        }
        if (REL) {
          const uint32_t b = __reduce_or_sync(0xffffffffu, bits);
          if (lane == 0) atomicOr(&s_bits, b);
          __syncthreads();
          bits = s_bits;
        }
        S.s2 = sums[lane];
        S.ai = sums[96 + lane]; S.ao = sums[128 + lane]; S.bi = sums[32 + lane]; S.bo = sums[64 + lane];
      }
    if (wid == 0) {
      if (over) {
        if (lane == 0) { heavy[atomicAdd(nheavy, 1ull)] = p; flag[p] = 0; }
      } else {
        uint8_t f; double ar; double4 e4; uint32_t b4;
        pair_result<AREA, REL>(S, want, hit, rtouch, bits, f, ar, e4, b4);
        if (lane == 0) {
          flag[p] = f;
          if (area) area[p] = ar;
          if (ev) { ev[p] = e4; evb[p] = b4; }
          atomicAdd(epairs, (unsigned long long)na * (unsigned long long)nb);
        }
      }
    }
  }
}

// oversized pairs: the same pair routine with per-warp edge lists in global scratch. The filtered variant also
// keeps its candidate list there (cph entries); a pair with more candidates runs the full sweeps instead.
template <bool F>
__host__ __device__ constexpr size_t scratch_per_warp(int cap, int cph) {
  return ((2 * (size_t)cap * EDGE_BYTES + (F ? (size_t)cph * 6 + 2 * ((size_t)cap + 1) * 4 + ((size_t)(2 * cap + 64) + NBK + 1) * 4 : 0)) + 15) &
         ~(size_t)15;
}
template <bool F>
__global__ void __launch_bounds__(128) k_refine_scratch(DLayer P, DLayer R, const uint2* __restrict__ pairs, const uint32_t* __restrict__ heavy,
                                                       const unsigned long long* nheavy, RefineArgs rp, uint8_t* flag, double* area, double4* ev, uint32_t* evb,
                                                       unsigned char* scratch, int cap, int cph, int* err, unsigned long long* epairs,
                                                       unsigned long long* next, int same_layer) {
  const int lane = threadIdx.x & 31;
  const uint64_t nh = *nheavy;   // written by the bins launched before this kernel
  if (nh == 0) return;
  unsigned long long ep = 0;
  const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned char* base = scratch + w * scratch_per_warp<F>(cap, cph);
  EList LA = carve(base, cap), LB = carve(base + (size_t)cap * EDGE_BYTES, cap);
  FlatBuf fb;
  if constexpr (F) {   // cp (u32), sa, sb (u32), pj (u16) after the lists
    fb.cp = reinterpret_cast<uint32_t*>(base + 2 * (size_t)cap * EDGE_BYTES);
    fb.sa = fb.cp + cph;
    fb.sb = fb.sa + (cap + 1);
    fb.bl = fb.sb + (cap + 1);
    fb.boff = fb.bl + (2 * cap + 64);
    fb.pj = reinterpret_cast<uint16_t*>(fb.boff + (NBK + 1));
    fb.cap = cph;
    fb.blcap = 2 * cap + 64;
    fb.rec = LB.x0;   // cap doubles, unused by a self pair's single list
  }
  (void)nw;
  for (;;) {   // one listed pair at a time from a counter: their costs vary widely
    unsigned long long h = 0;
    if (lane == 0) h = atomicAdd(next, 1ull);
    h = __shfl_sync(0xffffffffu, h, 0);
    if (h >= nh) break;
    const uint32_t p = heavy[h];
    const uint2 pr = pairs[p];
    uint8_t f; double ar; double4 e4; uint32_t b4;
    bool ok;
    if constexpr (F) {   // candidate entries pack both edge indices in 16 bits each
      if (same_layer && pr.x == pr.y)   // a geometry with itself: one list, one contribution pass (B's list records it)
        ok = cap <= 0xFFFF && refine_pair_t<F, U_GLOBAL, true, true, true>(P, P, pr.x, pr.y, rp, LA, LA, cap, lane, f, ar, e4, b4, &fb, &ep);
      else
        ok = cap <= 0xFFFF && refine_pair_t<F, U_GLOBAL, true, true>(P, R, pr.x, pr.y, rp, LA, LB, cap, lane, f, ar, e4, b4, &fb, &ep);
      if (!ok) ok = refine_pair_t<F, U_GLOBAL>(P, R, pr.x, pr.y, rp, LA, LB, cap, lane, f, ar, e4, b4, nullptr, &ep);
    } else {
      ok = refine_pair_t<F, U_GLOBAL>(P, R, pr.x, pr.y, rp, LA, LB, cap, lane, f, ar, e4, b4, nullptr, &ep);
    }
    if (lane == 0) {
      if (!ok) *err = 1;
      else {
        flag[p] = f;
        if (area) area[p] = ar;
        if (ev) { ev[p] = e4; evb[p] = b4; }
      }
    }
    __syncwarp();
  }
  if (lane == 0 && ep) atomicAdd(epairs, ep);
}

// whether a join of layers whose largest geometry has `most` edges has pairs for the scratch bin (and its launch shape any effect)
bool uses_scratch_bin(int mode, uint32_t most, int bin_cap) { return most > (uint32_t)(mode == GSJ_REFINE_PLAIN ? bin_cap : CAP_BIG2); }

// Scratch-bin layout for a layer pair: list capacity (rounded to 8 edges, which keeps every double array of the slab
// 8-byte aligned), candidate entries (indices stay below 2^16) and bytes per warp.
struct ScratchGeom { int cap, cph; size_t per; };
template <bool F>
static ScratchGeom scratch_geom(const gsj_layer* P, const gsj_layer* R) {
  ScratchGeom g;
  g.cap = (int)((std::max<uint32_t>(std::max(P->max_geom_edges, R->max_geom_edges), 1u) + 7u) & ~7u);
  g.cph = std::min(8 * g.cap, 1 << 16);
  g.per = scratch_per_warp<F>(g.cap, g.cph);
  return g;
}

// One refinement = one graph launch between the counters' reset and their copy to pinned host memory: the
// shared-memory bins (pairs whose local lists fit), then the bins for the pairs that these listed as oversized or rich in
// cuts; they read their counts on the device, so no host round trip separates the bins; then one stream sync.
// The executable graph is built once per context, variant and set of bins and re-parameterised per call.
template <bool F, bool S32 = false, int W = W_ALL>
static void refine_t(gsj_ctx* c, const gsj_layer* P, const gsj_layer* R, const uint2* pairs, uint64_t np, const RefineArgs& rp, uint8_t* flag,
                     double* area, double4* ev, uint32_t* evb) {
  cudaStream_t s = c->stream;
  constexpr int variant = F ? 1 + 4 * S32 + W : 0;   // plain, filtered x W, filtered FP32 x W
  const int bit = 1 << variant;
  if (!(c->refine_attr & bit)) {
    GSJ_CK(cudaFuncSetAttribute(k_refine<F, S32, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<F, W>::smem));
    if (F) {
      GSJ_CK(cudaFuncSetAttribute(k_refine_block<S32, W, CAP_BIG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)block_smem(CAP_BIG)));
      if constexpr (W != W_FLAG) GSJ_CK(cudaFuncSetAttribute(k_refine_split<S32, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<F, W>::smem));
      GSJ_CK(cudaFuncSetAttribute(k_refine_block<S32, W, CAP_BIG2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)block_smem(CAP_BIG2)));
    }
    c->refine_attr |= bit;
  }
  const RefineShape& sh = c->shape;
  unsigned long long* ctr = c->counters.as<unsigned long long>(16);
  int* err = reinterpret_cast<int*>(ctr + 1);
  uint32_t* heavy = c->heavy.as<uint32_t>(np);
  const int bin_cap = std::min(sh.bin_cap, Cfg<F, W>::cap), run = sh.run, runs = sh.runs;
  int blocks;
  if constexpr (F) {
    // enough warps to cover every pair with `runs` fetches each, spread over all SMs; more than one wave of blocks
    // is rounded up to whole waves, so the last wave's blocks share the remaining pairs (the counter hands them out)
    // instead of leaving part of the GPU idle while a partial wave runs
    const uint64_t per_block = (uint64_t)RB_WARPS * runs * run, wave = (uint64_t)c->sm_count * Cfg<F, W>::minb;
    uint64_t cover = (np + per_block - 1) / per_block;
    if (cover > wave) cover = (cover + wave - 1) / wave * wave;
    const uint64_t spread = std::min<uint64_t>((np + (uint64_t)RB_WARPS * run - 1) / ((uint64_t)RB_WARPS * run), wave);
    blocks = (int)std::min<uint64_t>(std::max<uint64_t>(cover, spread), 1u << 30);
  } else {
    blocks = (int)std::min<uint64_t>((np + RB_WARPS - 1) / RB_WARPS, (uint64_t)c->sm_count * 8);
  }
  // The filtered bins of a warp per pair hand pairs with more local edges a side than they hold, or more cuts than they have room for, to the
  // block bin, and that bin pairs with more local edges to the next: the bins that no geometry of the layers can need are not
  // launched (stage: 0 - 2, how many behind the first block bin; plain: behind the shared-memory bin).
  const uint32_t most = std::max(P->max_geom_edges, R->max_geom_edges);
  const bool two = F && most > (uint32_t)CAP_BIG, scr = uses_scratch_bin(F ? GSJ_REFINE_FILTERED : GSJ_REFINE_PLAIN, most, bin_cap), spl = F && W != W_FLAG;
  const int stage = (two ? 1 : 0) + (scr ? 1 : 0);
  uint32_t* heavy2 = F ? c->heavy2.as<uint32_t>(np) : heavy;   // a pair leaves a bin's list before the next bin runs: the third list is the first's memory
  const ScratchGeom sg = scratch_geom<F>(P, R);
  int sblocks = 0;
  unsigned char* sbuf = nullptr;
  if (scr) {   // warps: the shape's share of every SM, at most one per pair and at most 1 GiB of lists
    uint64_t nwarps = std::min<uint64_t>((uint64_t)c->sm_count * sh.scratch_wpsm, std::max<uint64_t>(1, (1ull << 30) / sg.per));
    nwarps = std::min<uint64_t>(nwarps, np);
    nwarps = (nwarps + 3) / 4 * 4;
    sblocks = (int)(nwarps / 4);
    sbuf = c->scratch.as<unsigned char>(sg.per * nwarps);
  }
  // self bin: a layer joined with itself (filtered variants); its pairs of a geometry with itself go to
  // k_refine_self, the others stay in the shared-memory bin, and the two run side by side
  const bool self = F && P == R;
  int iblocks = 1, fblocks = 1;
  uint32_t* sidx = nullptr;
  const int self_cap = std::min(2 * sh.bin_cap, CAP_SELF);   // twice the shape's shared-memory bin threshold: one list instead of two
  if (self) {
    const int sbit = 1 << (16 + variant);
    if (!(c->refine_attr & sbit)) {
      GSJ_CK(cudaFuncSetAttribute(k_refine_self<S32, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SELF_SMEM));
      c->refine_attr |= sbit;
    }
    sidx = c->selfidx.as<uint32_t>(np);
    iblocks = (int)std::min<uint64_t>((np + 255) / 256, (uint64_t)c->sm_count * 8);
    // at most one self pair per probe geometry: cover that many with `runs` fetches per warp, whole waves
    const uint64_t ub = std::min<uint64_t>(np, P->d.n), per_block = (uint64_t)RB_WARPS * runs * run, wave = (uint64_t)c->sm_count * SELF_MINB;
    uint64_t cover = (ub + per_block - 1) / per_block;
    if (cover > wave) cover = (cover + wave - 1) / wave * wave;
    const uint64_t spread = std::min<uint64_t>((ub + (uint64_t)RB_WARPS * run - 1) / ((uint64_t)RB_WARPS * run), wave);
    fblocks = (int)std::min<uint64_t>(std::max<uint64_t>(cover, spread), 1u << 30);
  }
  unsigned long long* h = c->h_refine.as<unsigned long long>(4);
  // counters: [0] oversized pairs, [1] error word, [2] pair counter, [3] local edge pairs, [4] scratch pair counter,
  // [5] self pairs, [6] self pair counter, [7] the block bin's oversized pairs, [8] block pair counter,
  // [REFINE_ROWS] the caller's, set to 0 here, [10], [11] as [7], [8] of the second block bin, [NSPLIT] pairs with an edge of
  // many split points, [NSPLIT + 1] counter of these
  auto a_main = kernel_args(k_refine<F, S32, W>, P->d, R->d, pairs, np, rp, flag, area, ev, evb, heavy, ctr, ctr + 2, ctr + 3, run, runs, bin_cap,
                            self ? 1 : 0);
  auto a_big = kernel_args(k_refine_block<S32, W, CAP_BIG>, P->d, R->d, pairs, heavy, ctr, rp, flag, area, ev, evb, heavy2, ctr + 7, ctr + 8, ctr + 3, P == R);
  auto a_big2 = kernel_args(k_refine_block<S32, W, CAP_BIG2>, P->d, R->d, pairs, heavy2, ctr + 7, rp, flag, area, ev, evb, heavy, ctr + 10, ctr + 11, ctr + 3,
                            P == R);
  auto a_scr = kernel_args(k_refine_scratch<F>, P->d, R->d, pairs, heavy, F ? ctr + 10 : ctr, rp, flag, area, ev, evb, sbuf, sg.cap, sg.cph, err, ctr + 3, ctr + 4,
                           P == R ? 1 : 0);
  auto a_idx = kernel_args(k_self_index, pairs, np, sidx, ctr + 5);
  auto a_self = kernel_args(k_refine_self<S32, W>, P->d, pairs, sidx, ctr + 5, rp, flag, area, ev, evb, heavy, ctr, ctr + 6, ctr + 3, run, runs, self_cap);
  constexpr int WS = W == W_FLAG ? W_AREA : W;   // the flag alone has no cuts: not launched
  auto a_split = kernel_args(k_refine_split<S32, WS>, P->d, R->d, pairs, np, rp, flag, area, ev, evb, heavy, ctr + NSPLIT, ctr + NSPLIT + 1, ctr + 3);
  cudaKernelNodeParams km{}, ks{}, ki{}, kf{}, kb{}, kb2{}, kp{};
  kb.func = (void*)k_refine_block<S32, W, CAP_BIG>;
  kb.gridDim = dim3((unsigned)std::min<uint64_t>(np, (uint64_t)c->sm_count * 4));
  kb.blockDim = dim3(block_warps(CAP_BIG) * 32);
  kb.sharedMemBytes = (unsigned)block_smem(CAP_BIG);
  kb.kernelParams = a_big.ptr;
  kb2 = kb;
  kb2.func = (void*)k_refine_block<S32, W, CAP_BIG2>;
  kb2.gridDim = dim3((unsigned)std::min<uint64_t>(np, (uint64_t)c->sm_count * 2));
  kb2.blockDim = dim3(block_warps(CAP_BIG2) * 32);
  kb2.sharedMemBytes = (unsigned)block_smem(CAP_BIG2);
  kb2.kernelParams = a_big2.ptr;
  km.func = (void*)k_refine<F, S32, W>;
  km.gridDim = dim3(blocks);
  km.blockDim = dim3(RB_WARPS * 32);
  km.sharedMemBytes = (unsigned)Cfg<F, W>::smem;
  km.kernelParams = a_main.ptr;
  kp = km;
  kp.func = (void*)k_refine_split<S32, WS>;
  kp.gridDim = dim3((unsigned)std::min<uint64_t>((np + RB_WARPS - 1) / RB_WARPS, (uint64_t)c->sm_count * Cfg<F, W>::minb));
  kp.kernelParams = a_split.ptr;
  ks.func = (void*)k_refine_scratch<F>;
  ks.gridDim = dim3(std::max(sblocks, 1));
  ks.blockDim = dim3(128);
  ks.kernelParams = a_scr.ptr;
  ki.func = (void*)k_self_index;
  ki.gridDim = dim3(iblocks);
  ki.blockDim = dim3(256);
  ki.kernelParams = a_idx.ptr;
  kf.func = (void*)k_refine_self<S32, W>;
  kf.gridDim = dim3(fblocks);
  kf.blockDim = dim3(RB_WARPS * 32);
  kf.sharedMemBytes = (unsigned)SELF_SMEM;
  kf.kernelParams = a_self.ptr;
  RefineGraph& g = c->rgraph[variant * 6 + stage * 2 + (self ? 1 : 0)];
  if (!g.exec) {   // the graph is kept with its executable: the node handles used for the updates belong to it
    if (!g.graph) {
      GSJ_CK(cudaGraphCreate(&g.graph, 0));
      // shared-memory bin || (self index -> self bin), then the block bins after both, then the scratch bin; beside these the pairs
      // with an edge of many split points
      GSJ_CK(cudaGraphAddKernelNode(&g.n_main, g.graph, nullptr, 0, &km));
      std::vector<cudaGraphNode_t> before{g.n_main};
      if (self) {
        GSJ_CK(cudaGraphAddKernelNode(&g.n_idx, g.graph, nullptr, 0, &ki));
        GSJ_CK(cudaGraphAddKernelNode(&g.n_self, g.graph, &g.n_idx, 1, &kf));
        before.push_back(g.n_self);
      }
      if (spl) GSJ_CK(cudaGraphAddKernelNode(&g.n_split, g.graph, &g.n_main, 1, &kp));
      if (F) {
        GSJ_CK(cudaGraphAddKernelNode(&g.n_big, g.graph, before.data(), before.size(), &kb));
        before.assign(1, g.n_big);
      }
      if (two) {
        GSJ_CK(cudaGraphAddKernelNode(&g.n_big2, g.graph, before.data(), 1, &kb2));
        before.assign(1, g.n_big2);
      }
      if (scr) GSJ_CK(cudaGraphAddKernelNode(&g.n_scr, g.graph, before.data(), before.size(), &ks));
    }
    GSJ_CK(cudaGraphInstantiate(&g.exec, g.graph, 0));
  } else {
    GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_main, &km));
    if (self) {
      GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_idx, &ki));
      GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_self, &kf));
    }
    if (spl) GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_split, &kp));
    if (F) GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_big, &kb));
    if (two) GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_big2, &kb2));
    if (scr) GSJ_CK(cudaGraphExecKernelNodeSetParams(g.exec, g.n_scr, &ks));
  }
  GSJ_CK(cudaMemsetAsync(ctr, 0, 14 * sizeof(unsigned long long), s));
  GSJ_CK(cudaGraphLaunch(g.exec, s));
  c->launches += 1 + (F ? 1 : 0) + (spl ? 1 : 0) + (two ? 1 : 0) + (scr ? 1 : 0) + (self ? 2 : 0);
  GSJ_CK(cudaMemcpyAsync(h, ctr, 32, cudaMemcpyDeviceToHost, s));
  c->refine_pending = true;
}

void refine_enqueue(gsj_ctx* c, const gsj_layer* P, const gsj_layer* R, const uint2* pairs, uint64_t np, const RefineArgs& rp, int mode,
                    uint8_t* flag, double* area, double4* ev, uint32_t* evb, bool hits_only) {
  if (!np) return;
  const int w = !rp.want_relate ? (rp.want_area ? W_AREA : W_FLAG) : (hits_only && !area ? W_REL : W_ALL);
  auto go = [&](auto s32) {
    constexpr bool S32 = decltype(s32)::value;
    if (w == W_FLAG) refine_t<true, S32, W_FLAG>(c, P, R, pairs, np, rp, flag, area, ev, evb);
    else if (w == W_AREA) refine_t<true, S32, W_AREA>(c, P, R, pairs, np, rp, flag, area, ev, evb);
    else if (w == W_REL) refine_t<true, S32, W_REL>(c, P, R, pairs, np, rp, flag, area, ev, evb);
    else refine_t<true, S32, W_ALL>(c, P, R, pairs, np, rp, flag, area, ev, evb);
  };
  if (mode == GSJ_REFINE_FILTERED_FP32) go(std::true_type{});
  else if (mode == GSJ_REFINE_FILTERED) go(std::false_type{});
  else refine_t<false>(c, P, R, pairs, np, rp, flag, area, ev, evb);
}

uint64_t refine_result(gsj_ctx* c) {
  if (!c->refine_pending) return 0;
  c->refine_pending = false;
  const unsigned long long* h = c->h_refine.as<unsigned long long>(4);
  if (reinterpret_cast<const int*>(h + 1)[0]) throw Error(GSJ_ERR_CUDA, "oversized pair exceeded the scratch edge capacity");
  c->edge_pairs += h[3];
  return h[0];
}

uint64_t refine(gsj_ctx* c, const gsj_layer* P, const gsj_layer* R, const uint2* pairs, uint64_t np, const RefineArgs& rp, int mode,
                uint8_t* flag, double* area, double4* ev, uint32_t* evb) {
  refine_enqueue(c, P, R, pairs, np, rp, mode, flag, area, ev, evb);
  GSJ_CK(cudaStreamSynchronize(c->stream));
  return refine_result(c);
}

}  // namespace gsj
