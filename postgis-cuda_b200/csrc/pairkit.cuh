// Warp-level building blocks shared by the pair kernels (refinement, distance, erosion): local edge lists,
// crossing parity, containment probes. Restating engine/engine.cuh:322-412 of landstats-us/postgis-cuda.
#pragma once
#include "geom.cuh"

namespace gsj {

__device__ __forceinline__ EList carve(unsigned char* base, int cap) {
  EList L;
  L.x0 = reinterpret_cast<double*>(base);
  L.y0 = L.x0 + cap; L.x1 = L.y0 + cap; L.y1 = L.x1 + cap;
  L.fl = reinterpret_cast<uint32_t*>(L.y1 + cap);
  return L;
}
// edge (x0, y0)-(x1, y1) entirely outside box [bx0, bx1] x [by0, by1], by comparisons only
__device__ __forceinline__ bool out_cmp(double x0, double y0, double x1, double y1, double bx0, double by0, double bx1, double by1) {
  return (x0 < bx0 && x1 < bx0) || (x0 > bx1 && x1 > bx1) || (y0 < by0 && y1 < by0) || (y0 > by1 && y1 > by1);
}
__device__ __forceinline__ bool edge_outside(double px, double py, double qx, double qy, const Box& o) {
  return fmax(px, qx) < o.x0 || fmin(px, qx) > o.x1 || fmax(py, qy) < o.y0 || fmin(py, qy) > o.y1;
}

// Whether the horizontal segment (ox, my) -> (mx, my) crosses the edge (x0, y0)-(x1, y1), which reaches the level my:
// so != sc && su != sv of the four orientations (engine.cuh:382-397), where ox lies left of both end points by at least about
// 1 (of the frame's unit). The side of (ox, my) is then the edge's direction in y, or in x for a level edge (the
// determinant is at least |y1 - y0| beside terms of a few hundred times that, so its rounding cannot turn it), and the
// orientations of the end points against the level segment are the signs of the plain products (their other term is 0).
template <bool S32 = false>
__device__ __forceinline__ bool ray_crosses(double x0, double y0, double x1, double y1, double ox, double mx, double my) {
  const bool so = y0 != y1 ? y1 > y0 : x1 > x0, sc = S32 ? left_of32(x0, y0, x1, y1, mx, my) : left_of(x0, y0, x1, y1, mx, my);
  const double a = mx - ox;
  return so != sc && (a * (y0 - my) > 0) != (a * (y1 - my) > 0);
}

// Edge i (p, q: its stored ends) of a ring of n vertices (the first is vertex s of the layer) in a pair frame: its ends and cut flags, whether it
// meets the overlap box, and its crossing of the level ray to (mx, my) into par (PIP).
struct GatherEdge { double x0, y0, x1, y1; uint32_t fl; bool in; };
template <bool F, bool PIP, bool S32>
__device__ __forceinline__ GatherEdge gather_edge(const Frame& A, const Box& ov, uint64_t s, uint32_t n, uint32_t i, double2 p, double2 q, double mx, double my,
                                                  bool& par) {
  const DLayer& S = *A.L;
  GatherEdge e{0, 0, 0, 0, 0u, false};
  if (i + 1 >= n) return e;
  e.x0 = A.shx + p.x; e.y0 = A.shy + p.y; e.x1 = A.shx + q.x; e.y1 = A.shy + q.y;
  if (S.synb) {
    e.fl = (uint32_t)S.syn(s + i) | (S.syn(s + (i > 0 ? i - 1 : n - 2)) ? 2u : 0u) | (S.syn(s + (i + 2 < n ? i + 1 : 0)) ? 4u : 0u);
  }
  e.in = F ? !out_cmp(e.x0, e.y0, e.x1, e.y1, ov.x0, ov.y0, ov.x1, ov.y1) : !edge_outside(e.x0, e.y0, e.x1, e.y1, ov);
  if (PIP && !((e.y0 > my) == (e.y1 > my) && e.y0 != my && e.y1 != my)) {
    if (ray_crosses<S32>(e.x0, e.y0, e.x1, e.y1, A.shx - (double)1, mx, my)) par = !par;
  }
  return e;
}

// all edges of geometry A meeting the overlap box, compacted in ring order with a warp ballot (engine.cuh:358-377).
// PIP: the same pass also takes the crossing parity of the segment (A's bbox left edge - 1, my) -> (mx, my) over
// every edge of A, as pip_full_warp does (an XOR over the edges, so the order is free), into *inside.
template <bool F, bool PIP = false, bool S32 = false, class EL>
static __device__ int collect(const Frame& A, const Box& ov, EL L, int cap, int lane, double mx = 0, double my = 0, bool* inside = nullptr) {
  const DLayer& S = *A.L;
  const unsigned lt = (1u << lane) - 1;
  bool par = false;
  int cnt = 0;
  // the next 32 vertices are on their way while these are tested (500k-parcel relate self-join 19.15 -> 18.6 ms, 150k-parcel
  // dwithin 2.53 -> 2.40 ms)
  const uint64_t none = 0;
  uint64_t s = A.r0 < A.r1 ? S.rvo[A.r0] : none, e1 = A.r0 < A.r1 ? S.rvo[A.r0 + 1] : none;
#pragma unroll 1
  for (uint32_t ra = A.r0; ra < A.r1; ra++) {
    const uint32_t n = (uint32_t)(e1 - s);   // a ring's vertices, indexed by 32 bits
    const uint64_t e2 = ra + 1 < A.r1 ? S.rvo[ra + 2] : none;
    const double2* v = S.xy + s;
    double2 p = make_double2(0, 0), q = p;
    if (lane + 1 < n) { p = v[lane]; q = v[lane + 1]; }
#pragma unroll 1
    for (uint32_t base = 0; base + 1 < n; base += 32) {
      double2 pn = make_double2(0, 0), qn = pn;
      const uint32_t in = base + 32 + lane;
      if (in + 1 < n) { pn = v[in]; qn = v[in + 1]; }
      const GatherEdge e = gather_edge<F, PIP, S32>(A, ov, s, n, base + lane, p, q, mx, my, par);
      p = pn; q = qn;
      const unsigned m = __ballot_sync(0xffffffffu, e.in);
      const int pos = cnt + __popc(m & lt);
      if (e.in && pos < cap) {
        L.x0[pos] = e.x0; L.y0[pos] = e.y0; L.x1[pos] = e.x1; L.y1[pos] = e.y1; L.fl[pos] = e.fl;
      }
      cnt += __popc(m);
    }
    s = e1; e1 = e2;
  }
  if (PIP) *inside = (__popc(__ballot_sync(0xffffffffu, par)) & 1) != 0;
  return cnt;
}

// crossing parity of segment (B's bbox left edge - 1, my) -> (mx, my) over all of B's edges (engine.cuh:382-397)
static __device__ bool pip_full_warp(const Frame& B, double mx, double my, int lane) {
  const DLayer& S = *B.L;
  const double ox = B.shx - (double)1;
  bool par = false;
#pragma unroll 1
  for (uint32_t r = B.r0; r < B.r1; r++) {
    const uint64_t s = S.rvo[r], e = S.rvo[r + 1];
#pragma unroll 1
    for (uint64_t j = s + 1 + lane; j < e; j += 32) {
      double x0, y0, x1, y1; B.v(j - 1, x0, y0); B.v(j, x1, y1);
      if (!((y0 > my) == (y1 > my) && y0 != my && y1 != my) && ray_crosses(x0, y0, x1, y1, ox, mx, my)) par = !par;
    }
  }
  return (__popc(__ballot_sync(0xffffffffu, par)) & 1) != 0;
}

// inside(x) = inside(c) xor crossings of c -> x with the local edges (engine.cuh:400-412)
// U: edges a step (lists in global memory: their loads overlap)
template <bool F, int U = 1, class EL>
__device__ __forceinline__ bool inside_from_c(const EL& L, int cnt, double cx, double cy, bool in_c, double x, double y) {
  bool in = in_c;
  const double sx0 = fmin(cx, x), sx1 = fmax(cx, x), sy0 = fmin(cy, y), sy1 = fmax(cy, y);
  auto step = [&](int k) {
    const double ex0 = L.x0[k], ey0 = L.y0[k], ex1 = L.x1[k], ey1 = L.y1[k];
    if (F ? out_cmp(ex0, ey0, ex1, ey1, sx0, sy0, sx1, sy1)
          : (fmax(ex0, ex1) < sx0 || fmin(ex0, ex1) > sx1 || fmax(ey0, ey1) < sy0 || fmin(ey0, ey1) > sy1)) return false;
    bool sc = left_of(ex0, ey0, ex1, ey1, cx, cy), sx = left_of(ex0, ey0, ex1, ey1, x, y);
    if (sc == sx) return false;
    bool su = orient(cx, cy, x, y, ex0, ey0) > 0, sv = orient(cx, cy, x, y, ex1, ey1) > 0;
    if (su != sv) in = !in;
    return false;
  };
#pragma unroll U
  for (int k = 0; k < cnt; k++) step(k);
  return in;
}

// The same parity for one query point shared by the whole warp: lanes split the edges, a ballot counts crossings
// (the parity does not depend on the order of the edges). S32: the four orientation signs through the certified FP32 filter (the same
// booleans).
template <bool S32 = false, class EL>
static __device__ bool inside_from_c_warp(const EL& L, int cnt, double cx, double cy, bool in_c, double x, double y, int lane) {
  const double sx0 = fmin(cx, x), sx1 = fmax(cx, x), sy0 = fmin(cy, y), sy1 = fmax(cy, y);
  bool par = false;
#pragma unroll 1
  for (int k = lane; k < cnt; k += 32) {
    const double ex0 = L.x0[k], ey0 = L.y0[k], ex1 = L.x1[k], ey1 = L.y1[k];
    if (out_cmp(ex0, ey0, ex1, ey1, sx0, sy0, sx1, sy1)) continue;
    const bool sc = S32 ? left_of32(ex0, ey0, ex1, ey1, cx, cy) : left_of(ex0, ey0, ex1, ey1, cx, cy);
    const bool sx = S32 ? left_of32(ex0, ey0, ex1, ey1, x, y) : left_of(ex0, ey0, ex1, ey1, x, y);
    if (sc == sx) continue;
    const bool su = (S32 ? orient_sign32(cx, cy, x, y, ex0, ey0) : orient(cx, cy, x, y, ex0, ey0)) > 0;
    const bool sv = (S32 ? orient_sign32(cx, cy, x, y, ex1, ey1) : orient(cx, cy, x, y, ex1, ey1)) > 0;
    if (su != sv) par = !par;
  }
  const bool odd = (__popc(__ballot_sync(0xffffffffu, par)) & 1) != 0;
  return in_c != odd;
}

__device__ __forceinline__ bool probe_vertex(const Frame& A, uint32_t r, double& x, double& y) {   // engine.cuh:322-327
  const DLayer& S = *A.L;
  uint64_t v = S.rvo[r], e = S.rvo[r + 1];
  if (S.synb) { while (v + 1 < e && S.syn(v)) v++; if (v + 1 >= e) return false; }
  A.v(v, x, y);
  return true;
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// the box of an edge on the 15-bit grid, packed so that one subtraction per axis tests both ends: bit 31 of (B - A) is
// B's upper end >= A's lower end, bit 15 A's upper end >= B's lower end (fields of 16 bits, no borrow between them).
// Every step is monotone in the coordinate, so boxes that meet are never told apart; coordinates outside the overlap
// box clamp to its sides.
struct QGrid { double x0, y0; float sx, sy; };
struct QBox { int x0, y0, x1, y1; };
__device__ __forceinline__ QGrid qgrid(const Box& ov) {
  QGrid g{ov.x0, ov.y0, 0.f, 0.f};
  const float w = (float)(ov.x1 - ov.x0), h = (float)(ov.y1 - ov.y0);
  if (w > 1e-30f) g.sx = 1.f / w;
  if (h > 1e-30f) g.sy = 1.f / h;
  return g;
}
__device__ __forceinline__ int qcell(double v, double o, float s) { return __float2int_rd(__saturatef((float)(v - o) * s) * 32767.f); }
template <class EL>
__device__ __forceinline__ QBox qbox(const QGrid& g, const EL& L, int i) {
  const int px = qcell(L.x0[i], g.x0, g.sx), py = qcell(L.y0[i], g.y0, g.sy), qx = qcell(L.x1[i], g.x0, g.sx), qy = qcell(L.y1[i], g.y0, g.sy);
  return QBox{min(px, qx), min(py, qy), max(px, qx), max(py, qy)};
}

// the boxes of a list's edges as B boxes, guard bits set; t of nt: the calling thread among those that fill them
template <class EL>
__device__ __forceinline__ void fill_boxes(const EL& L, int n, const QGrid& g, uint2* qb, int t, int nt) {
#pragma unroll 1
  for (int j = t; j < n; j += nt) {
    const QBox b = qbox(g, L, j);
    qb[j] = make_uint2(0x80008000u + (uint32_t)(b.x1 << 16 | (0x7FFF - b.x0)), 0x80008000u + (uint32_t)(b.y1 << 16 | (0x7FFF - b.y0)));
  }
}

// Finds the pairs (i of A, j of B) of local edges whose boxes come within (padx, pady) of each other, or a little more
// (TRI: one list, j > i only), and hands them to wave(i << SH | j, act) 32 at a time, one per lane; wave is called by
// the whole warp and ends the search by returning true (for all lanes). on_block(w, bits): lane i's pairs with B's 32
// edges from 32 w on, on_row(ic): A's 32 edges from ic on are done. qb: B's boxes (fill_boxes over the same box); the
// warp takes the 32 A edges from ic0 on, then those from ic0 + step on. Lists of up to 1 << SH edges (Q: the queue's type).
// A lane keeps the grid box of one A edge (per 32) in registers and tests B's edges one after the other, each read once
// for the whole warp (a shared-memory broadcast): 7 integer instructions a pair against ~24 with FP64 boxes. The pairs
// go through a queue, since a lane's own edge has few: the waves are full.
constexpr int QCAP = 64;
template <bool TRI, int SH, class EL, class Q, class Block, class Row, class Wave>
__device__ __forceinline__ void scan_edge_pairs(const EL& LA, int na, const EL& LB, int nb, const Box& box, double padx, double pady, const uint2* qb, Q* q,
                                                int ic0, int step, int lane, Block&& on_block, Row&& on_row, Wave&& wave) {
  const int nbw = (nb + 31) >> 5;
  const unsigned lt = (1u << lane) - 1;
  const QGrid g = qgrid(box);
  const int cx = 2 + (int)fminf((float)padx * g.sx * 32767.f, 32767.f), cy = 2 + (int)fminf((float)pady * g.sy * 32767.f, 32767.f);   // in cells, rounded up
  int qn = 0, ic = ic0, w = -1;   // ic, w: the 32 A edges and the 32 B edges being tested
  uint32_t bits = 0;
  uint2 ab = make_uint2(0u, 0u);
#pragma unroll 1
  for (bool more = ic0 < na && nb > 0; more || qn > 0;) {
#pragma unroll 1
    while (more && qn < 32) {
      const unsigned m = __ballot_sync(0xffffffffu, bits != 0);
      if (m) {   // each lane queues one of its pairs
        if (bits) {
          q[qn + __popc(m & lt)] = (Q)((ic + lane) << SH | ((w << 5) + __ffs(bits) - 1));
          bits &= bits - 1;
        }
        qn += __popc(m);
        continue;
      }
      if (w < 0 || ++w >= nbw) {   // next 32 A edges
        if (w >= nbw) {
          on_row(ic);
          ic += step;
          if (ic >= na) { more = false; break; }
        }
        w = TRI ? ic >> 5 : 0;
        const int i = ic + lane;
        if (i < na) {
          const QBox b = qbox(g, LA, i);
          ab = make_uint2((uint32_t)(max(b.x0 - cx, 0) << 16 | (0x7FFF - min(b.x1 + cx, 0x7FFF))),
                          (uint32_t)(max(b.y0 - cy, 0) << 16 | (0x7FFF - min(b.y1 + cy, 0x7FFF))));
        }
      }
      const uint2* qw = qb + (w << 5);
      const int n = min(32, nb - (w << 5));
#pragma unroll 1
      for (int j = 0; j < n; j += 4)   // up to 3 entries past the end are masked below
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint2 b = qw[j + k];
          if (((b.x - ab.x) & (b.y - ab.y) & 0x80008000u) == 0x80008000u) bits |= 1u << (j + k);
        }
      if (n < 32) bits &= (1u << n) - 1u;
      if (ic + lane >= na) bits = 0;
      if (TRI && w == (ic >> 5)) bits &= ~((2u << lane) - 1u);
      on_block(w, bits);
    }
    __syncwarp();
    const uint32_t e = q[lane];
    const Q rest = q[32 + lane];
    if (wave(e, lane < qn)) break;
    __syncwarp();
    qn = max(qn - 32, 0);
    if (lane < qn) q[lane] = rest;
    __syncwarp();
  }
  __syncwarp();
}

// filtered variants, no real boundary contact: intersects iff a real-edge vertex of one lies inside the other
// (engine.cuh:577-594); one probe at a time, the warp splitting the other polygon's edges (crossing parity is
// order-free). any: some probe vertex lies inside.
template <bool S32, class EL>
__device__ bool contains_warp(const Frame& A, const Frame& B, const EL& LA, int na, const EL& LB, int nb, bool inA_c, bool inB_c, const Box& ov, double cx,
                              double cy, int lane, bool& any) {
  bool h = false;
#pragma unroll 1
  for (int side = 0; side < 2 && !h; side++) {
    const Frame& S = side ? B : A;
    const EL& LO = side ? LA : LB;
    const int no_ = side ? na : nb;
    const bool inc = side ? inA_c : inB_c;
#pragma unroll 1
    for (uint32_t r = S.r0; r < S.r1 && !h; r++) {
      double x, y; const bool real = probe_vertex(S, r, x, y);
      if (!real) S.v(S.L->rvo[r], x, y);
      if (x >= ov.x0 && x <= ov.x1 && y >= ov.y0 && y <= ov.y1 && inside_from_c_warp<S32>(LO, no_, cx, cy, inc, x, y, lane)) {
        any = true; h = real;
      }
    }
  }
  return h;
}

}  // namespace gsj
