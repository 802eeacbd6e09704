// Candidate search: LBVH traversal. Many probes: QPT probe boxes per thread, probes taken in Morton order so the lanes of a warp
// walk neighbouring parts of the tree (the reference's k_traverse, engine/engine.cuh:233-259, runs a count pass
// and a write pass; here one pass appends with one atomic per warp step).
#include "engine.h"

namespace gsj {

constexpr int TRAV_STACK = 96;   // > tree depth (unique 64-bit keys bound the depth by 64)

__device__ __forceinline__ bool box_hit(const float4& c, const float4& b) {
  return !(c.x > b.z || c.z < b.x || c.y > b.w || c.w < b.y);
}

// QPT neighbouring probes per thread (adjacent in Morton order), walked in lockstep: each step issues all their node
// loads before testing any, so every lane keeps QPT independent load chains in flight (the walk is latency-bound:
// one dependent load per step otherwise).
constexpr int QPT = 4;
__global__ void __launch_bounds__(128) k_traverse(const float4* __restrict__ qbb, const uint32_t* __restrict__ qorder, uint32_t q0, uint32_t nq,
                                                  DBvh T, int upper, uint2* __restrict__ out, unsigned long long cap,
                                                  unsigned long long* counter, int* err, unsigned long long* visits) {
  const int lane = threadIdx.x & 31;
  const uint32_t t0 = (blockIdx.x * blockDim.x + threadIdx.x) * QPT;
  uint32_t qi[QPT];
  float4 b[QPT];
  int stack[QPT][TRAV_STACK];
  int sp[QPT], node[QPT];   // node: the next internal node to visit (register); only a second hit child is pushed
#pragma unroll
  for (int k = 0; k < QPT; k++) {
    const uint32_t t = t0 + k;
    sp[k] = 0; node[k] = -1; qi[k] = 0; b[k] = make_float4(0, 0, 0, 0);
    if (t < nq) {
      qi[k] = qorder ? qorder[q0 + t] : q0 + t;
      b[k] = qbb[qi[k]];
      node[k] = 0;
    }
  }
  const unsigned lt = (1u << lane) - 1;
  unsigned long long nvis = 0;
  for (;;) {
    bool any = false;
#pragma unroll
    for (int k = 0; k < QPT; k++) {
      if (node[k] < 0 && sp[k] > 0) node[k] = stack[k][--sp[k]];
      any = any || node[k] >= 0;
    }
    if (!__any_sync(0xffffffffu, any)) break;
    float4 lb[QPT], rb[QPT];
    int4 ch[QPT];
#pragma unroll
    for (int k = 0; k < QPT; k++)   // both loads first
      if (node[k] >= 0) {
        const BNode* np_ = T.nodes + node[k];
        lb[k] = __ldg(&np_->lb); rb[k] = __ldg(&np_->rb);
        ch[k] = __ldg(reinterpret_cast<const int4*>(&np_->l));
      }
    uint32_t hq[2 * QPT], hid[2 * QPT];
    int nh = 0;
#pragma unroll
    for (int k = 0; k < QPT; k++) {
      if (node[k] < 0) continue;
      nvis++;
      const bool hl = box_hit(lb[k], b[k]), hr = box_hit(rb[k], b[k]);
      int next = -1;
      if (hr) {
        if (ch[k].y < 0) { const uint32_t id = (uint32_t)~ch[k].y; if (!upper || id >= qi[k]) { hq[nh] = qi[k]; hid[nh] = id; nh++; } }
        else next = ch[k].y;
      }
      if (hl) {
        if (ch[k].x < 0) { const uint32_t id = (uint32_t)~ch[k].x; if (!upper || id >= qi[k]) { hq[nh] = qi[k]; hid[nh] = id; nh++; } }
        else {
          if (next >= 0) { if (sp[k] < TRAV_STACK) stack[k][sp[k]++] = next; else *err = 1; }
          next = ch[k].x;
        }
      }
      node[k] = next;
    }
    // warp-aggregated append: one atomic per warp step
    int x = nh;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int tot = __shfl_sync(0xffffffffu, x, 31);
    if (tot) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(counter, (unsigned long long)tot);
      base = __shfl_sync(0xffffffffu, base, 0);
      const unsigned long long pos = base + (unsigned long long)(x - nh);
#pragma unroll
      for (int h = 0; h < 2 * QPT; h++)
        if (h < nh && pos + h < cap) out[pos + h] = make_uint2(hq[h], hid[h]);
    }
  }
  (void)lt;
  for (int o = 16; o > 0; o >>= 1) nvis += __shfl_xor_sync(0xffffffffu, nvis, o);
  if (lane == 0 && nvis) atomicAdd(visits, nvis);
}

// Few probes: a warp per probe. Each lane takes one node of the probe's stack (in shared memory, newest first), so the
// warp walks up to 32 nodes a step and the walk takes about the tree's depth in steps instead of the nodes it visits.
// The stack: let b be the entries below the up to 32 that a step takes. None of these is above level b / 32 (whole part): it holds for the
// root; their children are a level deeper, and the next step's b is larger by 32 at most; and what a step leaves behind at
// place p < b' <= b + 32 is a child, at level b / 32 + 1 >= (p + 1) / 32 or deeper, so it holds as well when a later step reaches
// down to it. The deepest internal nodes are at level 63 (unique 64-bit keys), so a step that pushes has b / 32 <= 62: never more than
// 62 x 32 + 31 + 64 = 2079 entries.
constexpr int TW_WARPS = 4, TW_STACK = 32 * 65;
static_assert(TW_STACK >= 62 * 32 + 31 + 64, "the walk's bound");
// Against the thread form, ms: 200k parcels, 100 / 1k / 10k / 20k / 40k query boxes 0.029 / 0.029 / 0.054 / 0.077 / 0.127 against
// 0.078 / 0.090 / 0.103 / 0.103 / 0.113; 50 wide boxes over 20k zones 0.076 against 3.17 (one lane walked a whole box); a
// tree of 50 leaves under 20k boxes 0.051 against 0.041. Hence the lines:
constexpr uint32_t tw_probes(uint32_t leaves) { return leaves >= 8192 ? 24576 : 8192; }
__global__ void __launch_bounds__(TW_WARPS * 32) k_traverse_warp(const float4* __restrict__ qbb, const uint32_t* __restrict__ qorder, uint32_t q0, uint32_t nq,
                                                                 DBvh T, int upper, uint2* __restrict__ out, unsigned long long cap,
                                                                 unsigned long long* counter, int* err, unsigned long long* visits) {
  __shared__ int s_stack[TW_WARPS][TW_STACK];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1;
  int* stack = s_stack[threadIdx.x >> 5];
  const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= nq) return;
  const uint32_t qi = qorder ? qorder[q0 + t] : q0 + t;
  const float4 b = qbb[qi];
  unsigned long long nvis = 0;
  if (lane == 0) stack[0] = 0;
  __syncwarp();
  for (int sp = 1; sp > 0;) {
    const int take = min(sp, 32);
    int l = 0, r = 0;   // children: internal >= 0, leaves < 0
    bool hl = false, hr = false;
    if (lane < take) {
      const BNode* n = T.nodes + stack[sp - 1 - lane];
      const float4 lb = __ldg(&n->lb), rb = __ldg(&n->rb);
      const int4 ch = __ldg(reinterpret_cast<const int4*>(&n->l));
      l = ch.x; r = ch.y;
      hl = box_hit(lb, b); hr = box_hit(rb, b);
      if (l < 0 && upper && (uint32_t)~l < qi) hl = false;
      if (r < 0 && upper && (uint32_t)~r < qi) hr = false;
    }
    sp -= take;
    nvis += take;
    __syncwarp();
    const unsigned fl = __ballot_sync(0xffffffffu, hl && l < 0), fr = __ballot_sync(0xffffffffu, hr && r < 0);
    if (fl | fr) {   // one atomic per step
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(counter, (unsigned long long)(__popc(fl) + __popc(fr)));
      base = __shfl_sync(0xffffffffu, base, 0);
      const unsigned long long pl = base + __popc(fl & lt), pr = base + __popc(fl) + __popc(fr & lt);
      if (hl && l < 0 && pl < cap) out[pl] = make_uint2(qi, (uint32_t)~l);
      if (hr && r < 0 && pr < cap) out[pr] = make_uint2(qi, (uint32_t)~r);
    }
    const unsigned il = __ballot_sync(0xffffffffu, hl && l >= 0), ir = __ballot_sync(0xffffffffu, hr && r >= 0);
    const int more = __popc(il) + __popc(ir);
    if (sp + more > TW_STACK) { if (lane == 0) *err = 1; break; }
    if (hl && l >= 0) stack[sp + __popc(il & lt)] = l;
    if (hr && r >= 0) stack[sp + __popc(il) + __popc(ir & lt)] = r;
    sp += more;
    __syncwarp();
  }
  if (lane == 0 && nvis) atomicAdd(visits, nvis);
}

uint64_t traverse(gsj_ctx* c, const float4* qbb, const uint32_t* qorder, uint32_t q0, uint32_t nq, const DBvh& T, int upper, uint2* out,
                  uint64_t cap) {
  if (nq == 0) return 0;
  unsigned long long* ctr = c->counters.as<unsigned long long>(8);
  int* err = reinterpret_cast<int*>(ctr + 1);
  GSJ_CK(cudaMemsetAsync(ctr, 0, 24, c->stream));
  if (nq <= tw_probes(T.n)) k_traverse_warp<<<grid_for(nq, TW_WARPS), TW_WARPS * 32, 0, c->stream>>>(qbb, qorder, q0, nq, T, upper, out, cap, ctr, err, ctr + 2);
  else k_traverse<<<grid_for((nq + QPT - 1) / QPT, 128), 128, 0, c->stream>>>(qbb, qorder, q0, nq, T, upper, out, cap, ctr, err, ctr + 2);
  c->launches++;
  GSJ_CK(cudaGetLastError());
  unsigned long long* h = c->h_counters.as<unsigned long long>(3);
  GSJ_CK(cudaMemcpyAsync(h, ctr, 24, cudaMemcpyDeviceToHost, c->stream));
  GSJ_CK(cudaStreamSynchronize(c->stream));
  if (reinterpret_cast<int*>(h + 1)[0]) throw Error(GSJ_ERR_CUDA, "traversal stack overflow");
  c->node_visits += h[2];
  return h[0];
}

}  // namespace gsj
