// pcb_sparse.cuh — values and flows of the nodes outside dense blocks, one node and four examples per thread: shared by
// the kernels of single layers (pcb_em.cu) and of whole steps (pcb_chain.cu).
#pragma once
#include "pcb_internal.h"

namespace pcbsparse {
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ int64_t data_row(const int32_t* row_ids, uint32_t row_start, uint32_t b) {
  return row_ids ? (int64_t)row_ids[b] - 1 : (int64_t)row_start - 1 + b;
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 adds4(float4 a, float s) { return make_float4(a.x + s, a.y + s, a.z + s, a.w + s); }
__device__ __forceinline__ float4 max4(float4 a, float4 b) {
  return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
}
}  // namespace pcbsparse

// One thread per (node, four consecutive examples): every row access is a 16-byte load, so a warp
// keeps 512 bytes per request in flight (the chain node -> edge list -> child row is four dependent
// loads deep; with one example per thread it ran at a third of the memory roof).  Sum nodes: two
// passes over the children (max, then sum of exp), one exp per edge instead of the exp + log of a
// binary fold.  The last thread of a row may cover padding examples: the row pitch is a multiple
// of 32, and whatever lands in the padding is never read as a result.
struct PcbSparseUp {
  float* mars;
  uint32_t ld, B;
  const uint8_t* kind;
  const uint32_t* n_estart; const uint32_t* n_ecount; const uint32_t* n_pid0;
  const uint32_t* e_prime; const uint32_t* e_sub;
  const float* theta;
};
static inline PcbSparseUp pcb_sparse_up_args(const pcb_circuit* c, const pcb_workspace* ws) {
  return PcbSparseUp{ws->mars, ws->ld, ws->B, c->kind, c->n_estart, c->n_ecount, c->n_pid0, c->e_prime, c->e_sub, c->theta};
}
// node n, examples b .. b + 3; waits for the preceding launch of the chain
__device__ __forceinline__ void pcb_sparse_up_node(const PcbSparseUp& a, uint32_t n, uint32_t b) {
  using namespace pcbsparse;
  if (b >= a.B) return;
  float* const mars = a.mars;
  const uint32_t ld = a.ld;
  const uint32_t* const e_prime = a.e_prime;
  const uint32_t* const e_sub = a.e_sub;
  const uint32_t e0 = a.n_estart[n], cnt = a.n_ecount[n];
  pcb_grid_dep_wait();   // everything above is static circuit data
  auto child = [&](uint32_t j) {
    float4 v = ld4(mars + (size_t)e_prime[e0 + j] * ld + b);
    uint32_t sb = e_sub[e0 + j];
    if (sb != PCB_NONE) v = add4(v, ld4(mars + (size_t)sb * ld + b));
    return v;
  };
  float4 out;
  if (a.kind[n] == PCB_SUM) {
    const float* w = a.theta + a.n_pid0[n];
    float4 mx = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    for (uint32_t j = 0; j < cnt; ++j) mx = max4(mx, adds4(child(j), __ldg(w + j)));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t j = 0; j < cnt; ++j) {
      const float4 v = adds4(child(j), __ldg(w + j));
      // a maximum of -inf (every child impossible) gives exp(nan): masked below
      acc.x += __expf(v.x - mx.x); acc.y += __expf(v.y - mx.y); acc.z += __expf(v.z - mx.z); acc.w += __expf(v.w - mx.w);
    }
    out.x = mx.x == -INFINITY ? -INFINITY : mx.x + __logf(acc.x);
    out.y = mx.y == -INFINITY ? -INFINITY : mx.y + __logf(acc.y);
    out.z = mx.z == -INFINITY ? -INFINITY : mx.z + __logf(acc.z);
    out.w = mx.w == -INFINITY ? -INFINITY : mx.w + __logf(acc.w);
  } else {
    out = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t j = 0; j < cnt; ++j) out = add4(out, child(j));
  }
  *reinterpret_cast<float4*>(mars + (size_t)n * ld + b) = out;
}

// Pull-based top-down pass: flows[n][b] = sum over incoming edges of the edge flow
//   product parent: flows[parent]; sum parent: flows[parent] * exp(child value + logp - mars[parent]).
// The root (no incoming edge, last node) gets 1, any other parentless node 0.
// Multi-head circuits (head_mask != null): the flow of head h starts at head_mask[row, h], every
// other parentless node at 0 (src-jl/multi_head_pc/flow.jl:141-176).
struct PcbSparseDown {
  float* flows;
  const float* mars;
  uint32_t ld, B, root;
  const uint32_t* in_off; const PcbInEntry* in_ent;
  const float* theta;
  float* aggr;      // null: flows only
  PcbHeadInit hi;
};
static inline PcbSparseDown pcb_sparse_down_args(const pcb_circuit* c, const pcb_workspace* ws, const PcbHeadInit& hi) {
  return PcbSparseDown{ws->flows, ws->mars, ws->ld, ws->B, c->N - 1, c->in_off, c->in_ent, c->theta,
                       c->skip_stats ? nullptr : c->aggr, hi};
}
// node n, examples b .. b + 3 (all threads of a warp call it); waits for the preceding launch of the chain
__device__ __forceinline__ void pcb_sparse_down_node(const PcbSparseDown& a, uint32_t n, uint32_t b) {
  using namespace pcbsparse;
  float* const flows = a.flows;
  const float* const mars = a.mars;
  const uint32_t ld = a.ld, B = a.B, root = a.root;
  const uint32_t* const in_off = a.in_off;
  const PcbInEntry* const in_ent = a.in_ent;
  const float* const theta = a.theta;
  float* const aggr = a.aggr;
  const PcbHeadInit& hi = a.hi;
  const bool any = b < B;                      // examples b .. b+3, those below B count
  const uint32_t bb = any ? b : 0;
  const bool a0 = b < B, a1 = b + 1 < B, a2 = b + 2 < B, a3 = b + 3 < B;
  uint32_t i0 = in_off[n], i1 = in_off[n + 1];
  pcb_grid_dep_wait();   // everything above is static circuit data
  float4 acc;
  if (hi.head_mask) {
    const uint32_t h = hi.n_head[n];
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (h != PCB_NONE) {
      const float* mk = hi.head_mask + (size_t)hi.mask_rows * h;
      if (a0) acc.x = mk[data_row(hi.row_ids, hi.row_start, b)];
      if (a1) acc.y = mk[data_row(hi.row_ids, hi.row_start, b + 1)];
      if (a2) acc.z = mk[data_row(hi.row_ids, hi.row_start, b + 2)];
      if (a3) acc.w = mk[data_row(hi.row_ids, hi.row_start, b + 3)];
    }
  } else {
    const float init = (i0 == i1 && n == root) ? 1.0f : 0.0f;
    acc = make_float4(init, init, init, init);
  }
  const float4 my = ld4(mars + (size_t)n * ld + bb);
  for (uint32_t i = i0; i < i1; ++i) {
    PcbInEntry en = in_ent[i];
    float4 f = ld4(flows + (size_t)en.parent * ld + bb);
    if (en.pid != PCB_NONE) {
      const float4 pm = ld4(mars + (size_t)en.parent * ld + bb);
      const float lp = __ldg(theta + en.pid);
      // order of additions as in flow.jl:55-58: prime + logp, then + sub
      float4 child;
      if (en.sib == PCB_NONE) {
        child = adds4(my, lp);
      } else {
        const float4 sv = ld4(mars + (size_t)en.sib * ld + bb);
        child = (en.flags & 1u) ? add4(adds4(my, lp), sv) : add4(adds4(sv, lp), my);
      }
      f.x *= __expf(child.x - pm.x); f.y *= __expf(child.y - pm.y);
      f.z *= __expf(child.z - pm.z); f.w *= __expf(child.w - pm.w);
      if (aggr && (en.flags & 1u)) {   // aggr == null: flows only (uniform over the grid)
        float s = warp_sum((a0 ? f.x : 0.0f) + (a1 ? f.y : 0.0f) + (a2 ? f.z : 0.0f) + (a3 ? f.w : 0.0f));
        if ((threadIdx.x & 31) == 0) atomicAdd(aggr + en.pid, s);
      }
    }
    acc = add4(acc, f);
  }
  if (any) *reinterpret_cast<float4*>(flows + (size_t)n * ld + b) = acc;
}
