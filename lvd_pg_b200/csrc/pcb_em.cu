// pcb_em.cu — forward pass, backward flow pass, leaf statistics and the fused EM update.
//
// Reference kernels replaced (paths relative to VariationalJuice.jl/src):
//   leaf_forward_kernel    init_mar!_with_reg_kernel       regularization/reg_likelihood.jl:16-49
//   sparse_up_kernel       layer_up_kernel                 queries/likelihood.jl:4-68
//   sparse_down_kernel     layer_down_kernel / reg_layer_down_kernel
//                                                          queries/flow.jl:8-106, regularization/reg_flow.jl:120-222
//   leaf_flow_kernel       input_flows_circuit_with_reg_kernel   regularization/reg_flow.jl:24-48
//   em_update_*_kernel     add_pseudocount + aggr_node_flows + update_params + update_input_node_params
//                                                          regularization/reg_em.jl:292-299 (arithmetic:
//                                                          pretrain/mini_batch_warmup.jl:4-76, sgd/adam.jl:27-37,
//                                                          nodes/fixable_categorical_dist.jl:223-248)
//
// All kernels put the example index on threadIdx.x, so every access to a work matrix is a
// 128-byte coalesced row segment and edge metadata is a warp-wide broadcast.  The top-down pass
// is pull-based (CSR by child): a node sums the flows of its incoming edges itself, so node flows
// need no atomics and no zero-fill; only the per-edge statistics are reduced (warp shuffle, then
// one atomic per warp and edge).
#include <algorithm>

#include <cstring>

#include "pcb_internal.h"
#include "pcb_sparse.cuh"
#include "pcb_tc.cuh"

namespace {

constexpr int TPB = 128;  // threads per block along the example axis

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ int64_t data_row(const int32_t* row_ids, uint32_t row_start, uint32_t b) {
  return row_ids ? (int64_t)row_ids[b] - 1 : (int64_t)row_start - 1 + b;
}

__global__ void sparse_up_kernel(PcbSparseUp a, const uint32_t* __restrict__ nodes) {
  pcb_grid_dep_launch();
  pcb_sparse_up_node(a, nodes[blockIdx.x], (blockIdx.y * blockDim.x + threadIdx.x) * 4u);
}

__global__ void sparse_down_kernel(PcbSparseDown a, const uint32_t* __restrict__ nodes) {
  pcb_grid_dep_launch();
  pcb_sparse_down_node(a, nodes[blockIdx.x], (blockIdx.y * blockDim.x + threadIdx.x) * 4u);
}

// leaf statistics: aggr[foff + x_b] += flows[leaf][b] * w_b ; missing -> slot C
__global__ void leaf_flow_kernel(const float* __restrict__ flows, uint32_t ld, uint32_t B,
                                 float* __restrict__ aggr, const uint32_t* __restrict__ in_node,
                                 const uint32_t* __restrict__ in_var, const uint32_t* __restrict__ in_cats,
                                 const uint64_t* __restrict__ in_foff, const uint8_t* __restrict__ data,
                                 const uint8_t* __restrict__ miss, uint64_t num_rows,
                                 const int32_t* __restrict__ row_ids, uint32_t row_start,
                                 const float* __restrict__ weights) {
  uint32_t i = blockIdx.x;
  uint64_t fo = in_foff[i];
  if (fo == ~0ull) return;  // fixed leaf
  uint32_t b = blockIdx.y * blockDim.x + threadIdx.x;
  bool active = b < B;
  uint32_t slot = 0xffffffffu;
  float f = 0.0f;
  if (active) {
    int64_t row = data_row(row_ids, row_start, b);
    size_t di = (size_t)row + (size_t)num_rows * in_var[i];
    f = flows[(size_t)in_node[i] * ld + b];
    if (weights) f *= weights[row];
    slot = (miss && miss[di]) ? in_cats[i] : (uint32_t)data[di];
  }
  // combine the lanes of a warp that hit the same category before touching memory
  uint32_t peers = __match_any_sync(0xffffffffu, slot);
  uint32_t lane = threadIdx.x & 31;
  uint32_t leader = __ffs(peers) - 1;
  float total = 0.0f;
  for (uint32_t m = peers; m; m &= m - 1) {
    uint32_t src = __ffs(m) - 1;
    total += __shfl_sync(peers, f, src);
  }
  if (active && lane == leader) atomicAdd(aggr + fo + slot, total);
}

// ---- chunked leaf kernels -------------------------------------------------------------------------
// One block serves up to PCB_LEAF_CHUNK leaves of one variable for a tile of LBT examples: the
// variable's observed values are gathered once into shared memory (0xffff = missing) and reused
// by every leaf of the chunk, so the per-leaf work is a coalesced row read or write plus a
// table lookup that stays in L1.
constexpr int LBT = 2048;
constexpr int LTH = 256;

__device__ __forceinline__ void stage_values(uint16_t* xs, uint32_t b0, uint32_t nb, uint32_t var,
                                             const uint8_t* __restrict__ data, const uint8_t* __restrict__ miss,
                                             uint64_t num_rows, const int32_t* __restrict__ row_ids,
                                             uint32_t row_start) {
  for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) {
    int64_t row = data_row(row_ids, row_start, b0 + b);
    size_t di = (size_t)row + (size_t)num_rows * var;
    xs[b] = (miss && miss[di]) ? (uint16_t)0xffff : (uint16_t)data[di];
  }
}

__global__ void __launch_bounds__(LTH) leaf_forward_chunk_kernel(
    float* __restrict__ mars, uint32_t ld, uint32_t B, const float* __restrict__ theta,
    const uint32_t* __restrict__ in_node, const uint64_t* __restrict__ in_poff,
    const uint32_t* __restrict__ lchunk_var, const uint32_t* __restrict__ lchunk_off,
    const uint32_t* __restrict__ lchunk_inputs, const uint8_t* __restrict__ data,
    const uint8_t* __restrict__ miss, uint64_t num_rows, const int32_t* __restrict__ row_ids, uint32_t row_start) {
  __shared__ __align__(8) uint16_t xs[LBT];
  const uint32_t chunk = blockIdx.x, b0 = blockIdx.y * LBT;
  const uint32_t nb = min((uint32_t)LBT, B - b0);
  stage_values(xs, b0, nb, lchunk_var[chunk], data, miss, num_rows, row_ids, row_start);
  __syncthreads();
  // A thread takes four consecutive examples per pass (one 16-byte store per leaf and pass); its
  // examples are the same for every leaf of the group, so their values are fetched once.  The last
  // store of a row may reach into the padding of the row pitch (a multiple of 32).
  // A slice of at most 512 examples (the shard of a many-GPU step) leaves most threads without
  // examples: the block then walks several leaves at once, `tb` threads (whole warps) per leaf.
  constexpr uint32_t U = LBT / (4 * LTH);
  uint32_t tb = LTH;
  if (nb <= 2 * LTH) { tb = 32; while (4 * tb < nb) tb <<= 1; }
  const uint32_t te = threadIdx.x % tb, leaf_lane = threadIdx.x / tb, leaf_lanes = LTH / tb;
  uint16_t xv[U][4];
#pragma unroll
  for (uint32_t u = 0; u < U; ++u) {
    const uint32_t b = 4 * te + 4 * LTH * u;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) xv[u][j] = b + j < nb ? xs[b + j] : (uint16_t)0xffff;
  }
  for (uint32_t li = lchunk_off[chunk] + leaf_lane; li < lchunk_off[chunk + 1]; li += leaf_lanes) {
    uint32_t i = lchunk_inputs[li];
    const float* tab = theta + in_poff[i];
    float* out = mars + (size_t)in_node[i] * ld + b0;
    float v[U][4];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u)
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) v[u][j] = xv[u][j] == 0xffff ? 0.0f : __ldg(tab + xv[u][j]);
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t b = 4 * te + 4 * LTH * u;
      if (b < nb) *reinterpret_cast<float4*>(out + b) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
    }
  }
}

// Leaf statistics through a shared-memory histogram per leaf; a block that covers the whole
// batch owns its leaves' slots and adds without atomics.
__global__ void __launch_bounds__(LTH) leaf_flow_chunk_kernel(
    const float* __restrict__ flows, uint32_t ld, uint32_t B, float* __restrict__ aggr, uint32_t hstride,
    const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_cats,
    const uint64_t* __restrict__ in_foff, const uint32_t* __restrict__ lchunk_var,
    const uint32_t* __restrict__ lchunk_off, const uint32_t* __restrict__ lchunk_inputs,
    const uint8_t* __restrict__ data, const uint8_t* __restrict__ miss, uint64_t num_rows,
    const int32_t* __restrict__ row_ids, uint32_t row_start, const float* __restrict__ weights) {
  extern __shared__ float hist[];  // [PCB_LEAF_CHUNK][hstride]
  __shared__ uint16_t xs[LBT];
  const uint32_t chunk = blockIdx.x, b0 = blockIdx.y * LBT;
  const uint32_t nb = min((uint32_t)LBT, B - b0);
  const uint32_t l0 = lchunk_off[chunk], nl = lchunk_off[chunk + 1] - l0;
  for (uint32_t x = threadIdx.x; x < nl * hstride; x += LTH) hist[x] = 0.0f;
  stage_values(xs, b0, nb, lchunk_var[chunk], data, miss, num_rows, row_ids, row_start);
  __syncthreads();
  // a thread's examples (and their values and weights) are the same for every leaf of the chunk;
  // per leaf all of the thread's flow loads are issued before the first histogram update
  constexpr uint32_t U = LBT / LTH;
  uint16_t xv[U];
  float wv[U];
#pragma unroll
  for (uint32_t u = 0; u < U; ++u) {
    const uint32_t b = threadIdx.x + LTH * u;
    xv[u] = b < nb ? xs[b] : (uint16_t)0xfffe;   // 0xfffe: no example
    wv[u] = (weights && b < nb) ? weights[data_row(row_ids, row_start, b0 + b)] : 1.0f;
  }
  for (uint32_t l = 0; l < nl; ++l) {
    uint32_t i = lchunk_inputs[l0 + l];
    if (in_foff[i] == ~0ull) continue;  // fixed leaf
    const uint32_t C = in_cats[i];
    const float* f = flows + (size_t)in_node[i] * ld + b0;
    float* h = hist + l * hstride;
    float v[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t b = threadIdx.x + LTH * u;
      v[u] = f[b < nb ? b : 0u];
    }
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t slot = xv[u] == 0xffff ? C : (uint32_t)xv[u];   // missing value -> the extra slot
      if (xv[u] != 0xfffe && slot <= C) atomicAdd(h + slot, v[u] * wv[u]);
    }
  }
  __syncthreads();
  const bool whole = gridDim.y == 1;
  for (uint32_t x = threadIdx.x; x < nl * hstride; x += LTH) {
    uint32_t l = x / hstride, sl = x - l * hstride;
    uint32_t i = lchunk_inputs[l0 + l];
    uint64_t fo = in_foff[i];
    if (fo == ~0ull || sl > in_cats[i]) continue;
    float v = hist[x];
    if (v == 0.0f) continue;
    if (whole) aggr[fo + sl] += v; else atomicAdd(aggr + fo + sl, v);
  }
}

// Leaf statistics by sorted examples: the examples of the block's slice are sorted by the
// variable's value once (counting sort in shared memory), and every thread keeps up to LSE consecutive
// positions of the sorted order in registers for the whole group: the example behind each position,
// its value segment and (if given) its weight.  Then every leaf row of the group streams through a
// three-deep ring of shared-memory buffers (one bulk copy per row); a thread gathers its LSE values
// (independent loads, the same work for every thread whatever the histogram of the values looks
// like), sums runs of equal segment in registers and adds one partial sum per run to the row's
// shared-memory histogram; after the barrier the histogram leaves with one RED per slot while the
// next row is already being gathered into the other histogram.  A missing value sorts into the
// extra segment C.  The group's leaves share one variable, so one sort serves up to 64 rows.
constexpr int LSB = 2048;   // examples per block slice
constexpr int LST = 256;    // threads
constexpr int LSE = LSB / LST;   // sorted positions per thread
constexpr int LSR = 4;      // row buffers; the last one holds the sort's arrays until the sort is done
constexpr int LSC = 508;    // most categories of a variable (static + dynamic shared memory stay under 48 KB)
template <bool WEIGHTED>
__global__ void __launch_bounds__(LST) leaf_flow_sorted_kernel(
    const float* __restrict__ flows, uint32_t ld, uint32_t B, float* __restrict__ aggr,
    const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_foff,
    const uint32_t* __restrict__ lgrp_var, const uint32_t* __restrict__ lgrp_off,
    const uint32_t* __restrict__ linputs, uint32_t max_cats, const uint8_t* __restrict__ data,
    const uint8_t* __restrict__ miss, uint64_t num_rows, const int32_t* __restrict__ row_ids, uint32_t row_start,
    const float* __restrict__ weights, int* __restrict__ status) {
  __shared__ __align__(128) float rowbuf[LSR][LSB];
  __shared__ uint32_t binoff[LSC + 4];   // segment starts and the end; afterwards histogram 0
  __shared__ uint32_t cursor[LSC + 4];   // scatter cursors; afterwards histogram 1
  __shared__ uint64_t s_fo[PCB_LEAF_GROUP];   // the group's leaves: first statistics slot, categories
  __shared__ uint32_t s_cats[PCB_LEAF_GROUP];
  __shared__ __align__(8) uint64_t bar[LSR];
  static_assert(sizeof(float) * LSB == 2 * sizeof(uint16_t) * LSB, "the sort's two arrays fill one row buffer");
  uint16_t* xs = reinterpret_cast<uint16_t*>(rowbuf[LSR - 1]);   // values of the examples
  uint16_t* perm = xs + LSB;                                      // examples in sorted order
  const uint32_t grp = blockIdx.x, b0 = blockIdx.y * LSB, tid = threadIdx.x;
  const uint32_t nb = min((uint32_t)LSB, B - b0);
  const uint32_t l0 = lgrp_off[grp], nl = lgrp_off[grp + 1] - l0;
  // segments: values 0 .. max_cats (a value equal to a leaf's category count lands in that leaf's
  // extra slot, larger ones are dropped, as in the atomic kernel), then the missing-value segment
  constexpr uint32_t NOSEG = 0xffffffffu;
  const uint32_t miss_bin = max_cats + 1, nbins = max_cats + 2;
  if (tid == 0) {
    for (int r = 0; r < LSR; ++r) pcbtc::mbar_init(&bar[r], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (uint32_t x = tid; x <= nbins; x += LST) { binoff[x] = 0; }
  if (tid < nl) {
    const uint32_t i = linputs[l0 + tid];
    s_fo[tid] = in_foff[i];
    s_cats[tid] = in_cats[i];
  }
  stage_values(xs, b0, nb, lgrp_var[grp], data, miss, num_rows, row_ids, row_start);
  __syncthreads();
  // rows are requested as early as possible: the sort below hides their latency
  const uint32_t rowbytes = ((nb + 3u) & ~3u) * 4u;   // the pitch is a multiple of 32 floats: stays inside the row
  auto request = [&](uint32_t l) {
    const uint32_t i = linputs[l0 + l];
    pcbtc::mbar_arrive_expect_tx(&bar[l % LSR], rowbytes);
    pcbtc::bulk_g2s(rowbuf[l % LSR], flows + (size_t)in_node[i] * ld + b0, rowbytes, &bar[l % LSR]);
  };
  if (tid == 0) for (uint32_t l = 0; l < min(nl, (uint32_t)LSR - 1u); ++l) request(l);
  // counting sort of the examples by value
  for (uint32_t b = tid; b < nb; b += LST) {
    const uint32_t x = xs[b] == 0xffff ? miss_bin : xs[b] <= max_cats ? (uint32_t)xs[b] : NOSEG;
    if (x <= miss_bin) atomicAdd(&binoff[x + 1], 1u);
  }
  __syncthreads();
  if (tid < 32) {   // inclusive scan of the counts, one warp
    uint32_t carry = 0;
    for (uint32_t base = 0; base <= nbins; base += 32) {
      const uint32_t idx = base + tid;
      uint32_t v = idx <= nbins ? binoff[idx] : 0u;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, d);
        if ((int)tid >= d) v += u;
      }
      v += carry;
      if (idx <= nbins) binoff[idx] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  for (uint32_t x = tid; x < nbins; x += LST) cursor[x] = binoff[x];
  __syncthreads();
  for (uint32_t b = tid; b < nb; b += LST) {
    const uint32_t x = xs[b] == 0xffff ? miss_bin : xs[b] <= max_cats ? (uint32_t)xs[b] : NOSEG;
    if (x <= miss_bin) perm[atomicAdd(&cursor[x], 1u)] = (uint16_t)b;
  }
  __syncthreads();
  // this thread's sorted positions LSE * tid .. + LSE - 1: example, segment, weight
  uint32_t pos[LSE], seg[LSE];
  float wv[LSE];
  {
    // the sorted examples are dealt out evenly: a slice of fewer than 2048 examples still keeps every
    // thread busy, with fewer positions each
    const uint32_t total = binoff[nbins], per = (total + LST - 1u) / LST, j0 = per * tid;
    // segment of position j0: the last x with binoff[x] <= j0
    uint32_t lo = 0, hi = nbins;   // invariant: binoff[lo] <= j0 (binoff[0] = 0), answer in [lo, hi)
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (binoff[mid] <= j0) lo = mid; else hi = mid;
    }
    uint32_t x = lo;
#pragma unroll
    for (uint32_t e = 0; e < (uint32_t)LSE; ++e) {
      const uint32_t j = j0 + e;
      const bool in = e < per && j < total;
      while (in && binoff[x + 1] <= j) ++x;   // empty segments are stepped over
      pos[e] = in ? (uint32_t)perm[j] : 0u;
      seg[e] = in ? x : NOSEG;
      wv[e] = (WEIGHTED && in) ? weights[data_row(row_ids, row_start, b0 + pos[e])] : 1.0f;
    }
  }
  __syncthreads();   // binoff, cursor and the sort's arrays have been read by everyone
  if (tid == 0 && nl >= (uint32_t)LSR) {   // the last row buffer is free now
    pcbtc::fence_proxy_async();
    request(LSR - 1);
  }
  float* hist0 = reinterpret_cast<float*>(binoff);
  float* hist1 = reinterpret_cast<float*>(cursor);
  for (uint32_t x = tid; x < nbins; x += LST) { hist0[x] = 0.0f; hist1[x] = 0.0f; }
  __syncthreads();
  bool ok = true;
  for (uint32_t l = 0; l < nl; ++l) {
    const uint64_t fo = s_fo[l];
    const uint32_t C = s_cats[l];
    ok = ok && pcbtc::mbar_wait(&bar[l % LSR], (l / LSR) & 1u, status);
    const float* row = rowbuf[l % LSR];
    float* h = (l & 1u) ? hist1 : hist0;
    const bool live = ok && fo != ~0ull;
    if (live) {
      float v[LSE];
#pragma unroll
      for (uint32_t e = 0; e < (uint32_t)LSE; ++e) v[e] = row[pos[e]];
      float acc = 0.0f;
#pragma unroll
      for (uint32_t e = 0; e < (uint32_t)LSE; ++e) {
        if (e > 0 && seg[e] != seg[e - 1]) {   // positions past the end come last and carry NOSEG
          atomicAdd(h + seg[e - 1], acc);
          acc = 0.0f;
        }
        acc += WEIGHTED ? v[e] * wv[e] : v[e];
      }
      if (seg[LSE - 1] != NOSEG) atomicAdd(h + seg[LSE - 1], acc);
    }
    __syncthreads();   // the row has been read and its histogram is complete
    if (tid == 0 && ok && l + LSR < nl) {
      pcbtc::fence_proxy_async();
      request(l + LSR);
    }
    if (live) {
      // one fire-and-forget RED per slot; the histogram is cleared for the row after the next
      for (uint32_t x = tid; x < nbins; x += LST) {
        const float a = h[x];
        if (a == 0.0f) continue;
        h[x] = 0.0f;
        // leaf slot: value x <= C -> x, missing -> C; values beyond the leaf's categories are dropped
        const uint32_t slot = x == miss_bin ? C : x;
        if (slot <= C) atomicAdd(aggr + fo + slot, a);
      }
    }
  }
  if (!ok && tid == 0) {   // a wait was lost: let the copies in flight land before the block ends
    for (int r = 0; r < LSR; ++r) pcbtc::mbar_wait(&bar[r], 0, status);
  }
}

// Leaf statistics, lanes over leaves.  A block takes 32 leaves of one variable and walks its share of the batch in slices of 256
// examples: the rows of the leaves land in a tile in shared memory (16-byte loads along the examples, XOR-swizzled so
// that a column of 32 leaves lies in 32 banks; the next slice is in flight), then every warp walks its eighth of the
// slice's examples IN SORTED ORDER OF THEIR VALUE with one leaf per lane.  All lanes meet the same value at the same
// time, so a run of equal values is summed in a register and added to the histograms at its end without divergence; only
// the first and last run of a warp's share can be another warp's too and take an atomic.  About seven instructions per
// 32 (leaf, example) pairs; with the positions of a row dealt out over lanes instead it was fifteen, and a scan per row.
// The sorted order is made once per batch and variable by leaf_sort_kernel, beside the backward chain.  The histograms
// stay in shared memory over the slices and leave once, as REDs that nothing waits for.  Bound: HBM (the leaf rows of the flow matrix) once there are blocks for every SM.
// Alone on the GPU: 256 examples x 24576 leaves x 256 categories 67 -> 24 us, 512 x 98304 leaves 177 -> 134 us, 512 x
// 50176 leaves x 2 categories 601 -> 37 us, 256 x 1024 leaves x 2 categories 42 -> 6 us.
constexpr uint32_t LTT = 256, LTL = 32, LTS = 256, LTG = PCB_LEAF_GROUP / LTL;   // threads, leaves, examples of a slice
constexpr uint32_t LT_NOSEG = 0xffffu;

// order[slice][variable][256] = example | segment << 16 in order of the segments (values 0 .. max_cats, then missing);
// past the end of the slice LT_NOSEG
__global__ void __launch_bounds__(LTT) leaf_sort_kernel(
    uint32_t* __restrict__ order, uint32_t V, uint32_t B, uint32_t max_cats, const uint8_t* __restrict__ data,
    const uint8_t* __restrict__ miss, uint64_t num_rows, const int32_t* __restrict__ row_ids, uint32_t row_start) {
  __shared__ uint32_t cursor[LSC + 4];
  __shared__ uint16_t xs[LTS];
  const uint32_t var = blockIdx.x, tid = threadIdx.x, lane = tid & 31, miss_bin = max_cats + 1, nbins = max_cats + 2;
  for (uint32_t slice = blockIdx.y; slice < (B + LTS - 1) / LTS; slice += gridDim.y) {   // one unless there are more than the grid holds
    const uint32_t b0 = slice * LTS, nb = min(LTS, B - b0);
    uint32_t* const out = order + ((size_t)slice * V + var) * LTS;
    for (uint32_t x = tid; x <= nbins; x += LTT) cursor[x] = 0;
    stage_values(xs, b0, nb, var, data, miss, num_rows, row_ids, row_start);
    __syncthreads();
    const uint32_t x = tid >= nb ? LT_NOSEG : xs[tid] == 0xffff ? miss_bin : xs[tid] <= max_cats ? (uint32_t)xs[tid] : LT_NOSEG;
    const bool in = x <= miss_bin;
    if (in) atomicAdd(&cursor[x + 1], 1u);
    __syncthreads();
    if (tid < 32) {   // starts of the segments: exclusive sums of their sizes
      uint32_t carry = 0;
      for (uint32_t base = 0; base <= nbins; base += 32) {
        const uint32_t idx = base + lane;
        uint32_t v = idx <= nbins ? cursor[idx] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t u = __shfl_up_sync(0xffffffffu, v, d);
          if ((int)lane >= d) v += u;
        }
        v += carry;
        if (idx <= nbins) cursor[idx] = v;
        carry = __shfl_sync(0xffffffffu, v, 31);
      }
    }
    __syncthreads();
    const uint32_t total = cursor[nbins];
    __syncthreads();
    if (in) out[atomicAdd(&cursor[x], 1u)] = tid | (x << 16);
    if (tid >= total) out[tid] = LT_NOSEG << 16;
    __syncthreads();
  }
}

template <bool WEIGHTED>
__global__ void __launch_bounds__(LTT) leaf_flow_tile_kernel(
    const float* __restrict__ flows, uint32_t ld, uint32_t B, float* __restrict__ aggr,
    const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_foff,
    const uint32_t* __restrict__ lgrp_var, const uint32_t* __restrict__ lgrp_off,
    const uint32_t* __restrict__ linputs, uint32_t max_cats, const uint32_t* __restrict__ order, uint32_t V,
    const int32_t* __restrict__ row_ids, uint32_t row_start, const float* __restrict__ weights) {
  extern __shared__ float lt_hist[];   // [LTL][pitch], pitch odd
  __shared__ __align__(16) float tile[LTL * LTS];
  __shared__ uint64_t s_fo[LTL];
  __shared__ uint32_t s_cats[LTL];
  const uint32_t grp = blockIdx.x / LTG, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t l0 = lgrp_off[grp] + blockIdx.x % LTG * LTL, end = lgrp_off[grp + 1];
  if (l0 >= end) return;
  const uint32_t nl = min(LTL, end - l0), miss_bin = max_cats + 1, nbins = max_cats + 2, pitch = nbins | 1u, var = lgrp_var[grp];
  if (threadIdx.x < nl) {
    const uint32_t i = linputs[l0 + threadIdx.x];
    s_fo[threadIdx.x] = in_foff[i]; s_cats[threadIdx.x] = in_cats[i];
  }
  // this warp loads leaves 4 warp .. + 3: element (leaf, example) lies at leaf * 256 + (example ^ leaf)
  const float* src[4];
#pragma unroll
  for (uint32_t r = 0; r < 4; ++r) src[r] = flows + (size_t)in_node[linputs[l0 + min(warp * 4 + r, nl - 1)]] * ld + 4 * lane;
  float4 next[4][2];
  auto fetch = [&](uint32_t b0) {
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const bool in = b0 + 128 * u + 4 * lane < B;   // the pitch is a multiple of 32: a group of four is inside the row
#pragma unroll
      for (uint32_t r = 0; r < 4; ++r)
        next[r][u] = in ? __ldcs(reinterpret_cast<const float4*>(src[r] + b0 + 128 * u)) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (WEIGHTED) {
        float w[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
          const uint32_t b = b0 + 128 * u + 4 * lane + k;
          w[k] = b < B ? weights[data_row(row_ids, row_start, b)] : 0.0f;
        }
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r) { next[r][u].x *= w[0]; next[r][u].y *= w[1]; next[r][u].z *= w[2]; next[r][u].w *= w[3]; }
      }
    }
  };
  const uint32_t first = blockIdx.y * LTS, step = gridDim.y * LTS;   // this block's slices
  fetch(first);
  for (uint32_t x = threadIdx.x; x < LTL * pitch; x += LTT) lt_hist[x] = 0.0f;
  float* const h = lt_hist + lane * pitch;
  const float* const column = tile + lane * LTS;
  for (uint32_t b0 = first; b0 < B; b0 += step) {
    const uint32_t word = __ldg(order + ((size_t)(b0 / LTS) * V + var) * LTS + threadIdx.x);   // 32 sorted examples of this warp
    __syncthreads();   // the tile has been read (and, first, the histograms are clear)
    float4* const to = reinterpret_cast<float4*>(tile) + warp * 4 * (LTS / 4);
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const uint32_t g = (lane + 32 * u) ^ warp;
      to[g] = next[0][u];
      to[LTS / 4 + g] = make_float4(next[1][u].y, next[1][u].x, next[1][u].w, next[1][u].z);
      to[2 * (LTS / 4) + g] = make_float4(next[2][u].z, next[2][u].w, next[2][u].x, next[2][u].y);
      to[3 * (LTS / 4) + g] = make_float4(next[3][u].w, next[3][u].z, next[3][u].y, next[3][u].x);
    }
    __syncthreads();
    if (b0 + step < B) fetch(b0 + step);
    uint32_t seg = __shfl_sync(0xffffffffu, word, 0) >> 16;
    const uint32_t last = __shfl_sync(0xffffffffu, word, 31) >> 16;
    bool edge = true;   // the first run may have begun in the warp before
    float acc = 0.0f;
#pragma unroll 8
    for (uint32_t j = 0; j < 32; ++j) {
      const uint32_t w = __shfl_sync(0xffffffffu, word, j), s = w >> 16;
      if (s != seg) {   // the same for all lanes
        if (edge) atomicAdd(h + seg, acc); else h[seg] += acc;
        edge = false;
        acc = 0.0f;
        seg = s;
      }
      acc += s != LT_NOSEG ? column[(w & 0xffffu) ^ lane] : 0.0f;
    }
    if (last != LT_NOSEG) atomicAdd(h + last, acc);
  }
  __syncthreads();
  // value x <= C -> slot x, missing -> C, others are dropped
  for (uint32_t l = warp; l < nl; l += LTT / 32) {
    const uint32_t C = s_cats[l];
    const uint64_t fo = s_fo[l];
    if (fo == ~0ull) continue;   // fixed leaf
    for (uint32_t x = lane; x <= C; x += 32) {
      const float v = lt_hist[l * pitch + x] + (x == C ? lt_hist[l * pitch + miss_bin] : 0.0f);
      if (v != 0.0f) atomicAdd(aggr + fo + x, v);   // no return value: nothing waits for the statistics' old values
    }
  }
}

// ---- leaves under soft evidence / soft regularisation ----------------------------------------------
// One block per leaf, threads over the examples.  soft != null: per-category log-weights
// soft[row, var, c] ([rows, V, C] column-major) stand where the observed category stands
// (init_mar!_with_reg_cat_kernel, regularization/reg_likelihood.jl:51-91); else hard evidence with
// soft_reg > 0 (soft_loglikelihood, reg_likelihood.jl:4-14).
__global__ void leaf_forward_gen_kernel(float* __restrict__ mars, uint32_t ld, uint32_t B, const float* __restrict__ theta,
                                        const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_var,
                                        const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_poff,
                                        uint32_t num_vars, const uint8_t* __restrict__ data, const uint8_t* __restrict__ miss,
                                        const float* __restrict__ soft, uint64_t num_rows,
                                        const int32_t* __restrict__ row_ids, uint32_t row_start, float soft_reg, int32_t width) {
  const uint32_t i = blockIdx.x, b = blockIdx.y * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t row = data_row(row_ids, row_start, b);
  const uint32_t C = in_cats[i], var = in_var[i];
  const float* tab = theta + in_poff[i];
  float v;
  if (soft) {
    const float* sp = soft + (size_t)row + (size_t)num_rows * var;
    const size_t cs = (size_t)num_rows * num_vars;
    float mx = -INFINITY;
    for (uint32_t c = 0; c < C; ++c) mx = fmaxf(mx, sp[c * cs] + __ldg(tab + c));
    float acc = 0.0f;
    for (uint32_t c = 0; c < C; ++c) acc += expf(sp[c * cs] + __ldg(tab + c) - mx);
    v = mx == -INFINITY ? -INFINITY : mx + logf(acc);
  } else {
    const size_t di = (size_t)row + (size_t)num_rows * var;
    if (miss && miss[di]) {
      v = 0.0f;
    } else {
      const int32_t x = data[di];
      const int32_t c_start = max(0, x - width / 2), c_end = min(c_start + width - 1, (int32_t)C - 1);
      float sp = 0.0f;
      for (int32_t c = c_start; c <= c_end; ++c) sp += expf(__ldg(tab + c));
      sp /= (float)(c_end - c_start + 1);
      const float u = __ldg(tab + x) + logf(1.0f - soft_reg), w = logf(sp) + logf(soft_reg);
      const float m = fmaxf(u, w);
      v = (isfinite(u) && isfinite(w)) ? m + log1pf(expf(-fabsf(u - w))) : m;
    }
  }
  mars[(size_t)in_node[i] * ld + b] = v;
}

// Leaf statistics of the same two forms (input_flows_circuit_with_reg_cat_kernel reg_flow.jl:50-82;
// soft_flow reg_flow.jl:3-22, which uses the stored LOG-probabilities where it says heap[...]: kept
// as written).  A warp reduces its 32 examples per category before touching memory.
__global__ void leaf_flow_gen_kernel(const float* __restrict__ flows, const float* __restrict__ mars, uint32_t ld, uint32_t B,
                                     float* __restrict__ aggr, const float* __restrict__ theta,
                                     const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_var,
                                     const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_poff,
                                     const uint64_t* __restrict__ in_foff, uint32_t num_vars,
                                     const uint8_t* __restrict__ data, const uint8_t* __restrict__ miss,
                                     const float* __restrict__ soft, uint64_t num_rows, const int32_t* __restrict__ row_ids,
                                     uint32_t row_start, const float* __restrict__ weights, float soft_reg, int32_t width) {
  const uint32_t i = blockIdx.x, b = blockIdx.y * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const uint64_t fo = in_foff[i];
  if (fo == ~0ull) return;   // fixed leaf
  const bool active = b < B;
  const int64_t row = active ? data_row(row_ids, row_start, b) : 0;
  const uint32_t C = in_cats[i], var = in_var[i];
  const float* tab = theta + in_poff[i];
  float f = active ? flows[(size_t)in_node[i] * ld + b] : 0.0f;
  if (active && weights) f *= weights[row];
  if (soft) {
    const float logp = active ? mars[(size_t)in_node[i] * ld + b] : 0.0f;
    const float* sp = soft + (size_t)row + (size_t)num_rows * var;
    const size_t cs = (size_t)num_rows * num_vars;
    for (uint32_t c = 0; c < C; ++c) {
      float v = active ? expf(sp[c * cs] + __ldg(tab + c) - logp) * f : 0.0f;
      v = warp_sum(v);
      if (lane == 0 && v != 0.0f) atomicAdd(aggr + fo + c, v);
    }
    return;
  }
  if (!active) return;
  const size_t di = (size_t)row + (size_t)num_rows * var;
  if (miss && miss[di]) { atomicAdd(aggr + fo + C, f); return; }
  const int32_t x = data[di];
  const int32_t c_start = max(0, x - width / 2), c_end = min(c_start + width - 1, (int32_t)C - 1);
  float sp = 0.0f;
  for (int32_t c = c_start; c <= c_end; ++c) sp += expf(__ldg(tab + c));
  sp /= (float)(c_end - c_start + 1);
  const float base = (1.0f - soft_reg) * __ldg(tab + x) + soft_reg * sp;
  atomicAdd(aggr + fo + x, (1.0f - soft_reg) * __ldg(tab + x) * f / base);
  for (int32_t c = c_start; c <= c_end; ++c)
    atomicAdd(aggr + fo + c, soft_reg / (float)(c_end - c_start + 1) * __ldg(tab + c) * f / base);
}

// ---- soft evidence, the leaves of one variable together ----------------------------------------------
// logsumexp_c(s[b][c] + log p[leaf][c]) = ms[b] + log(sum_c p[leaf][c] * x[b][c]) with x = exp(s - ms), ms the largest
// weight of the example: the exponentials depend on the example alone and the rest is a product of two small matrices,
// where the kernels above take two exponentials per (leaf, example, category) and fetch the weights again for every leaf.
// The sum of a leaf whose probable categories all have negligible weights can leave the fp32 range that way: such a
// value (outside [1e-30, 1e30], or not a number) is computed as above, and so is its share of the statistics.
// Bound: the gather of the weights (rows of a batch are scattered) until there are enough blocks for the FMA pipes.
// 300 examples x 7200 leaves x 33 categories: forward 321 -> 50 us, statistics 184 -> 49 us.
// SOFT_MAX_CATS is what the two tiles of the forward kernel take of its 48 KB of static shared memory (36 + 64 words per
// category; 64 fill half of it, the next multiple of 64 would not fit) and the sums that a thread of the statistics
// holds (16).  More categories stay with the general kernels: 512 leaves x 4096 examples, 64 categories 93 and 84 us, 65
// categories 917 and 451 us.  CPT follows the categories because the products of the statistics do: 33 categories with ten
// sums a thread 39 us, with sixteen 60 us; 8 with two 23 us, with sixteen 45 us; 16 with four 27 us, with sixteen 49 us.
constexpr uint32_t SOFT_MAX_CATS = 64, SFT = 256, SFE = 32, SFP = SFE + 4;   // threads, examples of a tile, pitch of a row

__device__ __forceinline__ bool soft_in_range(float sum) { return sum >= 1e-30f && sum <= 1e30f; }

// x = exp(s - ms) [categories][SFP], ms [SFE] of examples b0 .. b0 + 31 of variable `var`; rows past C up to Cp are 0.
// Called by all threads; complete after the caller's barrier.
__device__ __forceinline__ void soft_stage(float* x, float* ms, uint32_t b0, uint32_t nb, uint32_t C, uint32_t Cp, uint32_t var,
                                           uint32_t num_vars, const float* __restrict__ soft, uint64_t num_rows,
                                           const int32_t* __restrict__ row_ids, uint32_t row_start) {
  const uint32_t e = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t row = e < nb ? data_row(row_ids, row_start, b0 + e) : 0;
  const float* sp = soft + (size_t)row + (size_t)num_rows * var;
  const size_t cs = (size_t)num_rows * num_vars;
#pragma unroll 4
  for (uint32_t c = w; c < Cp; c += SFT / 32) x[c * SFP + e] = c < C && e < nb ? sp[c * cs] : -INFINITY;
  __syncthreads();
  float m = -INFINITY;   // every warp finds the maximum for itself: 33 rows are read faster than exchanged
  for (uint32_t c = 0; c < C; ++c) m = fmaxf(m, x[c * SFP + e]);
  if (w == 0) ms[e] = m;
  __syncthreads();
  for (uint32_t c = w; c < Cp; c += SFT / 32) x[c * SFP + e] = c < C && e < nb ? expf(x[c * SFP + e] - m) : 0.0f;
}

// grid: (groups of up to 64 leaves of one variable, tiles of 32 examples)
__global__ void __launch_bounds__(SFT) leaf_forward_soft_kernel(
    float* __restrict__ mars, uint32_t ld, uint32_t B, const float* __restrict__ theta, const uint32_t* __restrict__ in_node,
    const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_poff, const uint32_t* __restrict__ lgrp_var,
    const uint32_t* __restrict__ lgrp_off, const uint32_t* __restrict__ linputs, uint32_t Cp, uint32_t num_vars,
    const float* __restrict__ soft, uint64_t num_rows, const int32_t* __restrict__ row_ids, uint32_t row_start) {
  __shared__ __align__(16) float x[SOFT_MAX_CATS * SFP], p[PCB_LEAF_GROUP * SOFT_MAX_CATS];
  __shared__ float ms[SFE];
  __shared__ uint32_t s_cats[PCB_LEAF_GROUP], top;
  const uint32_t l0 = lgrp_off[blockIdx.x], nl = lgrp_off[blockIdx.x + 1] - l0;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) top = 0;
  __syncthreads();
  if (threadIdx.x < nl) {
    s_cats[threadIdx.x] = in_cats[linputs[l0 + threadIdx.x]];
    atomicMax(&top, s_cats[threadIdx.x]);
  }
  __syncthreads();
  for (uint32_t l = warp; l < nl; l += SFT / 32) {
    const float* tab = theta + in_poff[linputs[l0 + l]];
    for (uint32_t c = lane; c < Cp; c += 32) p[l * Cp + c] = c < s_cats[l] ? expf(__ldg(tab + c)) : 0.0f;
  }
  for (uint32_t b0 = blockIdx.y * SFE; b0 < B; b0 += gridDim.y * SFE) {   // one tile unless there are more than the grid holds
    const uint32_t nb = min(SFE, B - b0);
    soft_stage(x, ms, b0, nb, top, Cp, lgrp_var[blockIdx.x], num_vars, soft, num_rows, row_ids, row_start);
    __syncthreads();
    for (uint32_t l = warp; l < nl; l += SFT / 32) {   // one example per lane
      float acc = 0.0f;
      const float4* pl = reinterpret_cast<const float4*>(p + l * Cp);   // Cp is a multiple of four
      for (uint32_t c = 0; c < Cp; c += 4) {
        const float4 w = pl[c / 4];
        acc = fmaf(w.x, x[c * SFP + lane], acc);
        acc = fmaf(w.y, x[(c + 1) * SFP + lane], acc);
        acc = fmaf(w.z, x[(c + 2) * SFP + lane], acc);
        acc = fmaf(w.w, x[(c + 3) * SFP + lane], acc);
      }
      if (lane >= nb) continue;
      const uint32_t i = linputs[l0 + l];
      float v = ms[lane] + logf(acc);
      if (!soft_in_range(acc)) {
        const float* tab = theta + in_poff[i];
        const float* sp = soft + (size_t)data_row(row_ids, row_start, b0 + lane) + (size_t)num_rows * lgrp_var[blockIdx.x];
        const size_t cs = (size_t)num_rows * num_vars;
        float mx = -INFINITY, sum = 0.0f;
        for (uint32_t c = 0; c < s_cats[l]; ++c) mx = fmaxf(mx, sp[c * cs] + __ldg(tab + c));
        for (uint32_t c = 0; c < s_cats[l]; ++c) sum += expf(sp[c * cs] + __ldg(tab + c) - mx);
        v = mx == -INFINITY ? -INFINITY : mx + logf(sum);
      }
      mars[(size_t)in_node[i] * ld + b0 + lane] = v;
    }
    if (b0 + gridDim.y * SFE < B) __syncthreads();
  }
}

// aggr[leaf][c] += p[leaf][c] * sum_b g[leaf][b] * x[b][c], g = flow * weight * exp(ms - value).  A block walks its share
// of the examples; thread (leaf, category mod 4) keeps the sums of up to CPT categories in registers.
// grid: (groups of up to 64 leaves of one variable, slices of the examples)
template <uint32_t CPT>
__global__ void __launch_bounds__(SFT) leaf_flow_soft_kernel(
    const float* __restrict__ flows, const float* __restrict__ mars, uint32_t ld, uint32_t B, float* __restrict__ aggr,
    const float* __restrict__ theta, const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_cats,
    const uint64_t* __restrict__ in_poff, const uint64_t* __restrict__ in_foff, const uint32_t* __restrict__ lgrp_var,
    const uint32_t* __restrict__ lgrp_off, const uint32_t* __restrict__ linputs, uint32_t num_vars,
    const float* __restrict__ soft, uint64_t num_rows, const int32_t* __restrict__ row_ids, uint32_t row_start,
    const float* __restrict__ weights) {
  constexpr uint32_t Cp = 4 * CPT;
  __shared__ __align__(16) float x[Cp * SFP], g[PCB_LEAF_GROUP * SFP];
  __shared__ float ms[SFE];
  __shared__ uint32_t s_cats[PCB_LEAF_GROUP], s_node[PCB_LEAF_GROUP], top;
  __shared__ uint64_t s_fo[PCB_LEAF_GROUP];
  const uint32_t l0 = lgrp_off[blockIdx.x], nl = lgrp_off[blockIdx.x + 1] - l0, var = lgrp_var[blockIdx.x];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, leaf = threadIdx.x & 63u, c0 = threadIdx.x >> 6;
  if (threadIdx.x == 0) top = 0;
  __syncthreads();
  if (threadIdx.x < nl) {
    const uint32_t i = linputs[l0 + threadIdx.x];
    s_cats[threadIdx.x] = in_cats[i]; s_node[threadIdx.x] = in_node[i]; s_fo[threadIdx.x] = in_foff[i];
    atomicMax(&top, s_cats[threadIdx.x]);
  }
  __syncthreads();
  const uint32_t C = top;
  float acc[CPT];
#pragma unroll
  for (uint32_t k = 0; k < CPT; ++k) acc[k] = 0.0f;
  for (uint32_t b0 = blockIdx.y * SFE; b0 < B; b0 += gridDim.y * SFE) {
    const uint32_t nb = min(SFE, B - b0);
    soft_stage(x, ms, b0, nb, C, Cp, var, num_vars, soft, num_rows, row_ids, row_start);
    const float wt = weights && lane < nb ? weights[data_row(row_ids, row_start, b0 + lane)] : 1.0f;
    for (uint32_t l = warp; l < PCB_LEAF_GROUP; l += SFT / 32) {
      float v = 0.0f;
      if (l < nl && lane < nb && s_fo[l] != ~0ull) {
        const float f = flows[(size_t)s_node[l] * ld + b0 + lane] * wt, val = mars[(size_t)s_node[l] * ld + b0 + lane];
        const float up = expf(ms[lane] - val);   // one over the sum that the value came from
        if (soft_in_range(up)) {
          v = f * up;
        } else {
          const float* tab = theta + in_poff[linputs[l0 + l]];
          const float* sp = soft + (size_t)data_row(row_ids, row_start, b0 + lane) + (size_t)num_rows * var;
          const size_t cs = (size_t)num_rows * num_vars;
          for (uint32_t c = 0; c < s_cats[l]; ++c) {
            const float share = expf(sp[c * cs] + __ldg(tab + c) - val) * f;
            if (share != 0.0f) atomicAdd(aggr + s_fo[l] + c, share);
          }
        }
      }
      g[l * SFP + lane] = v;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t e = 0; e < SFE; e += 4) {
      const float4 gv = *reinterpret_cast<const float4*>(g + leaf * SFP + e);
#pragma unroll
      for (uint32_t k = 0; k < CPT; ++k) {
        const float4 xv = *reinterpret_cast<const float4*>(x + (c0 + 4 * k) * SFP + e);   // the same for a warp
        acc[k] = fmaf(gv.x, xv.x, fmaf(gv.y, xv.y, fmaf(gv.z, xv.z, fmaf(gv.w, xv.w, acc[k]))));
      }
    }
    __syncthreads();
  }
  if (leaf >= nl || s_fo[leaf] == ~0ull) return;
  const float* tab = theta + in_poff[linputs[l0 + leaf]];
#pragma unroll
  for (uint32_t k = 0; k < CPT; ++k) {
    const uint32_t c = c0 + 4 * k;
    if (c < s_cats[leaf] && acc[k] != 0.0f) atomicAdd(aggr + s_fo[leaf] + c, expf(__ldg(tab + c)) * acc[k]);
  }
}

// Log-likelihoods of a multi-head circuit (extract_lls_from_root_nodes,
// src-jl/multi_head_pc/bit_circuit.jl:95-109): with a mask out[b] = logsumexp_h(mars[root_h][b] +
// log mask[row, h]) - log sum_h mask[row, h]; without one out is [B, H] with the roots' values.
__global__ void head_ll_kernel(const float* __restrict__ mars, uint32_t ld, uint32_t B, const uint32_t* __restrict__ roots,
                               uint32_t H, const float* __restrict__ head_mask, uint64_t mask_rows,
                               const int32_t* __restrict__ row_ids, uint32_t row_start, float* __restrict__ out) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  if (!head_mask) {
    for (uint32_t h = 0; h < H; ++h) out[(size_t)h * B + b] = mars[(size_t)roots[h] * ld + b];
    return;
  }
  const int64_t row = data_row(row_ids, row_start, b);
  float mx = -INFINITY, tot = 0.0f;
  for (uint32_t h = 0; h < H; ++h) {
    const float m = head_mask[(size_t)row + mask_rows * h];
    mx = fmaxf(mx, mars[(size_t)roots[h] * ld + b] + logf(m));
    tot += m;
  }
  float acc = 0.0f;
  for (uint32_t h = 0; h < H; ++h) {
    const float m = head_mask[(size_t)row + mask_rows * h];
    const float v = mars[(size_t)roots[h] * ld + b] + logf(m);
    if (v != -INFINITY) acc += expf(v - mx);
  }
  out[b] = (mx == -INFINITY ? -INFINITY : mx + logf(acc)) - logf(tot);
}

__global__ void scale_kernel(float* __restrict__ x, uint64_t n, float rate) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) x[i] = rate == 0.0f ? 0.0f : x[i] * rate;
}

// One warp per sum node: pseudocount, node normaliser, inertia blend, all in one pass.
__global__ void em_update_sum_kernel(float* __restrict__ theta, float* __restrict__ aggr,
                                     const uint32_t* __restrict__ grp_node, uint32_t n_groups,
                                     const uint32_t* __restrict__ n_pid0, const uint32_t* __restrict__ n_ecount,
                                     float pseudocount, float inertia) {
  uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t lane = threadIdx.x & 31;
  if (g >= n_groups) return;
  uint32_t n = grp_node[g];
  uint32_t p0 = n_pid0[n], cnt = n_ecount[n];
  float pc = pseudocount / (float)cnt;
  float tot = 0.0f;
  if ((cnt & 3u) == 0 && (p0 & 3u) == 0 && cnt <= 1024 && cnt > 1) {
    // aligned group of up to 1024 edges (every dense block): 16-byte accesses, statistics and
    // parameters loaded together and kept in registers between the two passes
    float4 a[8], th[8];
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      const uint32_t j = 4u * lane + 128u * u;
      if (j < cnt) {
        a[u] = *reinterpret_cast<const float4*>(aggr + p0 + j);
        th[u] = *reinterpret_cast<const float4*>(theta + p0 + j);
      }
    }
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      const uint32_t j = 4u * lane + 128u * u;
      if (j < cnt) {
        a[u].x += pc; a[u].y += pc; a[u].z += pc; a[u].w += pc;
        *reinterpret_cast<float4*>(aggr + p0 + j) = a[u];   // the reference keeps the pseudocount in edge_aggr
        tot += (a[u].x + a[u].y) + (a[u].z + a[u].w);
      }
    }
    tot = warp_sum(tot);
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      const uint32_t j = 4u * lane + 128u * u;
      if (j < cnt) {
        float4 o;
        o.x = logf(inertia * expf(th[u].x) + (1.0f - inertia) * a[u].x / tot);
        o.y = logf(inertia * expf(th[u].y) + (1.0f - inertia) * a[u].y / tot);
        o.z = logf(inertia * expf(th[u].z) + (1.0f - inertia) * a[u].z / tot);
        o.w = logf(inertia * expf(th[u].w) + (1.0f - inertia) * a[u].w / tot);
        *reinterpret_cast<float4*>(theta + p0 + j) = o;
      }
    }
    return;
  }
  for (uint32_t j = lane; j < cnt; j += 32) {
    float a = aggr[p0 + j] + pc;
    aggr[p0 + j] = a;  // the reference keeps the pseudocount in edge_aggr
    tot += a;
  }
  tot = warp_sum(tot);
  if (cnt == 1) return;  // single-edge sum nodes keep their parameter (reg_em.jl:150)
  for (uint32_t j = lane; j < cnt; j += 32) {
    float oldv = inertia * expf(theta[p0 + j]);
    float newv = (1.0f - inertia) * aggr[p0 + j] / tot;
    theta[p0 + j] = logf(oldv + newv);
  }
}

// One warp per learnable leaf (fixable_categorical_dist.jl:223-248).
__global__ void em_update_leaf_kernel(float* __restrict__ theta, const float* __restrict__ aggr,
                                      uint32_t n_inputs, const uint32_t* __restrict__ in_cats,
                                      const uint64_t* __restrict__ in_poff, const uint64_t* __restrict__ in_foff,
                                      float pseudocount, float inertia) {
  uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t lane = threadIdx.x & 31;
  if (i >= n_inputs) return;
  uint64_t fo = in_foff[i];
  if (fo == ~0ull) return;
  uint32_t C = in_cats[i];
  uint64_t po = in_poff[i];
  if (C <= 256) {
    // statistics and parameters of the leaf loaded together and kept in registers between the passes
    float a[8], th[8];
    float s = 0.0f;
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      const uint32_t k = lane + 32u * u;
      if (k < C) { a[u] = aggr[fo + k]; th[u] = theta[po + k]; }
    }
    const float missing_flow = aggr[fo + C];
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) if (lane + 32u * u < C) s += a[u];
    s = warp_sum(s);
    const float node_flow = s + (missing_flow + pseudocount);
    const float cat_pc = pseudocount / (float)C;
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      const uint32_t k = lane + 32u * u;
      if (k < C) {
        const float oldp = expf(th[u]);
        const float newv = (1.0f - inertia) * (a[u] + cat_pc + missing_flow * oldp) / node_flow;
        theta[po + k] = logf(inertia * oldp + newv);
      }
    }
    return;
  }
  float s = 0.0f;
  for (uint32_t k = lane; k < C; k += 32) s += aggr[fo + k];
  s = warp_sum(s);
  float missing_flow = aggr[fo + C];
  float node_flow = s + (missing_flow + pseudocount);
  float cat_pc = pseudocount / (float)C;
  for (uint32_t k = lane; k < C; k += 32) {
    float oldp = expf(theta[po + k]);
    float oldv = inertia * oldp;
    float newv = (1.0f - inertia) * (aggr[fo + k] + cat_pc + missing_flow * oldp) / node_flow;
    theta[po + k] = logf(oldv + newv);
  }
}

__global__ void iota_ids_kernel(int32_t* __restrict__ ids, int32_t first, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ids[i] = first + (int32_t)i;
}

__global__ void ll_sum_kernel(const float* __restrict__ root_mars, uint32_t B, float* __restrict__ out) {
  __shared__ float sh[32];
  float s = 0.0f;
  for (uint32_t b = threadIdx.x; b < B; b += blockDim.x) s += root_mars[b];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0f;
    v = warp_sum(v);
    if (threadIdx.x == 0) *out = v;
  }
}

dim3 grid2(uint32_t items, uint32_t B) { return dim3(items, (B + TPB - 1) / TPB, 1); }
// grid of the kernels that take four examples per thread
dim3 grid2v(uint32_t items, uint32_t B) { return dim3(items, (B + 4 * TPB - 1) / (4 * TPB), 1); }

}  // namespace

#define PCB_TRY(expr)              \
  do {                             \
    int32_t _s = (expr);           \
    if (_s != PCB_OK) return _s;   \
  } while (0)

// ---- checked mode (PCB_CHECKED=1) ------------------------------------------------------------------
// The circuit's own index arrays are validated on the host when it is compiled; what arrives on the
// device at run time and is used as an index is the batch: row ids and observed categories.  The
// reference reads both under @inbounds.  In checked mode every pass first runs this kernel, which
// touches only what it has found in range, waits for it and refuses the pass with the first finding
// (no kernel of the pass is launched on a bad index).  word: [code, example, variable, value],
// code 1 = row id outside [1, num_rows], 2 = category not below the variable's category count.
__global__ void check_batch_kernel(const int32_t* __restrict__ row_ids, uint32_t row_start, uint32_t B, uint64_t num_rows,
                                   const uint8_t* __restrict__ data, const uint8_t* __restrict__ miss, uint32_t V,
                                   const uint32_t* __restrict__ var_cats, int32_t* __restrict__ word) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const int64_t row = row_ids ? (int64_t)row_ids[b] - 1 : (int64_t)row_start - 1 + b;
  if (row < 0 || (uint64_t)row >= num_rows) {
    if (atomicCAS(word, 0, 1) == 0) { word[1] = (int32_t)b; word[2] = 0; word[3] = (int32_t)(row + 1); }
    return;
  }
  if (!data) return;
  for (uint32_t v = blockIdx.y; v < V; v += gridDim.y) {
    const size_t di = (size_t)row + (size_t)num_rows * v;
    if (miss && miss[di]) continue;
    const uint32_t x = data[di];
    if (x >= var_cats[v] && atomicCAS(word, 0, 2) == 0) { word[1] = (int32_t)b; word[2] = (int32_t)v; word[3] = (int32_t)x; }
  }
}

int32_t pcb_check_batch(pcb_circuit* c, const pcb_evidence& ev, cudaStream_t st) {
  PCB_CUDA(cudaMemsetAsync(c->check_word, 0, 4 * sizeof(int32_t), st));
  dim3 grid((ev.B + 127) / 128, std::min<uint32_t>(std::max<uint32_t>(c->V, 1u), 64u));
  check_batch_kernel<<<grid, 128, 0, st>>>(ev.row_ids_dev, ev.row_start, ev.B, ev.num_rows, ev.data_dev, ev.miss_dev, c->V,
                                           c->var_cats, c->check_word);
  int32_t w[4] = {0, 0, 0, 0};
  PCB_CUDA(cudaMemcpyAsync(w, c->check_word, sizeof(w), cudaMemcpyDeviceToHost, st));
  PCB_CUDA(cudaStreamSynchronize(st));
  if (w[0] == 1)
    return pcb_fail(PCB_ERR_INVALID, "checked mode: example " + std::to_string(w[1]) + " of the batch names row " +
                                         std::to_string(w[3]) + ", outside 1 .. " + std::to_string(ev.num_rows));
  if (w[0] == 2)
    return pcb_fail(PCB_ERR_INVALID, "checked mode: example " + std::to_string(w[1]) + " of the batch has value " +
                                         std::to_string(w[3]) + " for variable " + std::to_string(w[2] + 1) +
                                         ", which has fewer categories");
  return PCB_OK;
}

static int32_t forward_impl(pcb_circuit* c, pcb_workspace* ws, const pcb_evidence& ev, float* ll_out_dev,
                            cudaStream_t st) {
  const uint32_t B = ev.B;
  PCB_REQUIRE(ev.data_dev || ev.soft_dev, "null argument");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  PCB_REQUIRE(B >= 1 && B <= ws->max_batch, "batch size exceeds the workspace");
  PCB_REQUIRE(ev.row_ids_dev || (ev.row_start >= 1 && (uint64_t)ev.row_start - 1 + B <= ev.num_rows),
              "row range out of bounds");
  PCB_REQUIRE(ev.soft_reg >= 0.0f && ev.soft_reg < 1.0f, "soft_reg must lie in [0, 1)");
  PCB_REQUIRE(ev.soft_reg == 0.0f || ev.soft_dev || ev.soft_reg_width >= 1, "soft_reg_width must be at least 1");
  PCB_REQUIRE(!ev.head_mask_dev || c->n_heads, "a head mask needs a multi-head circuit");
  PCB_CUDA(cudaSetDevice(c->device));
  if (c->checked) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(st, &cap);
    if (cap == cudaStreamCaptureStatusNone) PCB_TRY(pcb_check_batch(c, ev, st));
  }
  ws->B = B; ws->data = ev.data_dev; ws->miss = ev.miss_dev; ws->num_rows = ev.num_rows;
  ws->row_ids = ev.row_ids_dev; ws->row_start = ev.row_start; ws->have_forward = false;
  ws->soft = ev.soft_dev; ws->head_mask = ev.head_mask_dev;
  ws->soft_reg = ev.soft_dev ? 0.0f : ev.soft_reg; ws->soft_width = ev.soft_reg_width;
  bool tensor = false;   // weight images are rebuilt only for a pass that reads them
  for (uint32_t t = 1; t <= c->n_steps && !tensor; ++t)
    tensor = c->h_dense_off[t + 1] > c->h_dense_off[t] && !pcb_chain_takes(c, ws, t);
  if (c->use_tc && tensor) PCB_TRY(pcb_dense_tc_refresh(c, st));
  // the arrival counters of the K-split dense tiles return to zero by themselves; a pass that a lost
  // wait cut short must not leave a stale count to the next one
  if (ws->mn_tickets && tensor) PCB_CUDA(cudaMemsetAsync(ws->mn_tickets, 0, 296 * sizeof(uint32_t), st));
  if (c->n_inputs) {
    PcbProfScope ps(c, st, PCB_K_LEAF_FWD);
    if (ws->soft && c->max_cats <= SOFT_MAX_CATS) {
      leaf_forward_soft_kernel<<<dim3(c->n_lgrps, std::min(65535u, (B + SFE - 1) / SFE)), SFT, 0, st>>>(
          ws->mars, ws->ld, B, c->theta, c->in_node, c->in_cats, c->in_poff, c->lgrp_var, c->lgrp_off, c->lchunk_inputs,
          pcb_round_up(c->max_cats, 4), c->V, ws->soft, ev.num_rows, ev.row_ids_dev, ev.row_start);
    } else if (ws->soft || ws->soft_reg > 0.0f) {
      leaf_forward_gen_kernel<<<grid2(c->n_inputs, B), TPB, 0, st>>>(
          ws->mars, ws->ld, B, c->theta, c->in_node, c->in_var, c->in_cats, c->in_poff, c->V, ev.data_dev, ev.miss_dev,
          ws->soft, ev.num_rows, ev.row_ids_dev, ev.row_start, ws->soft_reg, (int32_t)ws->soft_width);
    } else {
      dim3 grid(c->n_lgrps, (B + LBT - 1) / LBT);   // groups of up to 64 leaves of one variable share the staged values
      leaf_forward_chunk_kernel<<<grid, LTH, 0, st>>>(ws->mars, ws->ld, B, c->theta, c->in_node, c->in_poff,
                                                      c->lgrp_var, c->lgrp_off, c->lchunk_inputs, ev.data_dev,
                                                      ev.miss_dev, ev.num_rows, ev.row_ids_dev, ev.row_start);
    }
  }
  auto sparse_up = [&](const uint32_t* nodes, uint32_t n, cudaStream_t ss, bool pdl) -> int32_t {
    if (!n) return PCB_OK;
    PcbProfScope ps(c, ss, PCB_K_SPARSE_UP);
    PCB_CUDA(pcb_launch_pdl(sparse_up_kernel, grid2v(n, B), dim3(TPB), 0, ss, pdl, pcb_sparse_up_args(c, ws), nodes));
    return PCB_OK;
  };
  for (uint32_t t = 1; t <= c->n_steps; ++t) {
    if (pcb_chain_takes(c, ws, t)) {   // everything of the step in one launch
      PCB_TRY(pcb_chain_forward(c, ws, t, st));
      continue;
    }
    // The products that the step's dense blocks form over their sources come first here; the other nodes and the
    // blocks do not depend on each other (both read earlier steps only): with a side stream they run side by side.
    PCB_TRY(sparse_up(c->st_prod + c->h_st_prod_off[t], c->h_st_prod_off[t + 1] - c->h_st_prod_off[t], st, c->pdl));
    const uint32_t n = c->h_st_up_off[t + 1] - c->h_st_up_off[t];
    const bool split = c->side && !c->prof.on && c->fwd_split && n && c->h_dense_off[t + 1] > c->h_dense_off[t];
    if (split) {
      PCB_CUDA(cudaEventRecord(c->ev_fork, st));
      PCB_CUDA(cudaStreamWaitEvent(c->side, c->ev_fork, 0));
    }
    PCB_TRY(sparse_up(c->st_up + c->h_st_up_off[t], n, split ? c->side : st, c->pdl && !split));
    PCB_TRY(pcb_dense_forward(c, ws, t, st));
    if (split) {
      PCB_CUDA(cudaEventRecord(c->ev_join, c->side));
      PCB_CUDA(cudaStreamWaitEvent(st, c->ev_join, 0));
    }
  }
  if (ll_out_dev) {
    if (c->n_heads) {
      PcbProfScope ps(c, st, PCB_K_MISC);
      head_ll_kernel<<<(B + 255) / 256, 256, 0, st>>>(ws->mars, ws->ld, B, c->head_roots, c->n_heads, ws->head_mask,
                                                      ev.num_rows, ev.row_ids_dev, ev.row_start, ll_out_dev);
    } else {
      PCB_CUDA(cudaMemcpyAsync(ll_out_dev, ws->mars + (size_t)(c->N - 1) * ws->ld, B * sizeof(float),
                               cudaMemcpyDeviceToDevice, st));
    }
  }
  PCB_CUDA(cudaGetLastError());
  ws->have_forward = true;
  return PCB_OK;
}

static pcb_evidence hard_evidence(const uint8_t* data_dev, const uint8_t* miss_dev, uint64_t num_rows,
                                  const int32_t* row_ids_dev, uint32_t row_start, uint32_t B) {
  pcb_evidence ev;
  memset(&ev, 0, sizeof(ev));
  ev.data_dev = data_dev; ev.miss_dev = miss_dev; ev.num_rows = num_rows; ev.row_ids_dev = row_ids_dev;
  ev.row_start = row_start; ev.B = B; ev.soft_reg_width = 1;
  return ev;
}

extern "C" int32_t pcb_forward(pcb_circuit* c, pcb_workspace* ws, const uint8_t* data_dev,
                               const uint8_t* miss_dev, uint64_t num_rows, const int32_t* row_ids_dev,
                               uint32_t row_start, uint32_t B, float* ll_out_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws && data_dev, "null argument");
  return forward_impl(c, ws, hard_evidence(data_dev, miss_dev, num_rows, row_ids_dev, row_start, B), ll_out_dev,
                      (cudaStream_t)s);
}

extern "C" int32_t pcb_forward_ex(pcb_circuit* c, pcb_workspace* ws, const pcb_evidence* ev, float* ll_out_dev,
                                  pcb_stream s) {
  PCB_REQUIRE(c && ws && ev, "null argument");
  return forward_impl(c, ws, *ev, ll_out_dev, (cudaStream_t)s);
}

// Multi-GPU step: once every edge statistic of the batch is final (the sparse nodes' in stream order,
// the dense blocks' on the side stream) their slice of the statistics vector is summed over the ranks
// on the communication stream, while this stream goes on to the leaf statistics.
static int32_t comm_edges_begin(pcb_circuit* c, cudaStream_t st) {
  PCB_CUDA(cudaEventRecord(c->ev_c0, st));
  PCB_CUDA(cudaStreamWaitEvent(c->comm_stream, c->ev_c0, 0));
  if (c->side && c->side_busy) {
    PCB_CUDA(cudaEventRecord(c->ev_c1, c->side));
    PCB_CUDA(cudaStreamWaitEvent(c->comm_stream, c->ev_c1, 0));
  }
  PcbProfScope ps(c, c->comm_stream, PCB_K_ALLREDUCE);
  return pcb_allreduce_range(c, 0, c->n_inner, c->comm_stream);
}
// ... and the rest (leaf slots, batch log-likelihood) after them; the caller's stream waits for both.
static int32_t comm_rest_and_join(pcb_circuit* c, cudaStream_t st) {
  PCB_CUDA(cudaEventRecord(c->ev_c2, st));
  PCB_CUDA(cudaStreamWaitEvent(c->comm_stream, c->ev_c2, 0));
  { PcbProfScope ps(c, c->comm_stream, PCB_K_ALLREDUCE);
    PCB_TRY(pcb_allreduce_range(c, c->n_inner, c->aggr_len - c->n_inner, c->comm_stream)); }
  PCB_CUDA(cudaEventRecord(c->ev_c3, c->comm_stream));
  PCB_CUDA(cudaStreamWaitEvent(st, c->ev_c3, 0));
  return PCB_OK;
}

// early: a single-GPU step updates the sum parameters (and refreshes the weight images) on the side
// stream as soon as the last edge statistics are in, beside the leaf statistics of this stream.
struct EarlyUpdate { float pseudocount, inertia; bool done; };
static int32_t em_update_sums(pcb_circuit* c, float pseudocount, float inertia, cudaStream_t st);
static int32_t backward_impl(pcb_circuit* c, pcb_workspace* ws, const float* weights_dev, cudaStream_t st, bool split_comm,
                             EarlyUpdate* early = nullptr);

extern "C" int32_t pcb_backward(pcb_circuit* c, pcb_workspace* ws, const float* weights_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws, "null argument");
  return backward_impl(c, ws, weights_dev, (cudaStream_t)s, false);
}

// Whether lanes over leaves form the leaf statistics of hard evidence.  Few categories make long runs, where one thread
// per example contends for a histogram's few words; many examples per category give the sorted kernel whole rows to
// stream (each kernel alone on the GPU, 768 variables x 64 leaves: 2048 examples x 2 categories 1873 -> 115 us, 1024 x 100
// 158 -> 78 us, 1024 x 256 116 against 120 us, 2048 x 256 154 against 217 us).
static bool leaf_takes_tiles(const pcb_circuit* c, uint32_t B) {
  return c->max_cats <= LSC && c->leaf_flow_impl == 0 && (c->max_cats <= 128 || B < 1024);
}

static int32_t backward_impl(pcb_circuit* c, pcb_workspace* ws, const float* weights_dev, cudaStream_t st, bool split_comm,
                             EarlyUpdate* early) {
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  if (!ws->have_forward) return pcb_fail(PCB_ERR_STATE, "pcb_backward needs a preceding pcb_forward on this workspace");
  PCB_CUDA(cudaSetDevice(c->device));
  const uint32_t B = ws->B;
  PCB_REQUIRE(!c->n_heads || ws->head_mask, "the flows of a multi-head circuit need a head mask");
  const PcbHeadInit hi{c->n_head, ws->head_mask, ws->num_rows, ws->row_ids, ws->row_start};
  c->edge_lo = c->edge_hi = 0;
  auto sparse_down = [&](const uint32_t* nodes, uint32_t n, cudaStream_t ss, bool pdl) -> int32_t {
    if (!n) return PCB_OK;
    PcbProfScope ps(c, ss, PCB_K_SPARSE_DOWN);
    PCB_CUDA(pcb_launch_pdl(sparse_down_kernel, grid2v(n, B), dim3(TPB), 0, ss, pdl, pcb_sparse_down_args(c, ws, hi), nodes));
    return PCB_OK;
  };
  auto pulled = [&](uint32_t t, cudaStream_t ss, bool pdl) {
    return sparse_down(c->st_down + c->h_st_down_off[t], c->h_st_down_off[t + 1] - c->h_st_down_off[t], ss, pdl);
  };
  // Step t: its dense blocks push flows to their children (and to the nodes their fused products are products of),
  // and the other nodes of step t - 1, whose parents all lie in steps >= t and are never children of a step-t block,
  // pull theirs.  The first launch of the pass waits for the forward pass in full: the chain kernels read node values
  // before they wait for the launch ahead of them.
  const bool split = c->side2 && !c->prof.on && c->bwd_split;
  // the tile kernel's sorted order depends on the batch alone: it is made beside the first steps
  const bool leaf_tiles = c->n_inputs && !c->skip_stats && !ws->soft && ws->soft_reg == 0.0f && ws->leaf_order && leaf_takes_tiles(c, B);
  const bool sorted_beside = leaf_tiles && c->side2 && !c->prof.on;
  if (leaf_tiles) {
    cudaStream_t ss = sorted_beside ? c->side2 : st;
    if (sorted_beside) {
      PCB_CUDA(cudaEventRecord(c->ev_fork2, st));
      PCB_CUDA(cudaStreamWaitEvent(c->side2, c->ev_fork2, 0));
    }
    { PcbProfScope ps(c, ss, PCB_K_LEAF_FLOW);
      leaf_sort_kernel<<<dim3(c->V, std::min(65535u, (B + LTS - 1) / LTS)), LTT, 0, ss>>>(
          ws->leaf_order, c->V, B, c->max_cats, ws->data, ws->miss, ws->num_rows, ws->row_ids, ws->row_start); }
    if (sorted_beside) PCB_CUDA(cudaEventRecord(c->ev_sort, c->side2));
  }
  PCB_TRY(pulled(c->n_steps, st, false));
  for (uint32_t t = c->n_steps; t >= 1; --t) {
    const uint32_t dense = c->h_dense_off[t + 1] - c->h_dense_off[t], others = c->h_st_down_off[t] - c->h_st_down_off[t - 1];
    if (!dense) {
      PCB_TRY(pulled(t - 1, st, c->pdl));
    } else if (pcb_chain_takes(c, ws, t)) {
      PCB_TRY(pcb_dense_tc_note_edges(c, ws, t, st));
      PCB_TRY(pcb_chain_backward(c, ws, t, hi, st));
    } else {
      const bool beside = split && others;
      if (beside) {   // the pulling nodes beside the blocks on a second side stream
        PCB_CUDA(cudaEventRecord(c->ev_fork2, st));
        PCB_CUDA(cudaStreamWaitEvent(c->side2, c->ev_fork2, 0));
        PCB_TRY(pulled(t - 1, c->side2, false));
      }
      PCB_TRY(pcb_dense_backward(c, ws, t, st));
      PCB_TRY(sparse_down(c->st_src + c->h_st_src_off[t], c->h_st_src_off[t + 1] - c->h_st_src_off[t], st, c->pdl));
      if (beside) {
        PCB_CUDA(cudaEventRecord(c->ev_join2, c->side2));
        PCB_CUDA(cudaStreamWaitEvent(st, c->ev_join2, 0));
      } else {
        PCB_TRY(pulled(t - 1, st, c->pdl));
      }
    }
  }
  if (c->use_tc && !c->skip_stats) PCB_TRY(pcb_dense_tc_flush_edges(c, ws, st));
  if (split_comm) PCB_TRY(comm_edges_begin(c, st));
  if (early && c->side && c->use_tc && !c->prof.on) {
    // every edge statistic is final once this stream's kernels so far and the side stream's are done
    PCB_CUDA(cudaEventRecord(c->ev_fork, st));
    PCB_CUDA(cudaStreamWaitEvent(c->side, c->ev_fork, 0));
    PCB_TRY(em_update_sums(c, early->pseudocount, early->inertia, c->side));
    PCB_TRY(pcb_dense_tc_refresh(c, c->side));
    c->side_busy = true;
    early->done = true;
  }
  if (c->n_inputs && !c->skip_stats) {
    PcbProfScope ps(c, st, PCB_K_LEAF_FLOW);
    // sorted segments pay off once a variable has enough values to keep a block's threads busy;
    // PCB_LEAF_FLOW_IMPL=atomic / sorted (read when the circuit is created) forces one of the two kernels
    const bool want_sorted = c->leaf_flow_impl ? c->leaf_flow_impl == 2 : c->max_cats >= 16;
    if (ws->soft && c->max_cats <= SOFT_MAX_CATS) {
      // examples of a group shared out so that there are about four blocks per SM
      const uint32_t tiles = (B + SFE - 1) / SFE, slices = std::max(1u, std::min(tiles, 148 * 4 / std::max(1u, c->n_lgrps)));
      auto* kern = c->max_cats <= 8 ? leaf_flow_soft_kernel<2> : c->max_cats <= 16 ? leaf_flow_soft_kernel<4>
                 : c->max_cats <= 40 ? leaf_flow_soft_kernel<10> : leaf_flow_soft_kernel<16>;
      kern<<<dim3(c->n_lgrps, slices), SFT, 0, st>>>(
          ws->flows, ws->mars, ws->ld, B, c->aggr, c->theta, c->in_node, c->in_cats, c->in_poff, c->in_foff, c->lgrp_var,
          c->lgrp_off, c->lchunk_inputs, c->V, ws->soft, ws->num_rows, ws->row_ids, ws->row_start, weights_dev);
    } else if (ws->soft || ws->soft_reg > 0.0f) {
      leaf_flow_gen_kernel<<<grid2(c->n_inputs, B), TPB, 0, st>>>(
          ws->flows, ws->mars, ws->ld, B, c->aggr, c->theta, c->in_node, c->in_var, c->in_cats, c->in_poff, c->in_foff,
          c->V, ws->data, ws->miss, ws->soft, ws->num_rows, ws->row_ids, ws->row_start, weights_dev, ws->soft_reg,
          (int32_t)ws->soft_width);
    } else if (leaf_tiles) {
      static PcbPerDeviceOnce once;
      PCB_CUDA(once.run([] {
        const int most = (int)(LTL * (LSC + 3) * sizeof(float));
        const cudaError_t e = cudaFuncSetAttribute(leaf_flow_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        return e != cudaSuccess ? e : cudaFuncSetAttribute(leaf_flow_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      }));
      if (sorted_beside) PCB_CUDA(cudaStreamWaitEvent(st, c->ev_sort, 0));
      auto* kern = weights_dev ? leaf_flow_tile_kernel<true> : leaf_flow_tile_kernel<false>;
      // few leaves and many examples: the slices of a batch are dealt out so that there are about four blocks per SM
      // (a step of 8 variables x 16 latents x 65536 examples: 2 categories 1150 -> 252 us, 100 categories 1343 -> 261 us;
      // 64 variables x 16384 examples x 100 categories 752 -> 443 us)
      const uint32_t tiles = std::max(c->n_lgrps, (c->n_inputs + LTL - 1) / LTL), slices = (B + LTS - 1) / LTS;
      // (and no histogram adds up more than 256 slices one after the other)
      const uint32_t parts = std::min(65535u, std::max((slices + 255) / 256, std::min(slices, 148 * 4 / tiles)));
      kern<<<dim3(c->n_lgrps * LTG, parts), LTT, LTL * ((c->max_cats + 2) | 1u) * sizeof(float), st>>>(
          ws->flows, ws->ld, B, c->aggr, c->in_node, c->in_cats, c->in_foff, c->lgrp_var, c->lgrp_off, c->lchunk_inputs,
          c->max_cats, ws->leaf_order, c->V, ws->row_ids, ws->row_start, weights_dev);
    } else if (c->max_cats <= LSC && want_sorted) {
      dim3 grid(c->n_lgrps, (B + LSB - 1) / LSB);
      auto* kern = weights_dev ? leaf_flow_sorted_kernel<true> : leaf_flow_sorted_kernel<false>;
      kern<<<grid, LST, 0, st>>>(
          ws->flows, ws->ld, B, c->aggr, c->in_node, c->in_cats, c->in_foff, c->lgrp_var, c->lgrp_off,
          c->lchunk_inputs, c->max_cats, ws->data, ws->miss, ws->num_rows, ws->row_ids, ws->row_start, weights_dev,
          c->status);
    } else if (c->max_cats <= 1024) {
      uint32_t hstride = c->max_cats + 1;
      dim3 grid(c->n_lchunks, (B + LBT - 1) / LBT);
      leaf_flow_chunk_kernel<<<grid, LTH, PCB_LEAF_CHUNK * hstride * sizeof(float), st>>>(
          ws->flows, ws->ld, B, c->aggr, hstride, c->in_node, c->in_cats, c->in_foff, c->lchunk_var, c->lchunk_off,
          c->lchunk_inputs, ws->data, ws->miss, ws->num_rows, ws->row_ids, ws->row_start, weights_dev);
    } else {
      leaf_flow_kernel<<<grid2(c->n_inputs, B), TPB, 0, st>>>(ws->flows, ws->ld, B, c->aggr, c->in_node, c->in_var,
                                                              c->in_cats, c->in_foff, ws->data, ws->miss,
                                                              ws->num_rows, ws->row_ids, ws->row_start, weights_dev);
    }
  }
  PCB_TRY(pcb_side_join(c, st));  // the leaf statistics above overlap the last edge-statistics kernels
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

extern "C" int32_t pcb_clear_flows(pcb_circuit* c, float rate, pcb_stream s) {
  PCB_REQUIRE(c, "null argument");
  PCB_CUDA(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)s;
  if (rate == 0.0f) {
    PCB_CUDA(cudaMemsetAsync(c->aggr, 0, c->aggr_len * sizeof(float), st));
  } else {
    uint64_t n = c->aggr_len - 1;
    uint32_t blocks = (uint32_t)std::min<uint64_t>((n + 255) / 256, 148 * 16);
    if (n) { PcbProfScope ps(c, st, PCB_K_MISC); scale_kernel<<<blocks, 256, 0, st>>>(c->aggr, n, rate); }
    PCB_CUDA(cudaMemsetAsync(c->aggr + n, 0, sizeof(float), st));
    PCB_CUDA(cudaGetLastError());
  }
  return PCB_OK;
}

static int32_t em_update_sums(pcb_circuit* c, float pseudocount, float inertia, cudaStream_t st) {
  if (c->n_groups)
    { PcbProfScope ps(c, st, PCB_K_UPDATE); em_update_sum_kernel<<<(c->n_groups + 7) / 8, 256, 0, st>>>(c->theta, c->aggr, c->grp_node, c->n_groups,
                                                                c->n_pid0, c->n_ecount, pseudocount, inertia); }
  c->w_img_valid = false;  // the weights changed
  return PCB_OK;
}
static int32_t em_update_leaves(pcb_circuit* c, float pseudocount, float inertia, cudaStream_t st) {
  if (c->n_inputs)
    { PcbProfScope ps(c, st, PCB_K_UPDATE); em_update_leaf_kernel<<<(c->n_inputs + 7) / 8, 256, 0, st>>>(c->theta, c->aggr, c->n_inputs, c->in_cats,
                                                                 c->in_poff, c->in_foff, pseudocount, inertia); }
  return PCB_OK;
}

extern "C" int32_t pcb_em_update(pcb_circuit* c, float pseudocount, float inertia, pcb_stream s) {
  PCB_REQUIRE(c, "null argument");
  PCB_CUDA(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)s;
  PCB_TRY(em_update_sums(c, pseudocount, inertia, st));
  PCB_TRY(em_update_leaves(c, pseudocount, inertia, st));
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

// clear, forward, backward, (all-reduce,) update: the launches of one EM step on stream st.  The
// batch log-likelihood stays in the last slot of the statistics vector; pcb_em_step copies it out.
static int32_t em_step_body(pcb_circuit* c, pcb_workspace* ws, const pcb_evidence& ev, const float* weights_dev,
                            float clear_rate, float pseudocount, float inertia, cudaStream_t st) {
  pcb_stream s = (pcb_stream)st;
  const uint32_t B = ev.B;
  // With a communicator every rank enters the step holding the same summed statistics of the last
  // step (pseudocount included, as the reference keeps it in edge_aggr); the all-reduce below adds
  // the ranks' vectors, so each rank carries rate / nranks of them and the sum is rate * previous
  // + this step's flows, as reg_em.jl:276-284 computes it on one device.
  const float carried = (c->comm && c->nranks > 1) ? clear_rate / (float)c->nranks : clear_rate;
  PCB_TRY(pcb_clear_flows(c, carried, s));
  // multi-head circuits: the per-example log-likelihoods mix the heads (em.jl:71 of multi_head_pc)
  { PcbNvtxRange r("pcb forward"); PCB_TRY(forward_impl(c, ws, ev, c->n_heads ? ws->ll_tmp : nullptr, st)); }
  const bool multi = c->comm && c->nranks > 1 && c->comm_enabled;
  const bool split = multi && c->comm_split && !c->prof.on;   // per-class timing wants every class alone on the GPU
  EarlyUpdate early{pseudocount, inertia, false};
  { PcbNvtxRange r("pcb backward"); PCB_TRY(backward_impl(c, ws, weights_dev, st, split, (!multi && c->early_update) ? &early : nullptr)); }
  PcbNvtxRange r_update("pcb reduce + update");
  // batch log-likelihood into the last slot of the statistics vector, so it is reduced with them
  { PcbProfScope ps(c, st, PCB_K_MISC);
    ll_sum_kernel<<<1, 256, 0, st>>>(c->n_heads ? ws->ll_tmp : ws->mars + (size_t)(c->N - 1) * ws->ld, B,
                                     c->aggr + c->aggr_len - 1); }
  const bool pipe = multi && !split && c->comm_pipe && !c->prof.on && c->n_inner && c->comm_stream;
  if (pipe) {
    // Two collectives on the communication stream, edge statistics first; this stream updates the sum
    // parameters and rebuilds the weight images while the leaf slots are still being summed.
    PCB_CUDA(cudaEventRecord(c->ev_c0, st));
    PCB_CUDA(cudaStreamWaitEvent(c->comm_stream, c->ev_c0, 0));
    PCB_TRY(pcb_allreduce_range(c, 0, c->n_inner, c->comm_stream));
    PCB_CUDA(cudaEventRecord(c->ev_c1, c->comm_stream));
    PCB_TRY(pcb_allreduce_range(c, c->n_inner, c->aggr_len - c->n_inner, c->comm_stream));
    PCB_CUDA(cudaEventRecord(c->ev_c3, c->comm_stream));
    PCB_CUDA(cudaStreamWaitEvent(st, c->ev_c1, 0));
    PCB_TRY(em_update_sums(c, pseudocount, inertia, st));
    if (c->use_tc) PCB_TRY(pcb_dense_tc_refresh(c, st));
    PCB_CUDA(cudaStreamWaitEvent(st, c->ev_c3, 0));
    PCB_TRY(em_update_leaves(c, pseudocount, inertia, st));
    PCB_CUDA(cudaGetLastError());
    return PCB_OK;
  }
  if (split) PCB_TRY(comm_rest_and_join(c, st));
  else if (multi) { PcbProfScope ps(c, st, PCB_K_ALLREDUCE); PCB_TRY(pcb_allreduce_aggr(c, st)); }
  if (early.done) PCB_TRY(em_update_leaves(c, pseudocount, inertia, st));
  else PCB_TRY(pcb_em_update(c, pseudocount, inertia, s));
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

static int32_t em_step_impl(pcb_circuit* c, pcb_workspace* ws, pcb_evidence ev, const float* weights_dev,
                            float clear_rate, float pseudocount, float inertia, float* ll_sum_dev, pcb_stream s) {
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  const uint32_t B = ev.B;
  PCB_REQUIRE(B >= 1 && B <= ws->max_batch, "batch size exceeds the workspace");
  PCB_REQUIRE(!c->n_heads || ev.head_mask_dev, "the flows of a multi-head circuit need a head mask");
  if (c->comm_lost)
    return pcb_fail(PCB_ERR_STATE, "the communicator was aborted: pcb_comm_destroy, then attach a new one or train alone");
  PCB_CUDA(cudaSetDevice(c->device));
  if (c->n_heads && !ws->ll_tmp) PCB_CUDA(cudaMalloc(&ws->ll_tmp, (size_t)ws->max_batch * sizeof(float)));
  const uint8_t* data_dev = ev.data_dev;
  const uint8_t* miss_dev = ev.miss_dev;
  const uint64_t num_rows = ev.num_rows;
  const int32_t* row_ids_dev = ev.row_ids_dev;
  uint32_t row_start = ev.row_start;
  cudaStream_t st = (cudaStream_t)s;
  // the step reads the row ids from the workspace's own buffer, so a replayed graph sees the ids
  // of the current call
  if (row_ids_dev) {
    PCB_CUDA(cudaMemcpyAsync(ws->ids_stage, row_ids_dev, (size_t)B * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
  } else {
    // a row range becomes staged ids too, so that consecutive batches of an epoch replay one graph
    PCB_REQUIRE(row_start >= 1 && (uint64_t)row_start - 1 + B <= num_rows, "row range out of bounds");
    iota_ids_kernel<<<(B + 255) / 256, 256, 0, st>>>(ws->ids_stage, (int32_t)row_start, B);
    row_start = 1;
  }
  row_ids_dev = ws->ids_stage;
  ev.row_ids_dev = row_ids_dev; ev.row_start = row_start;
  if (c->checked) PCB_TRY(pcb_check_batch(c, ev, st));   // before the statistics are cleared
  // The log-likelihood leaves through a copy issued after the step (the update does not touch its
  // slot), outside any captured graph: a training loop hands in a different slot for every batch.
  auto ll_out = [&](cudaStream_t on) -> int32_t {
    if (ll_sum_dev)
      PCB_CUDA(cudaMemcpyAsync(ll_sum_dev, c->aggr + c->aggr_len - 1, sizeof(float), cudaMemcpyDeviceToDevice, on));
    return PCB_OK;
  };
  auto plain = [&]() -> int32_t {
    PCB_TRY(em_step_body(c, ws, ev, weights_dev, clear_rate, pseudocount, inertia, st));
    return ll_out(st);
  };
  if (!c->graph_enabled || c->prof.on || c->checked) return plain();   // checked mode synchronises inside the pass

  pcb_workspace::StepKey key;
  memset(&key, 0, sizeof(key));
  key.data = data_dev; key.miss = miss_dev; key.weights = weights_dev; key.comm = c->comm;
  key.stream = (void*)st; key.num_rows = num_rows; key.row_start = row_start; key.B = B;
  key.clear_rate = clear_rate; key.pseudocount = pseudocount; key.inertia = inertia;
  key.has_ids = row_ids_dev != nullptr; key.w_valid = c->w_img_valid; key.comm_on = c->comm_enabled;
  key.soft = ev.soft_dev; key.head_mask = ev.head_mask_dev; key.soft_reg = ev.soft_reg; key.soft_width = ev.soft_reg_width;

  // the legacy default stream cannot be captured: graphs run on a stream of the circuit's own,
  // ordered after and before the caller's stream with two events
  cudaStream_t gs = st;
  const bool legacy = st == nullptr || st == cudaStreamLegacy;
  if (legacy) {
    if (!c->gstream) {
      PCB_CUDA(cudaStreamCreateWithFlags(&c->gstream, cudaStreamNonBlocking));
      PCB_CUDA(cudaEventCreateWithFlags(&c->ev_g0, cudaEventDisableTiming));
      PCB_CUDA(cudaEventCreateWithFlags(&c->ev_g1, cudaEventDisableTiming));
    }
    gs = c->gstream;
  }
  auto enter = [&]() -> int32_t {
    if (legacy) { PCB_CUDA(cudaEventRecord(c->ev_g0, st)); PCB_CUDA(cudaStreamWaitEvent(gs, c->ev_g0, 0)); }
    return PCB_OK;
  };
  auto leave = [&]() -> int32_t {
    if (legacy) { PCB_CUDA(cudaEventRecord(c->ev_g1, gs)); PCB_CUDA(cudaStreamWaitEvent(st, c->ev_g1, 0)); }
    return PCB_OK;
  };

  if (ws->step_exec && !memcmp(&key, &ws->exec_key, sizeof(key))) {
    // replay; the host-side state is what the captured run left behind
    PCB_TRY(enter());
    PCB_CUDA(cudaGraphLaunch(ws->step_exec, gs));
    PCB_TRY(ll_out(gs));
    PCB_TRY(leave());
    for (int k = 0; k < PCB_K_COUNT; ++k) c->prof.launches[k] += ws->step_launches[k];
    ws->B = B; ws->data = data_dev; ws->miss = miss_dev; ws->num_rows = num_rows;
    ws->row_ids = row_ids_dev; ws->row_start = row_start; ws->have_forward = true;
    ws->soft = ev.soft_dev; ws->head_mask = ev.head_mask_dev;
    ws->soft_reg = ev.soft_dev ? 0.0f : ev.soft_reg; ws->soft_width = ev.soft_reg_width;
    c->w_img_valid = ws->exec_end_w_valid;
    return PCB_OK;
  }
  const bool capture = ws->have_key && !memcmp(&key, &ws->last_key, sizeof(key));
  ws->last_key = key;
  ws->have_key = true;
  if (!capture) return plain();

  if (ws->step_exec) { cudaGraphExecDestroy(ws->step_exec); ws->step_exec = nullptr; }
  uint64_t before[PCB_K_COUNT];
  for (int k = 0; k < PCB_K_COUNT; ++k) before[k] = c->prof.launches[k];
  PCB_TRY(enter());
  PCB_CUDA(cudaStreamBeginCapture(gs, cudaStreamCaptureModeRelaxed));
  int32_t body = em_step_body(c, ws, ev, weights_dev, clear_rate, pseudocount, inertia, gs);
  cudaGraph_t graph = nullptr;
  cudaError_t ce = cudaStreamEndCapture(gs, &graph);
  if (body != PCB_OK || ce != cudaSuccess || !graph) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    c->graph_enabled = false;   // this circuit's step does not capture: stay with plain launches
    if (body != PCB_OK) return body;
    for (int k = 0; k < PCB_K_COUNT; ++k) c->prof.launches[k] = before[k];
    c->w_img_valid = key.w_valid != 0;
    return plain();
  }
  ce = cudaGraphInstantiate(&ws->step_exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ce != cudaSuccess) {
    ws->step_exec = nullptr;
    c->graph_enabled = false;
    for (int k = 0; k < PCB_K_COUNT; ++k) c->prof.launches[k] = before[k];
    c->w_img_valid = key.w_valid != 0;
    cudaGetLastError();
    return plain();
  }
  for (int k = 0; k < PCB_K_COUNT; ++k) ws->step_launches[k] = c->prof.launches[k] - before[k];
  ws->exec_key = key;
  ws->exec_end_w_valid = c->w_img_valid;   // host-side state the captured step ends in
  PCB_CUDA(cudaGraphLaunch(ws->step_exec, gs));
  PCB_TRY(ll_out(gs));
  PCB_TRY(leave());
  return PCB_OK;
}

extern "C" int32_t pcb_em_step(pcb_circuit* c, pcb_workspace* ws, const uint8_t* data_dev,
                               const uint8_t* miss_dev, uint64_t num_rows, const int32_t* row_ids_dev,
                               uint32_t row_start, uint32_t B, const float* weights_dev, float clear_rate,
                               float pseudocount, float inertia, float* ll_sum_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws && data_dev, "null argument");
  return em_step_impl(c, ws, hard_evidence(data_dev, miss_dev, num_rows, row_ids_dev, row_start, B), weights_dev,
                      clear_rate, pseudocount, inertia, ll_sum_dev, s);
}

extern "C" int32_t pcb_em_step_ex(pcb_circuit* c, pcb_workspace* ws, const pcb_evidence* ev, const float* weights_dev,
                                  float clear_rate, float pseudocount, float inertia, float* ll_sum_dev,
                                  pcb_stream s) {
  PCB_REQUIRE(c && ws && ev, "null argument");
  PCB_REQUIRE(ev->data_dev || ev->soft_dev, "null argument");
  return em_step_impl(c, ws, *ev, weights_dev, clear_rate, pseudocount, inertia, ll_sum_dev, s);
}

static int32_t get_matrix(pcb_circuit* c, pcb_workspace* ws, const float* src, float* host, uint64_t n) {
  PCB_REQUIRE(c && ws && host, "null argument");
  PCB_REQUIRE(ws->have_forward, "no batch has been evaluated on this workspace");
  PCB_REQUIRE(n == (uint64_t)ws->B * c->N, "matrix has the wrong size");
  PCB_CUDA(cudaSetDevice(c->device));
  PCB_CUDA(cudaDeviceSynchronize());
  PCB_TRY(pcb_check_status(c));
  PCB_CUDA(cudaMemcpy2D(host, ws->B * sizeof(float), src, ws->ld * sizeof(float), ws->B * sizeof(float), c->N,
                        cudaMemcpyDeviceToHost));
  return PCB_OK;
}
extern "C" int32_t pcb_get_mars(pcb_circuit* c, pcb_workspace* ws, float* mars_host, uint64_t n) {
  return get_matrix(c, ws, ws ? ws->mars : nullptr, mars_host, n);
}
extern "C" int32_t pcb_get_flows(pcb_circuit* c, pcb_workspace* ws, float* flows_host, uint64_t n) {
  return get_matrix(c, ws, ws ? ws->flows : nullptr, flows_host, n);
}
