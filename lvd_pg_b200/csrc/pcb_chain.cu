// pcb_chain.cu — one step of a forward or backward pass in one launch, dense blocks in fp32.
//
// Reference kernels replaced (paths relative to VariationalJuice.jl/src): layer_up_kernel
// (queries/likelihood.jl:4-68), layer_down_kernel / reg_layer_down_kernel (queries/flow.jl:8-106,
// regularization/reg_flow.jl:120-222).
//
// A pass is a chain of dependent steps, most of them a handful of blocks: what such a step costs is latency, not
// arithmetic (a tensor-core tile of pcb_dense_mn.cu takes 8 - 15 us from launch to last store, most of it set-up,
// the staging of split operands, barriers and the drain of the accumulator).  The kernels here are built for that:
//   * everything of a step is one launch: the dense blocks, the products under them (their values are formed from the
//     nodes they multiply and their flows handed on to those, so a product layer is no step of its own) and the
//     nodes that are taken one by one;
//   * what does not depend on the step before (weights; on the way down also the node values) is fetched before the
//     wait on the preceding launch (programmatic stream serialization);
//   * a CTA takes 32 examples x 64 rows (children on the way down) of a block, values and weights in shared memory as
//     they are, and multiplies with mma.sync (m16n8k8, TF32 hi / lo split in registers, three passes as in
//     pcb_dense_mn.cu): no descriptors, barriers or tensor memory between the values and the result.  Register tiles
//     of FMAs are bound by shared-memory reads here: 4 x 4 outputs per thread reached 1.2e13 multiply-adds per
//     second (one block of 256 x 256 at 2048 examples 25 us, against 13 us this way).
// Bound: the launch-to-launch latency of a step (3 - 5 us) until the tensor pipe of the mma.sync path fills;
// pcb_chain_takes has the rule.
#include <algorithm>

#include "pcb_internal.h"
#include "pcb_sparse.cuh"

namespace {

constexpr uint32_t TPB = 256;    // threads: 8 example quads x 32 rows while values are fetched, 4 x 2 warp tiles of 16 x 16 outputs
constexpr uint32_t EX = 32;      // examples of a tile
constexpr uint32_t OUT = 64;     // rows (upward) or children (downward) of a CTA
constexpr uint32_t MAX_DIM = 512;
constexpr uint32_t RSTEP = TPB / 8;
constexpr uint32_t XP = EX + 8;  // pitch of the value tile and of the weights on the way down: the four rows and eight
constexpr uint32_t WPD = OUT + 8;   // columns that the lanes of an operand fragment read lie in 32 different banks
// 96 latents at 1024 examples 654 (tensor-core kernel) against 682 us a step, 128 at 2048 1134 against 1228 us
constexpr uint32_t EDGE_NARROW_DIM = 64;
constexpr uint32_t SPARSE = 128; // threads on one node outside the blocks: 512 examples

struct ChainArgs {
  float* mars;
  float* flows;
  float* blk_mx;
  const float* theta;
  const PcbDenseBlock* blk;   // dense blocks of the step
  const PcbDenseBlock* thin;  // upward: single sum nodes over consecutive children
  const uint32_t* src_list;
  uint32_t ld, nblk, nthin, tiles, tile_ctas, chunks, dense_ctas, sparse_tiles;
  const uint32_t* nodes;      // nodes taken one by one
  uint32_t n_nodes;
};

__device__ __forceinline__ float4 ld4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 max4(float4 a, float4 b) {
  return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
}
__device__ __forceinline__ float4 exp4(float4 v, float4 m) {   // exp(v - m)
  return make_float4(__expf(v.x - m.x), __expf(v.y - m.y), __expf(v.z - m.z), __expf(v.w - m.w));
}
__device__ __forceinline__ float4 exp4_below(float4 mx, float4 v) {
  return make_float4(pcb_exp_below(mx.x, v.x), pcb_exp_below(mx.y, v.y), pcb_exp_below(mx.z, v.z), pcb_exp_below(mx.w, v.w));
}
__device__ __forceinline__ float4 splat(float v) { return make_float4(v, v, v, v); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

// exp of `rows` x `cols` weights (row pitch `pitch` in theta) into shared memory (row pitch `sp`), zeros up to
// `rows_to` x `cols_to`; complete for this thread's own elements on return
__device__ __forceinline__ void stage_weights(float* w, const float* theta, uint32_t rows, uint32_t cols, size_t pitch,
                                              uint32_t rows_to, uint32_t cols_to, uint32_t sp) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // 16-byte copies where the rows allow it (64 latents and a first parameter that is a multiple of four do)
  const bool quads = ((reinterpret_cast<uintptr_t>(theta) & 15) | (pitch & 3) | (cols & 3)) == 0;
  if (quads) {
    for (uint32_t r = warp; r < rows; r += TPB / 32)
      for (uint32_t t = lane * 4; t < cols; t += 128) pcb_copy16_async(w + r * sp + t, theta + (size_t)r * pitch + t);
  } else {
    for (uint32_t r = warp; r < rows; r += TPB / 32)
      for (uint32_t t = lane; t < cols; t += 32) pcb_copy4_async(w + r * sp + t, theta + (size_t)r * pitch + t);
  }
  for (uint32_t r = warp; r < rows_to; r += TPB / 32)
    for (uint32_t t = (r < rows ? cols : 0) + lane; t < cols_to; t += 32) w[r * sp + t] = 0.0f;
  pcb_copies_wait();
  if (quads) {
    for (uint32_t r = warp; r < rows; r += TPB / 32)
      for (uint32_t t = lane * 4; t < cols; t += 128) {
        float* const p = w + r * sp + t;
        st4(p, exp4(*reinterpret_cast<const float4*>(p), splat(0.0f)));
      }
  } else {
    for (uint32_t r = warp; r < rows; r += TPB / 32)
      for (uint32_t t = lane; t < cols; t += 32) w[r * sp + t] = __expf(w[r * sp + t]);
  }
}

// D += A * B for a 16 x 8 piece of outputs and 8 values of the contraction, fp32 operands split as they are used:
// v = hi + lo with hi the top 19 bits, hi * hi + lo * hi + hi * lo
struct Frag4 { uint32_t hi[4], lo[4]; };
__device__ __forceinline__ void split(float v, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(v) & 0xffffe000u;
  lo = __float_as_uint(v - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// this warp's 16 x 16 outputs: rows m0 .. m0 + 15 of the weights, examples e0 .. e0 + 15 of the values.  Weight (m, k)
// lies at w[m * wm + k * wk], value (k, e) at x[k * XP + e]; kdim is a multiple of 8.
__device__ __forceinline__ void contract(float (&acc)[2][4], const float* w, uint32_t wm, uint32_t wk, const float* x,
                                         uint32_t kdim, uint32_t m0, uint32_t e0) {
  const uint32_t lane = threadIdx.x & 31, hi8 = lane >> 2, lo4 = lane & 3;
  const float* wp = w + (m0 + hi8) * wm + lo4 * wk;
  const float* xp = x + lo4 * XP + e0 + hi8;
#pragma unroll 4
  for (uint32_t k = 0; k < kdim; k += 8) {
    Frag4 a;
    split(wp[k * wk], a.hi[0], a.lo[0]);
    split(wp[8 * wm + k * wk], a.hi[1], a.lo[1]);
    split(wp[(k + 4) * wk], a.hi[2], a.lo[2]);
    split(wp[8 * wm + (k + 4) * wk], a.hi[3], a.lo[3]);
    uint32_t bh[2][2], bl[2][2];
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) {
      split(xp[k * XP + 8 * j], bh[j][0], bl[j][0]);
      split(xp[(k + 4) * XP + 8 * j], bh[j][1], bl[j][1]);
    }
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) mma_tf32(acc[j], a.lo, bh[j][0], bh[j][1]);
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) mma_tf32(acc[j], a.hi, bl[j][0], bl[j][1]);
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) mma_tf32(acc[j], a.hi, bh[j][0], bh[j][1]);
  }
}

// the maximum / sum over the rows of a tile's example quads: over the four rows of a warp, then over the warps
template <typename Op>
__device__ __forceinline__ float4 over_rows(float4 v, float4 (&red)[TPB / 32][8], Op op) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (uint32_t o = 8; o < 32; o <<= 1)
    v = op(v, make_float4(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o),
                          __shfl_xor_sync(0xffffffffu, v.z, o), __shfl_xor_sync(0xffffffffu, v.w, o)));
  __syncthreads();   // what `red` held has been read
  if (lane < 8) red[warp][lane] = v;
  __syncthreads();
  v = red[0][lane & 7];
#pragma unroll
  for (uint32_t u = 1; u < TPB / 32; ++u) v = op(v, red[u][lane & 7]);
  return v;
}

// A single sum node over consecutive children (the root, so the likelihood itself): in fp32 and with the weights inside
// the maximum, as the kernel of single nodes sums it, so that children far below one without weight count in full.
template <uint32_t BATCH>
__device__ __forceinline__ void up_single(const ChainArgs& a, const PcbDenseBlock& k, float* w, float4 (&red)[TPB / 32][8]) {
  const uint32_t q = threadIdx.x & 7, g = threadIdx.x >> 3, ld = a.ld, K = k.K;
  float* const x = w + ((K + 3u) & ~3u);   // [K][XP]
  for (uint32_t t = threadIdx.x; t < K; t += TPB) w[t] = a.theta[k.pid0 + t];
  __syncthreads();
  pcb_grid_dep_wait();   // everything above is the step's parameters
  for (uint32_t tile = blockIdx.x % a.tile_ctas; tile < a.tiles; tile += a.tile_ctas) {
    const uint32_t b = tile * EX + q * 4;
    const float* const pa = a.mars + (size_t)k.c0 * ld + b;
    const float* const pb = a.mars + (size_t)(k.d0 != PCB_NONE ? k.d0 : k.c0) * ld + b;
    float4 mx = splat(-INFINITY);
#pragma unroll BATCH
    for (uint32_t t = g; t < K; t += RSTEP) {
      float4 v = ld4(pa + (size_t)t * ld);
      if (k.d0 != PCB_NONE) v = add4(v, ld4(pb + (size_t)t * ld));
      v = add4(v, splat(w[t]));
      mx = max4(mx, v);
      st4(x + t * XP + q * 4, v);
    }
    mx = over_rows(mx, red, [](float4 u, float4 v) { return max4(u, v); });
    float4 s = splat(0.0f);   // an example for which no child is possible: NaN here, -inf below
    for (uint32_t t = g; t < K; t += RSTEP) s = add4(s, exp4(*reinterpret_cast<const float4*>(x + t * XP + q * 4), mx));
    s = over_rows(s, red, [](float4 u, float4 v) { return add4(u, v); });
    if (g == 0)
      st4(a.mars + (size_t)k.p0 * ld + b,
          make_float4(mx.x == -INFINITY ? -INFINITY : __logf(s.x) + mx.x, mx.y == -INFINITY ? -INFINITY : __logf(s.y) + mx.y,
                      mx.z == -INFINITY ? -INFINITY : __logf(s.z) + mx.z, mx.w == -INFINITY ? -INFINITY : __logf(s.w) + mx.w));
  }
}

// mars[r][b] = log(sum_t exp(theta[r][t]) * exp(M[t][b] - mx[b])) + mx[b], M = prime + sub, mx the maximum over t.
// A CTA walks the example tiles tile0, tile0 + tile_ctas, ... with its weights in place; the first rows of the next tile
// are fetched while this one is multiplied.  BATCH: rows per thread whose loads are in flight together.
template <uint32_t BATCH>
__global__ void __launch_bounds__(TPB, BATCH <= 2 ? 4 : 2) chain_up_kernel(ChainArgs a, PcbSparseUp sp) {
  extern __shared__ float4 chain_smem[];
  __shared__ float4 red[TPB / 32][8];
  __shared__ float mxs[EX];
  __shared__ uint32_t src[PCB_MAX_SOURCES + 1];
  pcb_grid_dep_launch();
  if (blockIdx.x >= a.dense_ctas) {
    const uint32_t i = (blockIdx.x - a.dense_ctas) * (TPB / SPARSE) + threadIdx.x / SPARSE;
    if (i < a.n_nodes * a.sparse_tiles)
      pcb_sparse_up_node(sp, a.nodes[i / a.sparse_tiles], (i % a.sparse_tiles * SPARSE + threadIdx.x % SPARSE) * 4u);
    return;
  }
  const uint32_t rest = blockIdx.x / a.tile_ctas, bi = rest / a.chunks, r0 = rest % a.chunks * OUT;
  const PcbDenseBlock k = bi < a.nblk ? a.blk[bi] : a.thin[bi - a.nblk];
  if (r0 >= k.R) return;
  if (bi >= a.nblk) {
    up_single<BATCH>(a, k, reinterpret_cast<float*>(chain_smem), red);
    return;
  }
  const uint32_t rows = min(OUT, k.R - r0), K = k.K, K8 = (K + 7u) & ~7u, wp = K8 + 4u, ld = a.ld;
  float* const w = reinterpret_cast<float*>(chain_smem);   // [OUT][wp]
  float* const x = w + OUT * wp;                           // [K8][XP]
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = threadIdx.x & 7, g = threadIdx.x >> 3;
  const uint32_t nsrc = k.src != PCB_NONE ? a.src_list[k.src] : 0;
  if (threadIdx.x < nsrc) src[threadIdx.x] = a.src_list[k.src + 1 + threadIdx.x];
  stage_weights(w, a.theta + k.pid0 + (size_t)r0 * K, rows, K, K, OUT, K8, wp);
  for (uint32_t t = K + warp; t < K8; t += TPB / 32) x[t * XP + lane] = 0.0f;
  __syncthreads();
  const float* const pa = a.mars + (size_t)(nsrc ? src[0] : k.c0) * ld;
  const float* const pb = k.d0 != PCB_NONE ? a.mars + (size_t)k.d0 * ld : nullptr;
  const float* const pc = nsrc > 1 ? a.mars + (size_t)src[1] * ld : nullptr;
  float4 v[BATCH], y[BATCH], z[BATCH];   // the first three addends of a batch of rows: in flight together
  auto fetch = [&](uint32_t tile, uint32_t t0) {
    const uint32_t b = tile * EX + q * 4;
#pragma unroll
    for (uint32_t u = 0; u < BATCH; ++u) {
      const size_t at = (size_t)(t0 + RSTEP * u) * ld + b;
      const bool in = t0 + RSTEP * u < K;
      v[u] = in ? ld4(pa + at) : splat(0.0f);
      y[u] = in && pb ? ld4(pb + at) : splat(0.0f);
      z[u] = in && pc ? ld4(pc + at) : splat(0.0f);
    }
  };
  pcb_grid_dep_wait();   // everything above is static circuit data or the step's parameters
  fetch(blockIdx.x % a.tile_ctas, g);
  for (uint32_t tile = blockIdx.x % a.tile_ctas; tile < a.tiles; tile += a.tile_ctas) {
    const uint32_t b = tile * EX + q * 4;
    float4 mx = splat(-INFINITY);
    for (uint32_t t0 = g; t0 < K; t0 += RSTEP * BATCH) {
      if (t0 != g) fetch(tile, t0);
      if (nsrc) {
#pragma unroll
        for (uint32_t u = 0; u < BATCH; ++u) v[u] = add4(v[u], z[u]);
#pragma unroll 2
        for (uint32_t s = 2; s < nsrc; ++s) {
          const float* const ps = a.mars + (size_t)src[s] * ld + b;
#pragma unroll
          for (uint32_t u = 0; u < BATCH; ++u)
            if (t0 + RSTEP * u < K) v[u] = add4(v[u], ld4(ps + (size_t)(t0 + RSTEP * u) * ld));
        }
        if (r0 == 0)   // the products' own values: the statistics and the way down read them
#pragma unroll
          for (uint32_t u = 0; u < BATCH; ++u)
            if (t0 + RSTEP * u < K) st4(a.mars + (size_t)(k.c0 + t0 + RSTEP * u) * ld + b, v[u]);
      }
#pragma unroll
      for (uint32_t u = 0; u < BATCH; ++u)
        if (t0 + RSTEP * u < K) {
          v[u] = add4(v[u], y[u]);
          mx = max4(mx, v[u]);
          st4(x + (t0 + RSTEP * u) * XP + q * 4, v[u]);
        }
    }
    if (tile + a.tile_ctas < a.tiles) fetch(tile + a.tile_ctas, g);
#pragma unroll
    for (uint32_t o = 8; o < 32; o <<= 1)
      mx = max4(mx, make_float4(__shfl_xor_sync(0xffffffffu, mx.x, o), __shfl_xor_sync(0xffffffffu, mx.y, o),
                                __shfl_xor_sync(0xffffffffu, mx.z, o), __shfl_xor_sync(0xffffffffu, mx.w, o)));
    if (lane < 8) red[warp][lane] = mx;
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < TPB / 32; ++u) mx = max4(mx, red[u][q]);
    if (g == 0) {
      st4(mxs + q * 4, mx);
      if (r0 == 0) st4(a.blk_mx + (size_t)k.mx_row * ld + b, mx);
    }
    // an example for which no child is possible: exp(x - inf) = 0
    const float4 sh = make_float4(mx.x == -INFINITY ? INFINITY : mx.x, mx.y == -INFINITY ? INFINITY : mx.y,
                                  mx.z == -INFINITY ? INFINITY : mx.z, mx.w == -INFINITY ? INFINITY : mx.w);
    for (uint32_t t = g; t < K; t += RSTEP) {
      float* const p = x + t * XP + q * 4;
      st4(p, exp4(*reinterpret_cast<const float4*>(p), sh));
    }
    __syncthreads();
    const uint32_t m0 = (warp & 3u) * 16, e0 = (warp >> 2) * 16;
    if (m0 < rows) {
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      contract(acc, w, wp, 1, x, K8, m0, e0);
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j) {
        const uint32_t e = e0 + 8 * j + 2 * (lane & 3u);
        const float2 m = *reinterpret_cast<const float2*>(mxs + e);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t r = m0 + (lane >> 2) + 8 * h;
          if (r < rows)
            *reinterpret_cast<float2*>(a.mars + (size_t)(k.p0 + r0 + r) * ld + tile * EX + e) =
                make_float2(m.x == -INFINITY ? -INFINITY : __logf(acc[j][2 * h]) + m.x,
                            m.y == -INFINITY ? -INFINITY : __logf(acc[j][2 * h + 1]) + m.y);
        }
      }
    }
    if (tile + a.tile_ctas < a.tiles) __syncthreads();   // the next tile's values replace these
  }
}

// flows[t][b] = exp(M[t][b] - mx[b]) * sum_r exp(theta[r][t]) * flows[r][b] * exp(mx[b] - mars[r][b]) for prime and sub
// child t, and for every node that a fused product t multiplies.
template <uint32_t BATCH>
__global__ void __launch_bounds__(TPB, BATCH <= 2 ? 4 : 2) chain_down_kernel(ChainArgs a, PcbSparseDown sp) {
  extern __shared__ float4 chain_smem[];
  __shared__ uint32_t src[PCB_MAX_SOURCES + 1];
  pcb_grid_dep_launch();
  if (blockIdx.x >= a.dense_ctas) {
    const uint32_t i = (blockIdx.x - a.dense_ctas) * (TPB / SPARSE) + threadIdx.x / SPARSE;
    if (i < a.n_nodes * a.sparse_tiles)
      pcb_sparse_down_node(sp, a.nodes[i / a.sparse_tiles], (i % a.sparse_tiles * SPARSE + threadIdx.x % SPARSE) * 4u);
    return;
  }
  const uint32_t rest = blockIdx.x / a.tile_ctas, t0 = rest % a.chunks * OUT;
  const PcbDenseBlock k = a.blk[rest / a.chunks];
  if (t0 >= k.K) return;
  const uint32_t cols = min(OUT, k.K - t0), R = k.R, R8 = (R + 7u) & ~7u, ld = a.ld;
  float* const w = reinterpret_cast<float*>(chain_smem);   // [R8][WPD]
  float* const y = w + R8 * WPD;                           // [R8][XP]
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = threadIdx.x & 7, g = threadIdx.x >> 3;
  const uint32_t nsrc = k.src != PCB_NONE ? a.src_list[k.src] : 0;
  if (threadIdx.x < nsrc) src[threadIdx.x] = a.src_list[k.src + 1 + threadIdx.x];
  stage_weights(w, a.theta + k.pid0 + t0, R, cols, k.K, R8, OUT, WPD);
  for (uint32_t r = R + warp; r < R8; r += TPB / 32) y[r * XP + lane] = 0.0f;
  const uint32_t m0 = (warp & 3u) * 16, e0 = (warp >> 2) * 16, tr = m0 + (lane >> 2), te = e0 + 2 * (lane & 3u);
  bool waited = false;
  for (uint32_t tile = blockIdx.x % a.tile_ctas; tile < a.tiles; tile += a.tile_ctas) {
    const uint32_t b = tile * EX + q * 4;
    // node values are final since the forward pass: fetched ahead of the wait
    const float* const mxrow = a.blk_mx + (size_t)k.mx_row * ld;
    const float4 mx = ld4(mxrow + b);
    for (uint32_t r1 = g; r1 < R; r1 += RSTEP * BATCH) {
      float4 v[BATCH];
#pragma unroll
      for (uint32_t u = 0; u < BATCH; ++u) v[u] = r1 + RSTEP * u < R ? ld4(a.mars + (size_t)(k.p0 + r1 + RSTEP * u) * ld + b) : splat(0.0f);
#pragma unroll
      for (uint32_t u = 0; u < BATCH; ++u)
        if (r1 + RSTEP * u < R) st4(y + (r1 + RSTEP * u) * XP + q * 4, exp4_below(mx, v[u]));
    }
    float2 xv[2][2];   // exp(M - mx) of this thread's outputs: [examples 8 j][children 8 h]
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) {
      const size_t at = (size_t)tile * EX + te + 8 * j;
      const float2 m = __ldcg(reinterpret_cast<const float2*>(mxrow + at));
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        xv[j][h] = make_float2(0.0f, 0.0f);
        if (tr + 8 * h < cols) {
          float2 c = __ldcg(reinterpret_cast<const float2*>(a.mars + (size_t)(k.c0 + t0 + tr + 8 * h) * ld + at));
          if (k.d0 != PCB_NONE) {
            const float2 d = __ldcg(reinterpret_cast<const float2*>(a.mars + (size_t)(k.d0 + t0 + tr + 8 * h) * ld + at));
            c.x += d.x; c.y += d.y;
          }
          xv[j][h] = make_float2(m.x == -INFINITY ? 0.0f : __expf(c.x - m.x), m.y == -INFINITY ? 0.0f : __expf(c.y - m.y));
        }
      }
    }
    if (!waited) { pcb_grid_dep_wait(); waited = true; }
    for (uint32_t r1 = g; r1 < R; r1 += RSTEP * BATCH) {
      float4 v[BATCH];
#pragma unroll
      for (uint32_t u = 0; u < BATCH; ++u) v[u] = r1 + RSTEP * u < R ? ld4(a.flows + (size_t)(k.p0 + r1 + RSTEP * u) * ld + b) : splat(0.0f);
#pragma unroll
      for (uint32_t u = 0; u < BATCH; ++u)
        if (r1 + RSTEP * u < R) {
          float* const p = y + (r1 + RSTEP * u) * XP + q * 4;
          const float4 e = *reinterpret_cast<const float4*>(p);
          st4(p, make_float4(v[u].x * e.x, v[u].y * e.y, v[u].z * e.z, v[u].w * e.w));
        }
    }
    __syncthreads();
    if (m0 < cols) {
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      contract(acc, w, 1, WPD, y, R8, m0, e0);
#pragma unroll
      for (uint32_t j = 0; j < 2; ++j)
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t t = t0 + tr + 8 * h;
          if (tr + 8 * h >= cols) continue;
          // a masked example keeps 0 whatever the accumulator holds
          const float2 f = make_float2(xv[j][h].x == 0.0f ? 0.0f : acc[j][2 * h] * xv[j][h].x,
                                       xv[j][h].y == 0.0f ? 0.0f : acc[j][2 * h + 1] * xv[j][h].y);
          const size_t at = (size_t)tile * EX + te + 8 * j;
          auto put = [&](uint32_t n) { *reinterpret_cast<float2*>(a.flows + (size_t)n * ld + at) = f; };
          put(k.c0 + t);
          if (k.d0 != PCB_NONE) put(k.d0 + t);
          for (uint32_t s = 0; s < nsrc; ++s) put(src[s] + t);
        }
    }
    if (tile + a.tile_ctas < a.tiles) __syncthreads();
  }
}

// Edge statistics of narrow blocks: aggr[r][t] += exp(theta[r][t]) * sum_b G[r][b] X[t][b] with
// G = flows[r] * exp(mx - mars[r]), X = exp(M[t] - mx).  pcb_dense_edge.cu works in tiles of 128 x 256 outputs, of which
// a block of 32 latents fills a thirtieth; here a CTA owns 64 x 64 outputs of one block in registers (mma.sync, operands
// as above) and walks its share of the examples in tiles of 32, the rows of the next tile in flight.  Bound: HBM (four
// rows per latent and example).  2159 blocks of 32 x 32 at 512 examples: 576 -> 317 us beside the chain, 233 us alone.
constexpr uint32_t EP = EX + 4;   // pitch of both operand tiles: eight rows x four examples of a fragment in 32 banks
__global__ void __launch_bounds__(TPB, 2) edge_narrow_kernel(
    const float* __restrict__ mars, const float* __restrict__ flows, const float* __restrict__ blk_mx,
    const float* __restrict__ theta, float* __restrict__ aggr, const PcbDenseBlock* __restrict__ blocks, uint32_t ld, uint32_t B,
    uint32_t rchunks, uint32_t cchunks, uint32_t slices) {
  __shared__ __align__(16) float gs[2][OUT * EP], xs[2][OUT * EP];
  const uint32_t slice = blockIdx.x % slices, c2 = blockIdx.x / slices % cchunks, rest = blockIdx.x / (slices * cchunks);
  const PcbDenseBlock k = blocks[rest / rchunks];
  const uint32_t r0 = rest % rchunks * OUT, t0 = c2 * OUT;
  if (r0 >= k.R || t0 >= k.K) return;
  const uint32_t rows = min(OUT, k.R - r0), cols = min(OUT, k.K - t0);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = threadIdx.x & 7, g = threadIdx.x >> 3;
  const uint32_t tiles = (B + EX - 1) / EX;
  const float* const mxrow = blk_mx + (size_t)k.mx_row * ld;
  float4 pm[2], pf[2], mc[2], md[2], mx;
  auto fetch = [&](uint32_t tile) {
    const uint32_t b = tile * EX + q * 4;
    mx = ld4(mxrow + b);
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const uint32_t r = g + 32 * u;
      if (r < rows) { pm[u] = ld4(mars + (size_t)(k.p0 + r0 + r) * ld + b); pf[u] = ld4(flows + (size_t)(k.p0 + r0 + r) * ld + b); }
      if (r < cols) {
        mc[u] = ld4(mars + (size_t)(k.c0 + t0 + r) * ld + b);
        md[u] = k.d0 != PCB_NONE ? ld4(mars + (size_t)(k.d0 + t0 + r) * ld + b) : splat(0.0f);
      }
    }
  };
  float acc[4][4];
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) acc[j][e] = 0.0f;
  const uint32_t m0 = (warp & 3u) * 16, n0 = (warp >> 2) * 32, hi8 = lane >> 2, lo4 = lane & 3;
  uint32_t buf = 0;
  if (slice < tiles) fetch(slice);
  for (uint32_t tile = slice; tile < tiles; tile += slices, buf ^= 1u) {
    const uint32_t b = tile * EX + q * 4;
    // examples past the batch and examples without a possible child count nowhere
    const bool v0 = b < B && mx.x != -INFINITY, v1 = b + 1 < B && mx.y != -INFINITY, v2 = b + 2 < B && mx.z != -INFINITY,
               v3 = b + 3 < B && mx.w != -INFINITY;
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const uint32_t r = g + 32 * u;
      float4 y = splat(0.0f), x = splat(0.0f);
      if (r < rows) {
        const float4 e = exp4_below(mx, pm[u]);
        y = make_float4(v0 ? pf[u].x * e.x : 0.f, v1 ? pf[u].y * e.y : 0.f, v2 ? pf[u].z * e.z : 0.f, v3 ? pf[u].w * e.w : 0.f);
      }
      if (r < cols) {
        const float4 e = exp4(add4(mc[u], md[u]), mx);
        x = make_float4(v0 ? e.x : 0.f, v1 ? e.y : 0.f, v2 ? e.z : 0.f, v3 ? e.w : 0.f);
      }
      st4(&gs[buf][r * EP + q * 4], y);
      st4(&xs[buf][r * EP + q * 4], x);
    }
    if (tile + slices < tiles) fetch(tile + slices);
    __syncthreads();   // two buffers: a warp that is ahead writes the other one
    if (m0 < rows && n0 < cols) {
      const float* const gp = &gs[buf][(m0 + hi8) * EP + lo4];
      const float* const xp = &xs[buf][(n0 + hi8) * EP + lo4];
#pragma unroll
      for (uint32_t e = 0; e < EX; e += 8) {
        Frag4 a;
        split(gp[e], a.hi[0], a.lo[0]);
        split(gp[8 * EP + e], a.hi[1], a.lo[1]);
        split(gp[e + 4], a.hi[2], a.lo[2]);
        split(gp[8 * EP + e + 4], a.hi[3], a.lo[3]);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
          uint32_t bh[2], bl[2];
          split(xp[8 * j * EP + e], bh[0], bl[0]);
          split(xp[8 * j * EP + e + 4], bh[1], bl[1]);
          mma_tf32(acc[j], a.lo, bh[0], bh[1]);
          mma_tf32(acc[j], a.hi, bl[0], bl[1]);
          mma_tf32(acc[j], a.hi, bh[0], bh[1]);
        }
      }
    }
  }
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
      const uint32_t r = m0 + hi8 + 8 * (e >> 1), t = n0 + 8 * j + 2 * lo4 + (e & 1u);
      if (r < rows && t < cols) {
        const size_t p = k.pid0 + (size_t)(r0 + r) * k.K + t0 + t;
        atomicAdd(aggr + p, __expf(__ldg(theta + p)) * acc[j][e]);
      }
    }
}

// Example tiles shared out over CTAs so that a launch stays about one wave: a CTA keeps its weights over its tiles.
// `per_tile` CTAs take one tile each; `smem` and `most` (registers) bound the CTAs of an SM.
uint32_t tile_ctas(uint32_t tiles, uint32_t per_tile, size_t smem, uint32_t most) {
  const uint32_t fit = 148 * (uint32_t)std::min<size_t>(most, std::max<size_t>(1, 227 * 1024 / (smem + 2048)));
  const uint32_t n = std::max(1u, std::min(tiles, fit / std::max(1u, per_tile)));
  const uint32_t rounds = (tiles + n - 1) / n;
  return (tiles + rounds - 1) / rounds;   // the same number of rounds with no more CTAs
}

}  // namespace

#define PCB_TRY(expr)              \
  do {                             \
    int32_t _s = (expr);           \
    if (_s != PCB_OK) return _s;   \
  } while (0)

// Which path takes a step.  Up to 64 latents a tensor-core tile of 128 x 256 is mostly padding and set-up: the chain
// kernels win at every batch (training step of a 784-variable circuit with 64 latents: 512 examples 1291 -> 1126 us,
// 2048 examples 3703 -> 3542 us).  Above that the line is where a step's multiply-adds at the mma.sync rate (1e13 per
// second) catch up with what the tensor-core kernels take for any small step (15 - 20 us): 2e8.  192 variables x 128
// latents: 512 examples 1378 -> 791 us, 2048 examples 2501 -> 2121 us (2330 us with the line at 1e8, 2238 us without
// one); 256 latents at 1024 examples 2687 -> 2484 us (3430 us without one).  A step without dense blocks always runs here.
bool pcb_chain_takes(const pcb_circuit* c, const pcb_workspace* ws, uint32_t step) {
  const uint32_t o0 = c->h_dense_off[step], o1 = c->h_dense_off[step + 1];
  if (!c->chain) return false;
  uint64_t macs = 0;
  uint32_t dim = 0;
  for (uint32_t i = o0; i < o1; ++i) {
    const PcbDenseBlock& b = c->h_dense[i];
    macs += (uint64_t)b.R * b.K * ws->B;
    dim = std::max(dim, std::max(b.R, b.K));
  }
  for (uint32_t i = c->h_st_thin_off[step]; i < c->h_st_thin_off[step + 1]; ++i) dim = std::max(dim, c->h_thin[i].K);
  if (dim > MAX_DIM) return false;
  const uint64_t limit = c->chain_macs ? c->chain_macs : dim <= 64 ? ~0ull : 200000000ull;
  return macs <= limit;
}

int32_t pcb_chain_forward(pcb_circuit* c, pcb_workspace* ws, uint32_t step, cudaStream_t st) {
  const uint32_t o0 = c->h_dense_off[step], o1 = c->h_dense_off[step + 1];
  const uint32_t h0 = c->h_st_thin_off[step], h1 = c->h_st_thin_off[step + 1];
  const uint32_t u0 = c->h_st_up_off[step], loose = c->h_st_up_off[step + 1] - u0 - (h1 - h0);
  ChainArgs a;
  a.mars = ws->mars; a.flows = nullptr; a.blk_mx = ws->blk_mx; a.theta = c->theta; a.blk = c->dense + o0; a.thin = c->thin + h0;
  a.src_list = c->src_list; a.ld = ws->ld; a.nblk = o1 - o0; a.nthin = h1 - h0; a.nodes = c->st_up + u0; a.n_nodes = loose;
  uint32_t R = 1, K = 1;
  for (uint32_t i = o0; i < o1; ++i) { R = std::max(R, c->h_dense[i].R); K = std::max(K, c->h_dense[i].K); }
  for (uint32_t i = h0; i < h1; ++i) K = std::max(K, c->h_thin[i].K);
  const uint32_t blocks = a.nblk + a.nthin;
  a.tiles = (ws->B + EX - 1) / EX;
  a.chunks = (R + OUT - 1) / OUT;
  const uint32_t K8 = pcb_round_up(K, 8);
  const size_t smem = blocks ? ((size_t)OUT * (K8 + 4) + (size_t)K8 * XP) * sizeof(float) : 0;
  a.tile_ctas = tile_ctas(a.tiles, blocks * a.chunks, smem, K <= 2 * RSTEP ? 4 : 2);
  a.dense_ctas = blocks * a.chunks * a.tile_ctas;
  a.sparse_tiles = (ws->B + 4 * SPARSE - 1) / (4 * SPARSE);
  const uint32_t sparse_ctas = (loose * a.sparse_tiles + TPB / SPARSE - 1) / (TPB / SPARSE);
  const uint32_t grid = a.dense_ctas + sparse_ctas;
  if (!grid) return PCB_OK;
  static PcbPerDeviceOnce once;
  PCB_CUDA(once.run([] {
    for (auto kernel : {chain_up_kernel<1>, chain_up_kernel<2>, chain_up_kernel<4>}) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)((OUT * (MAX_DIM + 4) + MAX_DIM * XP) * sizeof(float)));
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }));
  PcbProfScope ps(c, st, a.nblk ? PCB_K_DENSE_FWD : PCB_K_SPARSE_UP);
  auto kernel = K <= RSTEP ? chain_up_kernel<1> : K <= 2 * RSTEP ? chain_up_kernel<2> : chain_up_kernel<4>;
  PCB_CUDA(pcb_launch_pdl(kernel, dim3(grid), dim3(TPB), smem, st, c->pdl, a, pcb_sparse_up_args(c, ws)));
  return PCB_OK;
}

int32_t pcb_chain_backward(pcb_circuit* c, pcb_workspace* ws, uint32_t step, const PcbHeadInit& hi, cudaStream_t st) {
  const uint32_t o0 = c->h_dense_off[step], o1 = c->h_dense_off[step + 1];
  const uint32_t d0 = c->h_st_down_off[step - 1], loose = c->h_st_down_off[step] - d0;
  ChainArgs a;
  a.mars = ws->mars; a.flows = ws->flows; a.blk_mx = ws->blk_mx; a.theta = c->theta; a.blk = c->dense + o0; a.thin = nullptr;
  a.src_list = c->src_list; a.ld = ws->ld; a.nblk = o1 - o0; a.nthin = 0; a.nodes = c->st_down + d0; a.n_nodes = loose;
  uint32_t R = 1, K = 1;
  for (uint32_t i = o0; i < o1; ++i) { R = std::max(R, c->h_dense[i].R); K = std::max(K, c->h_dense[i].K); }
  a.tiles = (ws->B + EX - 1) / EX;
  a.chunks = (K + OUT - 1) / OUT;
  const size_t smem = (size_t)pcb_round_up(R, 8) * (WPD + XP) * sizeof(float);
  a.tile_ctas = tile_ctas(a.tiles, a.nblk * a.chunks, smem, R <= 2 * RSTEP ? 4 : 2);
  a.dense_ctas = a.nblk * a.chunks * a.tile_ctas;
  a.sparse_tiles = (ws->B + 4 * SPARSE - 1) / (4 * SPARSE);
  const uint32_t sparse_ctas = (loose * a.sparse_tiles + TPB / SPARSE - 1) / (TPB / SPARSE);
  static PcbPerDeviceOnce once;
  PCB_CUDA(once.run([] {
    for (auto kernel : {chain_down_kernel<1>, chain_down_kernel<2>, chain_down_kernel<4>}) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)(MAX_DIM * (WPD + XP) * sizeof(float)));
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }));
  PcbProfScope ps(c, st, PCB_K_DENSE_BWD_CHILD);
  auto kernel = R <= RSTEP ? chain_down_kernel<1> : R <= 2 * RSTEP ? chain_down_kernel<2> : chain_down_kernel<4>;
  PCB_CUDA(pcb_launch_pdl(kernel, dim3(a.dense_ctas + sparse_ctas), dim3(TPB),
                          smem, st, c->pdl, a, pcb_sparse_down_args(c, ws, hi)));
  return PCB_OK;
}

// Edge statistics of dense blocks [o0, o0 + n): true where the narrow kernel takes them.
bool pcb_edge_narrow_takes(const pcb_circuit* c) {
  return c->chain && c->max_dense_R <= EDGE_NARROW_DIM && c->max_dense_K <= EDGE_NARROW_DIM;
}

int32_t pcb_edge_narrow(pcb_circuit* c, pcb_workspace* ws, uint32_t o0, uint32_t n, cudaStream_t st) {
  const uint32_t rchunks = (c->max_dense_R + OUT - 1) / OUT, cchunks = (c->max_dense_K + OUT - 1) / OUT;
  const uint32_t tiles = (ws->B + EX - 1) / EX;
  // two waves of CTAs where the examples allow it
  const uint32_t slices = std::max(1u, std::min((tiles + 1) / 2, 148 * 4 / std::max(1u, n * rchunks * cchunks)));
  PCB_REQUIRE((uint64_t)n * rchunks * cchunks * slices <= 0x7fffffffull, "too many dense blocks for one launch");
  PcbProfScope ps(c, st, PCB_K_DENSE_BWD_EDGE);
  edge_narrow_kernel<<<n * rchunks * cchunks * slices, TPB, 0, st>>>(ws->mars, ws->flows, ws->blk_mx, c->theta, c->aggr, c->dense + o0,
                                                                     ws->ld, ws->B, rchunks, cchunks, slices);
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}
