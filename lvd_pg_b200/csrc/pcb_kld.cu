// pcb_kld.cu — KLD between two parameterisations of one circuit, its gradient, and Adam.
//
// Reference kernels replaced (paths relative to VariationalJuice.jl/src):
//   kld_leaf_kernel      init_kld!_kernel + kl_div      queries/kld.jl:6-37, nodes/fixable_categorical_dist.jl:178-196
//   kld_up_kernel        kld_layer_up_kernel            queries/kld.jl:71-133
//   kld_down_kernel      kld_layer_down_logparam_kernel queries/kld.jl:212-320 (+ merge_params, misc.jl:710-754)
//   kld_leaf_grad_kernel input_kld_down_kernel          queries/kld.jl:502-547, fixable_categorical_dist.jl:215-221
//   adam_kernel + renorm apply_gradients / hard_update_params / update_params_adam
//                                                       sgd/adam.jl:63-127,218-242,314-315
//
// "Examples" here are parameter sets: params are [S, P] column-major, work matrices are
// [N][ldS].  Threads are laid out (set, node): blockDim.x covers sets, blockDim.y nodes, so a
// single parameter set still fills the block.
#include <algorithm>
#include <cstring>

#include "pcb_internal.h"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

#ifdef PCB_DIAG
// Diagnostic builds only: block 0 of every kernel of the chain stamps the global timer on entry,
// after the wait on the preceding launch and on exit.
__device__ unsigned long long g_kld_trace[3 * 256];
__device__ unsigned int g_kld_slot;
__device__ __forceinline__ unsigned long long gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define KLD_T_ENTER() unsigned int _slot = 0xffffffffu; \
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) { _slot = atomicAdd(&g_kld_slot, 1u) & 255u; g_kld_trace[3 * _slot] = gtime(); }
#define KLD_T_WAITED() if (_slot != 0xffffffffu) g_kld_trace[3 * _slot + 1] = gtime();
#define KLD_T_EXIT() if (_slot != 0xffffffffu) g_kld_trace[3 * _slot + 2] = gtime();
#else
#define KLD_T_ENTER()
#define KLD_T_WAITED()
#define KLD_T_EXIT()
#endif

// Pins a value fetched ahead of griddepcontrol.wait: without a use in front of the wait the compiler
// is free to sink the load of read-only data below it, which puts the fetch back on the critical path.
__device__ __forceinline__ void keep(float& x) { asm volatile("" : "+f"(x)); }
__device__ __forceinline__ void keep(uint32_t& x) { asm volatile("" : "+r"(x)); }

struct Shape2 {
  dim3 block, grid;
};
// x = sets (up to 32), y = items: consecutive threads read consecutive words of a parameter matrix
Shape2 shape_for(uint32_t S, uint32_t items) {
  const uint32_t bx = std::min(S, 32u), by = 128 / bx;
  Shape2 s;
  s.block = dim3(bx, by, 1);
  s.grid = dim3((items + by - 1) / by, (S + bx - 1) / bx, 1);
  return s;
}

__global__ void kld_leaf_kernel(float* __restrict__ klds, uint32_t ld, uint32_t S, const float* __restrict__ p1,
                                const float* __restrict__ p2, uint32_t n_inputs, uint64_t P,
                                const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_cats,
                                const uint64_t* __restrict__ in_poff, int* __restrict__ bump,
                                float* __restrict__ zero_grads, uint32_t N) {
  pcb_grid_dep_launch();   // the first layer above may fetch its static operands meanwhile
  KLD_T_ENTER();
  KLD_T_WAITED();
  uint32_t i = blockIdx.x * blockDim.y + threadIdx.y;
  uint32_t s = blockIdx.y * blockDim.x + threadIdx.x;
  if (bump && i == 0 && s == 0) *bump += 1;   // the fused step counts its calls in a device word
  if (zero_grads && blockIdx.y == 0 && threadIdx.x == 0)   // the push pass of the fused step (one set) adds into these
    for (uint32_t k = i; k < N; k += gridDim.x * blockDim.y) zero_grads[(size_t)k * ld] = k == N - 1 ? 1.0f : 0.0f;
  if (i >= n_inputs || s >= S) return;
  float v = 0.0f;
  uint64_t po = in_poff[i];
  if (po < P) {  // learnable leaf; fixed leaves contribute 0
    uint32_t C = in_cats[i];
    for (uint32_t k = 0; k < C; ++k) {
      float a = p1[s + (size_t)S * (po + k)], b = p2[s + (size_t)S * (po + k)];
      v += expf(a) * (a - b);
    }
  }
  klds[(size_t)in_node[i] * ld + s] = v;
  KLD_T_EXIT();
}

// Row-major [S, P] to column-major: 128 parameters x up to 32 sets per block through shared memory, both sides in
// whole lines, twelve independent loads per thread in flight at 24 sets.  Bound: HBM (8 bytes per value).
// 24 x 1.7 M values: 72 us; the generic strided copy it replaces took 126 us.
constexpr uint32_t COLS_P = 128;
__global__ void __launch_bounds__(256) param_columns_kernel(float* __restrict__ dst, const float* __restrict__ src,
                                                            uint32_t S, uint64_t P) {
  __shared__ float tile[32][COLS_P + 1];
  const uint64_t p0 = (uint64_t)blockIdx.x * COLS_P;
  const uint32_t s0 = blockIdx.y * 32, St = min(32u, S - s0), np = (uint32_t)min((uint64_t)COLS_P, P - p0);
  const uint32_t lane = threadIdx.x % COLS_P, row = threadIdx.x / COLS_P;
  if (lane < np) {
#pragma unroll
    for (uint32_t s = 0; s < 32; s += 256 / COLS_P)
      if (s + row < St) tile[s + row][lane] = __ldcs(src + (uint64_t)(s0 + s + row) * P + p0 + lane);
  }
  __syncthreads();
  const uint32_t step_p = 256 / St, step_s = 256 % St;   // 256 elements further in [parameter][set] order
  uint32_t p = threadIdx.x / St, s = threadIdx.x % St;
  while (p < np) {
    dst[(p0 + p) * S + s0 + s] = tile[s][p];
    p += step_p; s += step_s;
    if (s >= St) { s -= St; ++p; }
  }
}

// ---- several parameter sets: one launch per layer --------------------------------------------------------
// A parameter row [S] of an edge and the rows of the edges behind it are contiguous, so a block of threads laid
// out (set, edge) with the set fastest reads whole runs.  Bound: HBM over the layers (both parameter matrices once
// upward, once more plus both gradient matrices downward), the chain of launches where a layer is small.  What does
// not depend on the neighbouring layer (the parameters of up to KLD_SLOTS steps per thread) is copied into shared
// memory with cp.async BEFORE the wait on the preceding launch: every step of a thread has a private slot, so all of
// a CTA's parameter bytes are in flight at once without holding registers (with loads through registers, four steps
// in flight, the widest layer ran at 1.6 TB/s).  The values of the neighbouring layer are staged for the whole CTA
// in one batch of loads after the wait, so a small layer costs one L2 round trip.  Dense blocks
// (children c0.., d0.. consecutive) need no edge list; the other nodes of the layer ride in the same launch.
// The launches follow the steps of the EM passes: a fused product is read as the sum of its sources by the block above
// it (three of them in flight; one at a time the upward pass took 236 us), so the chain has 11 launches instead of 19.
// 784 variables x 64 latents x 24 sets: upward 1164 -> 185 us over layers, 194 over steps; downward 1726 -> 207 -> 187 us.
// One set, both passes: 180 -> 155 us.
constexpr uint32_t KLD_THREADS = 256, KLD_SLOTS = 32;   // steps parked per thread; further ones are read directly
constexpr uint32_t KLD_STAGE = 8 * KLD_THREADS;         // staged values of the neighbouring layer (floats)

struct KldLayer {
  float* klds; float* grads; const float* p1; const float* p2; float* g1; float* g2;
  uint32_t ld, S, St;                    // sets, sets per tile (blockIdx.y)
  const PcbDenseBlock* blk; const PcbDenseBlock* thin; uint32_t nblk;   // thin: single sum nodes (up only), after the blocks
  const uint32_t* src_list;
  uint32_t per_blk, dense_ctas, rows;    // CTAs per block; rows (up) / children (down) of one
  uint32_t slots;
  const uint32_t* nodes; uint32_t count; // nodes outside dense blocks
  const uint8_t* kind; const uint32_t* n_estart; const uint32_t* n_ecount; const uint32_t* n_pid0;
  const uint32_t* e_prime; const uint32_t* e_sub; const uint32_t* in_off; const PcbInEntry* in_ent;
  uint32_t root; float* root_out;
};

__global__ void __launch_bounds__(KLD_THREADS) kld_up_layer_kernel(KldLayer a) {
  extern __shared__ float park[];   // [slots][p1 | p2][threads], then the staged values
  __shared__ float red[KLD_THREADS];
  __shared__ uint32_t src[PCB_MAX_SOURCES];
  pcb_grid_dep_launch();
  const uint32_t s0 = blockIdx.y * a.St, St = min(a.St, a.S - s0), J = KLD_THREADS / a.St;
  const uint32_t q = threadIdx.x / a.St, s = threadIdx.x % a.St;
  if (blockIdx.x < a.dense_ctas) {
    const uint32_t bi = blockIdx.x / a.per_blk;
    const PcbDenseBlock b = bi < a.nblk ? a.blk[bi] : a.thin[bi - a.nblk];
    const uint32_t i0 = blockIdx.x % a.per_blk * a.rows, JG = J / a.rows;
    if (i0 >= b.R) return;
    const uint32_t nsrc = b.src != PCB_NONE ? a.src_list[b.src] : 0;
    if (threadIdx.x < nsrc) src[threadIdx.x] = a.src_list[b.src + 1 + threadIdx.x];
    const uint32_t r = q / JG, jg = q % JG, i = i0 + r;
    const bool on = q < JG * a.rows && s < St && i < b.R;
    float* const stage = park + (size_t)a.slots * 2 * KLD_THREADS;
    float* const mine = park + threadIdx.x;
    const size_t base = ((size_t)b.pid0 + (size_t)(on ? i : 0) * b.K) * a.S + s0 + (on ? s : 0);
    if (on)
      for (uint32_t j = jg, m = 0; j < b.K && m < a.slots; j += JG, ++m) {
        pcb_copy4_async(mine + (2 * m) * KLD_THREADS, a.p1 + base + (size_t)j * a.S);
        pcb_copy4_async(mine + (2 * m + 1) * KLD_THREADS, a.p2 + base + (size_t)j * a.S);
      }
    __syncthreads();   // src is complete
    pcb_grid_dep_wait();
    const uint32_t cj = KLD_STAGE / a.St;
    float acc = 0.0f;
    uint32_t j = jg, m = 0;
    for (uint32_t c0 = 0; c0 < b.K; c0 += cj) {
      const uint32_t n = min(cj, b.K - c0);
      const float* kc = a.klds + (size_t)((nsrc ? src[0] : b.c0) + c0) * a.ld + s0 + s;
      const float* kd = a.klds + (size_t)((b.d0 != PCB_NONE ? b.d0 : b.c0) + c0) * a.ld + s0 + s;
      float v0[8], v1[8];
      for (uint32_t g0 = q; g0 < n; g0 += 8 * J) {
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
          const bool in = q < J && s < St && g0 + u * J < n;
          v0[u] = in ? kc[(size_t)(g0 + u * J) * a.ld] : 0.0f;
          v1[u] = in && b.d0 != PCB_NONE ? kd[(size_t)(g0 + u * J) * a.ld] : 0.0f;
        }
        for (uint32_t x = 1; x < nsrc; x += 3) {   // the other nodes that a fused product adds up, three of them in flight
          float y[3][8];
#pragma unroll
          for (uint32_t k = 0; k < 3; ++k) {
            const float* ks = a.klds + (size_t)(src[min(x + k, nsrc - 1)] + c0) * a.ld + s0 + s;
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) y[k][u] = x + k < nsrc && q < J && s < St && g0 + u * J < n ? ks[(size_t)(g0 + u * J) * a.ld] : 0.0f;
          }
#pragma unroll
          for (uint32_t k = 0; k < 3; ++k)
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) v0[u] += y[k][u];
        }
        if (nsrc && i0 == 0)   // the products' own values: the way down and the accessors read them
#pragma unroll
          for (uint32_t u = 0; u < 8; ++u)
            if (q < J && s < St && g0 + u * J < n) a.klds[(size_t)(b.c0 + c0 + g0 + u * J) * a.ld + s0 + s] = v0[u];
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u)
          if (q < J && s < St && g0 + u * J < n) stage[(g0 + u * J) * a.St + s] = v0[u] + v1[u];
      }
      if (c0 == 0) pcb_copies_wait();
      __syncthreads();
      if (on)
        for (; j < c0 + n; j += JG, ++m) {
          float x, y;
          if (m < a.slots) { x = mine[(2 * m) * KLD_THREADS]; y = mine[(2 * m + 1) * KLD_THREADS]; }
          else { x = a.p1[base + (size_t)j * a.S]; y = a.p2[base + (size_t)j * a.S]; }
          acc += expf(x) * (stage[(j - c0) * a.St + s] + x - y);
        }
      if (c0 + cj < b.K) __syncthreads();
    }
    red[threadIdx.x] = acc;   // the groups of a row lie St threads apart
    __syncthreads();
    if (on && jg == 0) {
      float t = 0.0f;
      for (uint32_t g = 0; g < JG; ++g) t += red[threadIdx.x + g * a.St];
      a.klds[(size_t)(b.p0 + i) * a.ld + s0 + s] = t;
      if (a.root_out && b.p0 + i == a.root) a.root_out[s0 + s] = t;
    }
    return;
  }
  // the other nodes, one per group of threads; one with many edges is taken by the whole block afterwards
  const uint32_t first = (blockIdx.x - a.dense_ctas) * J, k = first + q;
  const bool mine = q < J && s < St && k < a.count;
  const uint32_t n = mine ? a.nodes[k] : 0, cnt = mine ? a.n_ecount[n] : 0, e0 = mine ? a.n_estart[n] : 0;
  const bool wide = cnt > 8;
  const bool any_wide = __syncthreads_or(wide) != 0;
  auto edge = [&](uint32_t e, bool issum, uint32_t pid) {
    float v = a.klds[(size_t)a.e_prime[e] * a.ld + s0 + s];
    const uint32_t sb = a.e_sub[e];
    if (sb != PCB_NONE) v += a.klds[(size_t)sb * a.ld + s0 + s];
    if (issum) {
      const size_t at = (size_t)pid * a.S + s0 + s;
      const float x = a.p1[at], y = a.p2[at];
      v = expf(x) * (v + x - y);
    }
    return v;
  };
  pcb_grid_dep_wait();
  if (mine && !wide) {
    const bool issum = a.kind[n] == PCB_SUM;
    float acc = 0.0f;
    for (uint32_t j = 0; j < cnt; ++j) acc += edge(e0 + j, issum, a.n_pid0[n] + j);
    a.klds[(size_t)n * a.ld + s0 + s] = acc;
    if (a.root_out && n == a.root) a.root_out[s0 + s] = acc;
  }
  if (!any_wide) return;
  for (uint32_t x = first; x < min(first + J, a.count); ++x) {
    const uint32_t nx = a.nodes[x], ex = a.n_estart[nx], cx = a.n_ecount[nx];
    if (cx <= 8) continue;
    const bool issum = a.kind[nx] == PCB_SUM;
    float acc = 0.0f;
    if (q < J && s < St)
#pragma unroll 4
      for (uint32_t j = q; j < cx; j += J) acc += edge(ex + j, issum, a.n_pid0[nx] + j);
    red[threadIdx.x] = acc;
    __syncthreads();
    if (q == 0 && s < St) {
      float t = 0.0f;
      for (uint32_t g = 0; g < J; ++g) t += red[s + g * a.St];
      a.klds[(size_t)nx * a.ld + s0 + s] = t;
      if (a.root_out && nx == a.root) a.root_out[s0 + s] = t;
    }
    __syncthreads();
  }
}

// A few sets (kld_by_warps): one warp per (sum node, set), lanes over the node's edges.  Such a call is a chain of short dependent
// launches, so everything that does not depend on the step below (the run of children or the edge list, both parameters
// of the first 64 edges and exp of one) is fetched BEFORE the wait on the preceding launch; after it only the children's
// values are gathered, all of them in flight at once, so a step costs one round trip to L2.
// Blocks of threads: eight rows of a dense block each, then eight of the other nodes.
constexpr int KLD_PRE = 2;   // edges per lane held across the wait
__global__ void __launch_bounds__(256) kld_up_warp_kernel(KldLayer a) {
  __shared__ uint32_t src[PCB_MAX_SOURCES];
  pcb_grid_dep_launch();
  KLD_T_ENTER();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, s = blockIdx.y, S = a.S;
  float* const klds = a.klds + s;
  const size_t ld = a.ld;
  if (blockIdx.x < a.dense_ctas) {
    const uint32_t bi = blockIdx.x / a.per_blk;
    const PcbDenseBlock b = bi < a.nblk ? a.blk[bi] : a.thin[bi - a.nblk];
    const uint32_t i = blockIdx.x % a.per_blk * 8 + warp;
    if (blockIdx.x % a.per_blk * 8 >= b.R) return;
    uint32_t nsrc = b.src != PCB_NONE ? a.src_list[b.src] : 0;
    if (threadIdx.x < nsrc) src[threadIdx.x] = a.src_list[b.src + 1 + threadIdx.x];
    const size_t base = s + (size_t)S * (b.pid0 + (size_t)(i < b.R ? i : 0) * b.K);
    float wgt[KLD_PRE], dif[KLD_PRE];
#pragma unroll
    for (int r = 0; r < KLD_PRE; ++r) {
      const uint32_t j = lane + 32 * r;
      wgt[r] = dif[r] = 0.0f;
      if (j < b.K) {
        const float x = a.p1[base + (size_t)S * j], y = a.p2[base + (size_t)S * j];
        wgt[r] = expf(x);
        dif[r] = x - y;
      }
      keep(wgt[r]); keep(dif[r]);
    }
    keep(nsrc);
    if (nsrc) __syncthreads();   // the same for the block
    pcb_grid_dep_wait();
    KLD_T_WAITED();
    const uint32_t first = nsrc ? src[0] : b.c0, second = nsrc > 1 ? src[1] : first, sub = b.d0 != PCB_NONE ? b.d0 : first;
    // the first 64 children together, four sources of each in flight
    float k[KLD_PRE], pr[KLD_PRE], ks[KLD_PRE], acc = 0.0f;
#pragma unroll
    for (int r = 0; r < KLD_PRE; ++r) {
      const uint32_t j = min(lane + 32 * r, b.K - 1);
      const float k0 = klds[(size_t)(first + j) * ld], k1 = klds[(size_t)(second + j) * ld], k2 = klds[(size_t)(sub + j) * ld];
      pr[r] = k0 + (nsrc > 1 ? k1 : 0.0f);
      ks[r] = b.d0 != PCB_NONE ? k2 : 0.0f;
    }
    for (uint32_t x = 2; x < nsrc; x += 4) {
      float y[KLD_PRE][4];
#pragma unroll
      for (int r = 0; r < KLD_PRE; ++r)
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
          y[r][q] = x + q < nsrc ? klds[(size_t)(src[x + q] + min(lane + 32 * r, b.K - 1)) * ld] : 0.0f;
#pragma unroll
      for (int r = 0; r < KLD_PRE; ++r) pr[r] += (y[r][0] + y[r][1]) + (y[r][2] + y[r][3]);
    }
#pragma unroll
    for (int r = 0; r < KLD_PRE; ++r) {
      k[r] = pr[r] + ks[r];
      acc += lane + 32 * r < b.K ? wgt[r] * (k[r] + dif[r]) : 0.0f;
      if (nsrc && i == 0 && lane + 32 * r < b.K) klds[(size_t)(b.c0 + lane + 32 * r) * ld] = pr[r];   // the products' own values
    }
    for (uint32_t j = lane + 32 * KLD_PRE; j < b.K; j += 32) {
      float product = klds[(size_t)(first + j) * ld] + (nsrc > 1 ? klds[(size_t)(second + j) * ld] : 0.0f);
#pragma unroll 4
      for (uint32_t x = 2; x < nsrc; ++x) product += klds[(size_t)(src[x] + j) * ld];
      const float v = product + (b.d0 != PCB_NONE ? klds[(size_t)(sub + j) * ld] : 0.0f);
      const float x = a.p1[base + (size_t)S * j], y = a.p2[base + (size_t)S * j];
      acc += expf(x) * (v + x - y);
      if (nsrc && i == 0) klds[(size_t)(b.c0 + j) * ld] = product;
    }
    acc = warp_sum(acc);
    if (lane == 0 && i < b.R) {
      klds[(size_t)(b.p0 + i) * ld] = acc;
      if (a.root_out && b.p0 + i == a.root) a.root_out[s] = acc;
    }
    KLD_T_EXIT();
    return;
  }
  const uint32_t i = (blockIdx.x - a.dense_ctas) * 8 + warp;
  if (i >= a.count) return;
  const uint32_t n = a.nodes[i], e0 = a.n_estart[n], cnt = a.n_ecount[n], pid0 = a.n_pid0[n];
  const bool issum = a.kind[n] == PCB_SUM;
  uint32_t pr[KLD_PRE], sb[KLD_PRE];
  float wgt[KLD_PRE], dif[KLD_PRE];
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    const uint32_t j = lane + 32 * r;
    pr[r] = sb[r] = PCB_NONE; wgt[r] = 1.0f; dif[r] = 0.0f;
    if (j < cnt) {
      pr[r] = a.e_prime[e0 + j]; sb[r] = a.e_sub[e0 + j];
      if (issum) {
        const float x = a.p1[s + (size_t)S * (pid0 + j)], y = a.p2[s + (size_t)S * (pid0 + j)];
        wgt[r] = expf(x);
        dif[r] = x - y;
      }
    }
    keep(pr[r]); keep(sb[r]); keep(wgt[r]); keep(dif[r]);
  }
  pcb_grid_dep_wait();
  float k0[KLD_PRE], k1[KLD_PRE], acc = 0.0f;   // an edge without a second child reads the first one again
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    const uint32_t first = pr[r] != PCB_NONE ? pr[r] : n;
    k0[r] = klds[(size_t)first * ld];
    k1[r] = klds[(size_t)(sb[r] != PCB_NONE ? sb[r] : first) * ld];
  }
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    const float k = k0[r] + (sb[r] != PCB_NONE ? k1[r] : 0.0f);
    if (pr[r] != PCB_NONE) acc += issum ? wgt[r] * (k + dif[r]) : k;
  }
  for (uint32_t j = lane + 32 * KLD_PRE; j < cnt; j += 32) {
    float k = klds[(size_t)a.e_prime[e0 + j] * ld];
    const uint32_t sb = a.e_sub[e0 + j];
    if (sb != PCB_NONE) k += klds[(size_t)sb * ld];
    if (issum) {
      const float x = a.p1[s + (size_t)S * (pid0 + j)], y = a.p2[s + (size_t)S * (pid0 + j)];
      k = expf(x) * (k + x - y);
    }
    acc += k;
  }
  acc = warp_sum(acc);
  if (lane == 0) {
    klds[(size_t)n * ld] = acc;
    if (a.root_out && n == a.root) a.root_out[s] = acc;
  }
  KLD_T_EXIT();
}

// edge_klds of sum and product edges in up-edge order, [E][ldS]-free: written straight to a
// [S, E] column-major buffer (parity accessor only)
__global__ void kld_edge_kernel(const float* __restrict__ klds, uint32_t ld, uint32_t S, const float* __restrict__ p1,
                                const float* __restrict__ p2, const uint32_t* __restrict__ nodes, uint32_t count,
                                const uint8_t* __restrict__ kind, const uint32_t* __restrict__ n_estart,
                                const uint32_t* __restrict__ n_ecount, const uint32_t* __restrict__ n_pid0,
                                const uint32_t* __restrict__ e_prime, const uint32_t* __restrict__ e_sub,
                                float* __restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.y + threadIdx.y;
  uint32_t s = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= count || s >= S) return;
  uint32_t n = nodes[i];
  uint32_t e0 = n_estart[n], cnt = n_ecount[n];
  bool issum = kind[n] == PCB_SUM;
  uint32_t pid0 = n_pid0[n];
  for (uint32_t j = 0; j < cnt; ++j) {
    float k = klds[(size_t)e_prime[e0 + j] * ld + s];
    uint32_t sb = e_sub[e0 + j];
    if (sb != PCB_NONE) k += klds[(size_t)sb * ld + s];
    if (issum) {
      float a = p1[s + (size_t)S * (pid0 + j)], b = p2[s + (size_t)S * (pid0 + j)];
      k = expf(a) * (k + a - b);
    }
    out[s + (size_t)S * (e0 + j)] = k;
  }
}

// Gradients of one layer, in one launch: the dense blocks whose parents lie in the layer above hand their gradients
// to the children and write both parameter gradients; the other nodes of this layer pull from their parents.  All
// parents of either kind were completed by earlier launches.  g1 = pg * (exp(a) * (ck + a - b) + exp(a)) and
// g2 = -pg * exp(a): both factors of pg are formed before the wait.
__global__ void __launch_bounds__(KLD_THREADS) kld_down_layer_kernel(KldLayer a) {
  extern __shared__ float park[];
  __shared__ float red[KLD_THREADS];
  pcb_grid_dep_launch();
  const uint32_t s0 = blockIdx.y * a.St, St = min(a.St, a.S - s0), J = KLD_THREADS / a.St;
  const uint32_t q = threadIdx.x / a.St, s = threadIdx.x % a.St;
  if (blockIdx.x < a.dense_ctas) {
    const PcbDenseBlock b = a.blk[blockIdx.x / a.per_blk];
    const uint32_t JC = a.rows, IG = J / JC;
    const uint32_t nsrc = b.src != PCB_NONE ? a.src_list[b.src] : 0;
    const uint32_t jj = q % JC, ig = q / JC, j = blockIdx.x % a.per_blk * JC + jj;
    const bool on = ig < IG && s < St && j < b.K;
    const size_t base = ((size_t)b.pid0 + (on ? j : 0)) * a.S + s0 + (on ? s : 0), step = (size_t)b.K * a.S;
    float* const stage = park + (size_t)a.slots * 2 * KLD_THREADS;
    float* const mine = park + threadIdx.x;
    float ck = 0.0f;
    if (on) {
      for (uint32_t i = ig, m = 0; i < b.R && m < a.slots; i += IG, ++m) {
        pcb_copy4_async(mine + (2 * m) * KLD_THREADS, a.p1 + base + i * step);
        pcb_copy4_async(mine + (2 * m + 1) * KLD_THREADS, a.p2 + base + i * step);
      }
      ck = a.klds[(size_t)(b.c0 + j) * a.ld + s0 + s];
      if (b.d0 != PCB_NONE) ck += a.klds[(size_t)(b.d0 + j) * a.ld + s0 + s];
      pcb_copies_wait();
      for (uint32_t i = ig, m = 0; i < b.R && m < a.slots; i += IG, ++m) {
        const float x = mine[(2 * m) * KLD_THREADS], ea = expf(x);
        mine[(2 * m + 1) * KLD_THREADS] = ea * (ck + x - mine[(2 * m + 1) * KLD_THREADS]) + ea;
        mine[(2 * m) * KLD_THREADS] = ea;
      }
    }
    pcb_grid_dep_wait();
    const uint32_t ci = KLD_STAGE / a.St;
    float acc = 0.0f;
    uint32_t i = ig, m = 0;
    for (uint32_t c0 = 0; c0 < b.R; c0 += ci) {
      const uint32_t n = min(ci, b.R - c0);
      const float* pgp = a.grads + (size_t)(b.p0 + c0) * a.ld + s0 + s;
      float v[8];
      for (uint32_t g0 = q; g0 < n; g0 += 8 * J) {
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) v[u] = q < J && s < St && g0 + u * J < n ? pgp[(size_t)(g0 + u * J) * a.ld] : 0.0f;
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u)
          if (q < J && s < St && g0 + u * J < n) stage[(g0 + u * J) * a.St + s] = v[u];
      }
      __syncthreads();
      if (on)
        for (; i < c0 + n; i += IG, ++m) {
          const float pg = stage[(i - c0) * a.St + s];
          float ea, gx;
          if (m < a.slots) {
            ea = mine[(2 * m) * KLD_THREADS]; gx = mine[(2 * m + 1) * KLD_THREADS];
          } else {
            const float x = a.p1[base + i * step], y = a.p2[base + i * step];
            ea = expf(x); gx = ea * (ck + x - y) + ea;
          }
          __stcs(a.g1 + base + i * step, pg * gx);
          __stcs(a.g2 + base + i * step, -pg * ea);
          acc += pg * ea;
        }
      if (c0 + ci < b.R) __syncthreads();
    }
    red[threadIdx.x] = on ? acc : 0.0f;
    __syncthreads();
    if (on && ig == 0) {
      float t = 0.0f;
      for (uint32_t g = 0; g < IG; ++g) t += red[threadIdx.x + g * JC * a.St];
      if (!nsrc) a.grads[(size_t)(b.c0 + j) * a.ld + s0 + s] = t;
      for (uint32_t x = 0; x < nsrc; ++x) a.grads[(size_t)(a.src_list[b.src + 1 + x] + j) * a.ld + s0 + s] = t;   // what the product hands on
      if (b.d0 != PCB_NONE) a.grads[(size_t)(b.d0 + j) * a.ld + s0 + s] = t;
    }
    return;
  }
  const uint32_t k = (blockIdx.x - a.dense_ctas) * J + q;
  pcb_grid_dep_wait();
  if (q >= J || k >= a.count || s >= St) return;
  const uint32_t n = a.nodes[k], i0 = a.in_off[n], i1 = a.in_off[n + 1];
  float acc = (i0 == i1 && n == a.root) ? 1.0f : 0.0f;
  const float myk = a.klds[(size_t)n * a.ld + s0 + s];
  for (uint32_t x = i0; x < i1; ++x) {
    const PcbInEntry en = a.in_ent[x];
    const float pg = a.grads[(size_t)en.parent * a.ld + s0 + s];
    float eg = pg;
    if (en.pid != PCB_NONE) {
      const size_t at = (size_t)en.pid * a.S + s0 + s;
      const float p = a.p1[at], ea = expf(p);
      eg = pg * ea;
      if (en.flags & 1u) {
        const float ck = myk + (en.sib != PCB_NONE ? a.klds[(size_t)en.sib * a.ld + s0 + s] : 0.0f);
        a.g1[at] = pg * (ea * (ck + p - a.p2[at]) + ea);
        a.g2[at] = -pg * ea;
      }
    }
    acc += eg;
  }
  a.grads[(size_t)n * a.ld + s0 + s] = acc;
}

// one warp per (node, set): lanes over the node's incoming edges; the entries and the parameters of
// the first 64 of them are fetched before the wait on the preceding launch.  g2 may be null (the
// fused step needs the gradient with respect to the first parameter set only).
__global__ void kld_down_warp_kernel(float* __restrict__ grads, const float* __restrict__ klds, uint32_t ld,
                                     uint32_t S, const float* __restrict__ p1, const float* __restrict__ p2,
                                     const uint32_t* __restrict__ nodes, uint32_t count, uint32_t root,
                                     const uint32_t* __restrict__ in_off, const PcbInEntry* __restrict__ in_ent,
                                     float* __restrict__ g1, float* __restrict__ g2) {
  pcb_grid_dep_launch();
  KLD_T_ENTER();
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= count * S) return;
  const uint32_t i = w / S, s = w % S;
  const uint32_t n = nodes[i];
  const uint32_t i0 = in_off[n], i1 = in_off[n + 1];
  PcbInEntry en[KLD_PRE];
  float pa[KLD_PRE], pea[KLD_PRE], pb[KLD_PRE];
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    const uint32_t x = i0 + lane + 32 * r;
    en[r].parent = en[r].sib = en[r].pid = PCB_NONE; en[r].flags = 0; pa[r] = pb[r] = 0.0f; pea[r] = 1.0f;
    if (x < i1) {
      en[r] = in_ent[x];
      if (en[r].pid != PCB_NONE) {
        pa[r] = p1[s + (size_t)S * en[r].pid];
        pea[r] = expf(pa[r]);
        if (en[r].flags & 1u) pb[r] = p2[s + (size_t)S * en[r].pid];
      }
    }
    keep(en[r].parent); keep(en[r].sib); keep(en[r].pid); keep(en[r].flags); keep(pa[r]); keep(pea[r]); keep(pb[r]);
  }
  pcb_grid_dep_wait();   // everything above is static circuit data or this call's parameters
  KLD_T_WAITED();
  // every gather of the held entries is issued before the first use: one round trip to L2
  const float myk = klds[(size_t)n * ld + s];
  float pg[KLD_PRE], sk[KLD_PRE];
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    const uint32_t ap = en[r].parent != PCB_NONE ? en[r].parent : n;
    const uint32_t as = (g1 && en[r].sib != PCB_NONE) ? en[r].sib : n;
    pg[r] = grads[(size_t)ap * ld + s];
    sk[r] = klds[(size_t)as * ld + s];
  }
  float acc = 0.0f;
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    if (en[r].parent == PCB_NONE) continue;
    float eg = pg[r];
    if (en[r].pid != PCB_NONE) {
      eg = pg[r] * pea[r];
      if (g1 && (en[r].flags & 1u)) {
        const float ck = myk + (en[r].sib != PCB_NONE ? sk[r] : 0.0f);
        const float edge_kld = pea[r] * (ck + pa[r] - pb[r]);
        g1[s + (size_t)S * en[r].pid] = pg[r] * (edge_kld + pea[r]);
        if (g2) g2[s + (size_t)S * en[r].pid] = -pg[r] * pea[r];
      }
    }
    acc += eg;
  }
  for (uint32_t x = i0 + lane + 32 * KLD_PRE; x < i1; x += 32) {
    PcbInEntry e2 = in_ent[x];
    float pgx = grads[(size_t)e2.parent * ld + s];
    float eg = pgx;
    if (e2.pid != PCB_NONE) {
      float a = p1[s + (size_t)S * e2.pid];
      float ea = expf(a);
      eg = pgx * ea;
      if (g1 && (e2.flags & 1u)) {
        float b = p2[s + (size_t)S * e2.pid];
        float ck = myk + (e2.sib != PCB_NONE ? klds[(size_t)e2.sib * ld + s] : 0.0f);
        float edge_kld = ea * (ck + a - b);
        g1[s + (size_t)S * e2.pid] = pgx * (edge_kld + ea);
        if (g2) g2[s + (size_t)S * e2.pid] = -pgx * ea;
      }
    }
    acc += eg;
  }
  acc = warp_sum(acc);
  if (lane == 0) grads[(size_t)n * ld + s] = acc + ((i0 == i1 && n == root) ? 1.0f : 0.0f);
  KLD_T_EXIT();
}

__global__ void kld_leaf_grad_kernel(const float* __restrict__ grads, uint32_t ld, uint32_t S,
                                     const float* __restrict__ p1, const float* __restrict__ p2, uint32_t n_inputs,
                                     uint64_t P, const uint32_t* __restrict__ in_node,
                                     const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_poff,
                                     float* __restrict__ g1, float* __restrict__ g2) {
  pcb_grid_dep_launch();
  KLD_T_ENTER();
  uint32_t i = blockIdx.x * blockDim.y + threadIdx.y;
  uint32_t s = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n_inputs || s >= S) return;
  uint64_t po = in_poff[i];
  if (po >= P) return;
  const uint32_t node = in_node[i];
  uint32_t C = in_cats[i];
  uint32_t node_k = node;
  keep(node_k); keep(C);
  pcb_grid_dep_wait();
  KLD_T_WAITED();
  float g = grads[(size_t)node * ld + s];
  for (uint32_t k = 0; k < C; ++k) {
    float a = p1[s + (size_t)S * (po + k)], b = p2[s + (size_t)S * (po + k)];
    g1[s + (size_t)S * (po + k)] = g * (a - b + 1.0f);
    if (g2) g2[s + (size_t)S * (po + k)] = g * expf(a - b);  // plus sign, as the reference returns it for leaves
  }
  KLD_T_EXIT();
}

__global__ void copy_root_kernel(const float* __restrict__ klds_root, uint32_t S, float* __restrict__ out) {
  uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < S) out[s] = klds_root[s];
}

// t_dev != null: the step count comes from a device word (a replayed CUDA graph cannot take it as an
// argument) and the bias corrections 1 - beta^t are computed here
__global__ void adam_kernel(float* __restrict__ theta, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, uint64_t n, float lr, float b1, float b2, float eps, float c1,
                            float c2, float sign, const int* __restrict__ t_dev) {
  if (t_dev) {
    const float t = (float)*t_dev;
    c1 = 1.0f - powf(b1, t);
    c2 = 1.0f - powf(b2, t);
  }
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    float gi = g[i];
    float mi = b1 * m[i] + (1.0f - b1) * gi;
    float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float m_hat = mi / c1, v_hat = vi / c2;
    theta[i] += sign * lr * (m_hat / (sqrtf(v_hat) + eps));
  }
}

// one warp per normalised group: sum groups first, then learnable leaves
__global__ void renorm_kernel(float* __restrict__ theta, uint32_t n_groups, const uint32_t* __restrict__ grp_node,
                              const uint32_t* __restrict__ n_pid0, const uint32_t* __restrict__ n_ecount,
                              uint32_t n_inputs, uint64_t P, const uint32_t* __restrict__ in_cats,
                              const uint64_t* __restrict__ in_poff) {
  uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t lane = threadIdx.x & 31;
  uint64_t off;
  uint32_t cnt;
  if (w < n_groups) {
    uint32_t n = grp_node[w];
    off = n_pid0[n];
    cnt = n_ecount[n];
    if (cnt == 1) return;  // single-edge sum nodes are left alone (adam.jl:113)
  } else if (w < n_groups + n_inputs) {
    uint32_t i = w - n_groups;
    off = in_poff[i];
    cnt = in_cats[i];
    if (off >= P) return;
  } else {
    return;
  }
  float s = 0.0f;
  for (uint32_t j = lane; j < cnt; j += 32) s += expf(theta[off + j]);
  s = warp_sum(s);
  float ls = logf(s);
  for (uint32_t j = lane; j < cnt; j += 32) theta[off + j] -= ls;
}

// Which chain a call of a few sets takes: a warp per (node, set), or the tiles of the layer kernels.  One and two sets go
// by warps, as the fused step's upward pass does.  Up to eight go by warps where that is the shorter chain: in circuits
// without dense blocks (a thread of a layer kernel walks such a node's edges alone) and in small ones (both passes on the
// device, warps against tiles: 100 variables x 8 latents, four sets 37 against 98 us, eight 37 against 109; 100 x 32, four
// sets 47 against 55, eight 56 against 58; 300 x 32, three sets 70 against 78, four 74 against 76, six 96 against 82;
// 784 x 16, three sets 67 against 68, four 76 against 66; 784 x 64, three sets 285 against 109).  In a deep
// circuit the launches count: the way down by warps goes by layers, so it has to have no more of them than steps, and a
// step to be small (a chain of 300 variables x 64 latents: three sets 1635 against 2087 us, five 1763 against 2146; a
// lane holds 64 edges ahead of the wait: a chain of 100 x 100 latents, three sets 896 against 833; an image tree of 768
// variables x 16 latents, three sets 349 against 311).
constexpr uint32_t KLD_WARP_SETS = 2, KLD_WARP_SETS_SMALL = 8;
bool kld_by_warps(const pcb_circuit* c, uint32_t S) {
  if (S <= KLD_WARP_SETS || S > KLD_WARP_SETS_SMALL || c->n_dense == 0) return S <= KLD_WARP_SETS_SMALL;
  const uint64_t work = (uint64_t)S * c->n_inner;
  return c->n_steps <= 32 ? work <= 500000 : c->L == c->n_steps && c->max_dense_K <= 64 && work <= (uint64_t)25000 * c->n_steps;
}

// what the kernels of step t need; the caller adds the loose nodes and the shares of a CTA
KldLayer kld_layer(pcb_circuit* c, pcb_workspace* ws, const float* p1, const float* p2, uint32_t S, uint32_t t) {
  KldLayer a;
  memset(&a, 0, sizeof(a));
  a.klds = ws->klds; a.grads = ws->grads; a.p1 = p1; a.p2 = p2; a.ld = ws->ldS; a.S = S; a.St = std::min(S, 32u);
  a.nblk = pcb_step_blocks(c, t);
  if (a.nblk) a.blk = c->dense + c->h_dense_off[t];
  a.src_list = c->src_list;
  a.kind = c->kind; a.n_estart = c->n_estart; a.n_ecount = c->n_ecount; a.n_pid0 = c->n_pid0;
  a.e_prime = c->e_prime; a.e_sub = c->e_sub; a.in_off = c->in_off; a.in_ent = c->in_ent; a.root = c->N - 1;
  return a;
}
// the upward work of step t: thin blocks and the nodes taken one by one; returns the number of blocks
uint32_t kld_up_work(pcb_circuit* c, KldLayer& a, uint32_t t) {
  const uint32_t thin = c->h_st_thin_off[t + 1] - c->h_st_thin_off[t];
  a.thin = c->thin + c->h_st_thin_off[t];
  a.nodes = c->st_up + c->h_st_up_off[t];
  a.count = c->h_st_up_off[t + 1] - c->h_st_up_off[t] - thin;
  return a.nblk + thin;
}

cudaError_t kld_launch_layer(pcb_circuit* c, void (*kernel)(KldLayer), KldLayer& a, uint32_t blocks, bool chained,
                             cudaStream_t st) {
  static PcbPerDeviceOnce once;
  const size_t most = (2 * KLD_SLOTS * KLD_THREADS + KLD_STAGE) * sizeof(float);
  cudaError_t e = once.run([&]() {
    cudaError_t r = cudaFuncSetAttribute(kld_up_layer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    return r != cudaSuccess ? r : cudaFuncSetAttribute(kld_down_layer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  });
  if (e != cudaSuccess) return e;
  const uint32_t J = KLD_THREADS / a.St;
  a.dense_ctas = blocks * a.per_blk;
  const uint32_t ctas = a.dense_ctas + (a.count + J - 1) / J;
  ++c->prof.launches[PCB_K_KLD];
  return pcb_launch_pdl(kernel, dim3(ctas, (a.S + a.St - 1) / a.St), dim3(KLD_THREADS),
                        a.dense_ctas ? (2 * a.slots * KLD_THREADS + KLD_STAGE) * sizeof(float) : 0, st, c->pdl && chained, a);
}

// a warp per sum node or loose node (kld_up_warp_kernel, kld1_push_kernel)
cudaError_t kld_launch_warps(pcb_circuit* c, void (*kernel)(KldLayer), KldLayer& a, uint32_t blocks, uint32_t R, cudaStream_t st) {
  a.per_blk = (R + 7) / 8;
  a.dense_ctas = blocks * a.per_blk;
  const uint32_t ctas = a.dense_ctas + (a.count + 7) / 8;
  if (!ctas) return cudaSuccess;
  ++c->prof.launches[PCB_K_KLD];
  return pcb_launch_pdl(kernel, dim3(ctas, a.S), dim3(256), 0, st, c->pdl, a);
}

}  // namespace

extern "C" int32_t pcb_param_columns(float* dst_dev, const float* src_dev, uint32_t S, uint64_t P, pcb_stream s) {
  PCB_REQUIRE(dst_dev && src_dev && S >= 1, "null argument");
  PCB_REQUIRE((uint64_t)(S + 31) / 32 <= 65535 && (P + COLS_P - 1) / COLS_P <= 0x7fffffffull, "matrix too large");
  if (P)
    param_columns_kernel<<<dim3((uint32_t)((P + COLS_P - 1) / COLS_P), (S + 31) / 32), 256, 0, (cudaStream_t)s>>>(
        dst_dev, src_dev, S, P);
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

extern "C" int32_t pcb_kld(pcb_circuit* c, pcb_workspace* ws, const float* params1_dev, const float* params2_dev,
                           uint32_t S, float* kld_out_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws && params1_dev && params2_dev, "null argument");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  PCB_REQUIRE(S >= 1, "no parameter sets");
  PCB_CUDA(cudaSetDevice(c->device));
  int32_t st0 = pcb_ws_ensure_sets(ws, S, PCB_WS_NODES);
  if (st0 != PCB_OK) return st0;
  cudaStream_t st = (cudaStream_t)s;
  const uint32_t ld = ws->ldS;
  if (c->n_inputs) {
    Shape2 sh = shape_for(S, c->n_inputs);
    ++c->prof.launches[PCB_K_KLD];
    kld_leaf_kernel<<<sh.grid, sh.block, 0, st>>>(ws->klds, ld, S, params1_dev, params2_dev, c->n_inputs, c->P,
                                                  c->in_node, c->in_cats, c->in_poff, ws->kld_bump,
                                                  ws->kld_bump ? ws->grads : nullptr, c->N);
  }
  for (uint32_t t = 1; t <= c->n_steps; ++t) {
    KldLayer a = kld_layer(c, ws, params1_dev, params2_dev, S, t);
    const uint32_t blocks = kld_up_work(c, a, t);
    a.root_out = kld_out_dev;
    uint32_t R = 1, K = 1;
    pcb_step_extent(c, t, R, K);
    for (uint32_t i = c->h_st_thin_off[t]; i < c->h_st_thin_off[t + 1]; ++i) K = std::max(K, c->h_thin[i].K);
    if (kld_by_warps(c, S)) {
      PCB_CUDA(kld_launch_warps(c, kld_up_warp_kernel, a, blocks, R, st));
      continue;
    }
    // a thread should have about twelve edges (24 KB of parameters in flight per CTA): rows that share a CTA
    const uint32_t J = KLD_THREADS / a.St;
    a.rows = std::min({std::max(1u, (J * 12 + K / 2) / K), J, R});
    a.per_blk = (R + a.rows - 1) / a.rows;
    a.slots = std::min(KLD_SLOTS, (K + J / a.rows - 1) / (J / a.rows));
    PCB_CUDA(kld_launch_layer(c, kld_up_layer_kernel, a, blocks, true, st));
  }
  if (kld_out_dev && c->L == 0)   // the layer kernels write the root's value themselves
    ++c->prof.launches[PCB_K_KLD], copy_root_kernel<<<(S + 127) / 128, 128, 0, st>>>(ws->klds + (size_t)(c->N - 1) * ld, S, kld_out_dev);
  PCB_CUDA(cudaGetLastError());
  ws->have_kld = true;
  ws->kld_S = S;
  return PCB_OK;
}

extern "C" int32_t pcb_kld_backward(pcb_circuit* c, pcb_workspace* ws, const float* params1_dev,
                                    const float* params2_dev, uint32_t S, float* grads1_dev, float* grads2_dev,
                                    pcb_stream s) {
  PCB_REQUIRE(c && ws && params1_dev && params2_dev && grads1_dev && grads2_dev, "null argument");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  if (!ws->have_kld || ws->kld_S != S)
    return pcb_fail(PCB_ERR_STATE, "pcb_kld_backward needs a preceding pcb_kld with the same number of sets");
  PCB_CUDA(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)s;
  const uint32_t ld = ws->ldS;
  bool chained = false;   // the first launch of the pass waits for whatever the caller's stream holds before it
  if (kld_by_warps(c, S)) {
    for (int64_t lay = c->L; lay >= 0; --lay) {
      const uint32_t o0 = c->h_down_all_off[lay], o1 = c->h_down_all_off[lay + 1];
      if (o1 == o0) continue;
      ++c->prof.launches[PCB_K_KLD];
      PCB_CUDA(pcb_launch_pdl(kld_down_warp_kernel, dim3((uint32_t)(((uint64_t)(o1 - o0) * S + 7) / 8)), dim3(256), 0, st,
                              c->pdl && chained, ws->grads, (const float*)ws->klds, ld, S, params1_dev, params2_dev, c->down_all + o0,
                              o1 - o0, c->N - 1, c->in_off, c->in_ent, grads1_dev, grads2_dev));
      chained = true;
    }
  } else {
    for (int64_t t = c->n_steps; t >= 0; --t) {   // the blocks of step t + 1 and the other nodes of step t
      KldLayer a = kld_layer(c, ws, params1_dev, params2_dev, S, (uint32_t)t + 1);
      a.g1 = grads1_dev; a.g2 = grads2_dev;
      a.nodes = c->st_down + c->h_st_down_off[t];
      a.count = c->h_st_down_off[t + 1] - c->h_st_down_off[t];
      if (!a.count && !a.nblk) continue;
      uint32_t R = 1, K = 1;
      pcb_step_extent(c, (uint32_t)t + 1, R, K);
      // children of a CTA: whole 256-byte runs of parameters; the rest of the threads split the rows
      const uint32_t J = KLD_THREADS / a.St;
      a.rows = std::min({std::max(1u, 64 / a.St), J, K});
      a.per_blk = (K + a.rows - 1) / a.rows;
      a.slots = std::min(KLD_SLOTS, (R + J / a.rows - 1) / (J / a.rows));
      PCB_CUDA(kld_launch_layer(c, kld_down_layer_kernel, a, a.nblk, chained, st));
      chained = true;
    }
  }
  if (c->n_inputs) {
    Shape2 sh = shape_for(S, c->n_inputs);
    ++c->prof.launches[PCB_K_KLD];
    PCB_CUDA(pcb_launch_pdl(kld_leaf_grad_kernel, sh.grid, sh.block, 0, st, c->pdl, (const float*)ws->grads, ld, S,
                            params1_dev, params2_dev, c->n_inputs, c->P, c->in_node, c->in_cats, c->in_poff, grads1_dev,
                            grads2_dev));
  }
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

// klds [S, N] of the last pcb_kld call, column-major.
extern "C" int32_t pcb_get_klds(pcb_circuit* c, pcb_workspace* ws, uint32_t S, float* klds_host) {
  PCB_REQUIRE(c && ws && klds_host, "null argument");
  PCB_REQUIRE(ws->have_kld && ws->kld_S == S, "no matching pcb_kld call");
  PCB_CUDA(cudaSetDevice(c->device));
  PCB_CUDA(cudaDeviceSynchronize());
  PCB_CUDA(cudaMemcpy2D(klds_host, S * sizeof(float), ws->klds, ws->ldS * sizeof(float), S * sizeof(float), c->N,
                        cudaMemcpyDeviceToHost));
  return PCB_OK;
}

extern "C" int32_t pcb_kld_edge_klds(pcb_circuit* c, pcb_workspace* ws, const float* params1_dev,
                                     const float* params2_dev, uint32_t S, float* edge_klds_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws && params1_dev && params2_dev && edge_klds_dev, "null argument");
  PCB_REQUIRE(ws->have_kld && ws->kld_S == S, "no matching pcb_kld call");
  PCB_CUDA(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)s;
  uint32_t total = c->h_up_all_off[c->L];
  if (total) {
    Shape2 sh = shape_for(S, total);
    ++c->prof.launches[PCB_K_KLD];
    kld_edge_kernel<<<sh.grid, sh.block, 0, st>>>(ws->klds, ws->ldS, S, params1_dev, params2_dev, c->up_all, total,
                                                  c->kind, c->n_estart, c->n_ecount, c->n_pid0, c->e_prime, c->e_sub,
                                                  edge_klds_dev);
  }
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

extern "C" int32_t pcb_adam_step(pcb_circuit* c, float* theta_dev, const float* grad_dev, float* m_dev, float* v_dev,
                                 int32_t t, float lr, float beta1, float beta2, float eps, float sign, pcb_stream s) {
  PCB_REQUIRE(c && theta_dev && grad_dev && m_dev && v_dev, "null argument");
  PCB_REQUIRE(t >= 1, "Adam step count starts at 1");
  PCB_CUDA(cudaSetDevice(c->device));
  cudaStream_t st = (cudaStream_t)s;
  float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
  if (c->P) {
    uint32_t blocks = (uint32_t)std::min<uint64_t>((c->P + 255) / 256, 148 * 16);
    ++c->prof.launches[PCB_K_KLD];
    adam_kernel<<<blocks, 256, 0, st>>>(theta_dev, grad_dev, m_dev, v_dev, c->P, lr, beta1, beta2, eps, c1, c2, sign, nullptr);
    uint32_t warps = c->n_groups + c->n_inputs;
    ++c->prof.launches[PCB_K_KLD];
    renorm_kernel<<<(warps + 7) / 8, 256, 0, st>>>(theta_dev, c->n_groups, c->grp_node, c->n_pid0, c->n_ecount,
                                                   c->n_inputs, c->P, c->in_cats, c->in_poff);
  }
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

// ---- KLD + gradient + Adam as one unit --------------------------------------------------------------
// One step of the variational loop on a single parameter set q against p: kld (queries/kld.jl:164-206),
// kld_backward with respect to q (:593-649), Adam descent on q's log-parameters and the
// re-normalisation of every sum group and leaf (sgd/adam.jl:63-127,218-242).  A single parameter set
// has no batch dimension, so the step is a chain of ~2 L small launches: the second call with the same
// arguments captures the chain as a CUDA graph (the step count lives in a device word that the graph
// increments itself) and later calls replay it.
namespace {
__global__ void set_step_kernel(int* __restrict__ t, int value) { *t = value; }

// ---- the fused single-set step: node gradients pushed down by the parents -------------------------
// Steps from the root down: every parent of a step's nodes lies in a higher step, so their gradients are complete.  A
// block of threads takes eight rows of a dense block: a warp per row, lanes over the edges, so the parameters are read
// contiguously (the pull form reads them with the stride of the fan-in); pg * exp(theta) of the eight rows is added in
// shared memory and reaches the children (and the nodes that fused products multiply) as one atomic each.  The other
// nodes push edge by edge.  The sums are floating-point atomics, like the reference's CUDA.@atomic on partially owned
// nodes (queries/kld.jl:258-300): the order of the additions, and with it the last bits, can differ from run to run.
__global__ void __launch_bounds__(256) kld1_push_kernel(KldLayer a) {
  __shared__ float red[8][256];
  __shared__ uint32_t src[PCB_MAX_SOURCES];
  pcb_grid_dep_launch();
  KLD_T_ENTER();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const grads = a.grads;
  const size_t ld = a.ld;
  if (blockIdx.x < a.dense_ctas) {
    const PcbDenseBlock b = a.blk[blockIdx.x / a.per_blk];
    const uint32_t i0 = blockIdx.x % a.per_blk * 8, i = i0 + warp;
    if (i0 >= b.R) return;
    uint32_t nsrc = b.src != PCB_NONE ? a.src_list[b.src] : 0;
    if (threadIdx.x < nsrc) src[threadIdx.x] = a.src_list[b.src + 1 + threadIdx.x];
    const float* const p = a.p1 + b.pid0 + (size_t)(i < b.R ? i : 0) * b.K;
    float wgt[KLD_PRE];
#pragma unroll
    for (int r = 0; r < KLD_PRE; ++r) {
      wgt[r] = lane + 32 * r < b.K ? expf(p[lane + 32 * r]) : 0.0f;
      keep(wgt[r]);
    }
    keep(nsrc);
    pcb_grid_dep_wait();   // everything above is static circuit data or this call's parameters
    KLD_T_WAITED();
    const float pg = i < b.R ? grads[(size_t)(b.p0 + i) * ld] : 0.0f;
    for (uint32_t j0 = 0; j0 < b.K; j0 += 256) {   // the rows' shares of up to 256 children at a time
      if (j0) __syncthreads();
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const uint32_t j = lane + 32 * r;
        if (j0 + j < b.K) red[warp][j] = pg * (j0 == 0 && r < KLD_PRE ? wgt[r < KLD_PRE ? r : 0] : expf(p[j0 + j]));
      }
      __syncthreads();
      const uint32_t j = j0 + threadIdx.x;
      if (j < b.K) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][threadIdx.x];
        if (!nsrc) atomicAdd(grads + (size_t)(b.c0 + j) * ld, v);
        for (uint32_t x = 0; x < nsrc; ++x) atomicAdd(grads + (size_t)(src[x] + j) * ld, v);
        if (b.d0 != PCB_NONE) atomicAdd(grads + (size_t)(b.d0 + j) * ld, v);
      }
    }
    KLD_T_EXIT();
    return;
  }
  const uint32_t i = (blockIdx.x - a.dense_ctas) * 8 + warp;
  if (i >= a.count) return;
  const uint32_t n = a.nodes[i], e0 = a.n_estart[n], cnt = a.n_ecount[n], pid0 = a.n_pid0[n];
  const bool issum = a.kind[n] == PCB_SUM;
  uint32_t pr[KLD_PRE], sb[KLD_PRE];
  float wgt[KLD_PRE];
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    const uint32_t j = lane + 32 * r;
    pr[r] = sb[r] = PCB_NONE; wgt[r] = 0.0f;
    if (j < cnt) {
      pr[r] = a.e_prime[e0 + j]; sb[r] = a.e_sub[e0 + j];
      wgt[r] = issum ? expf(a.p1[pid0 + j]) : 1.0f;
    }
    keep(pr[r]); keep(sb[r]); keep(wgt[r]);
  }
  pcb_grid_dep_wait();
  const float pg = grads[(size_t)n * ld];
#pragma unroll
  for (int r = 0; r < KLD_PRE; ++r) {
    if (pr[r] != PCB_NONE) atomicAdd(grads + (size_t)pr[r] * ld, pg * wgt[r]);
    if (sb[r] != PCB_NONE) atomicAdd(grads + (size_t)sb[r] * ld, pg * wgt[r]);
  }
  for (uint32_t j = lane + 32 * KLD_PRE; j < cnt; j += 32) {
    const float eg = issum ? pg * expf(a.p1[pid0 + j]) : pg;
    atomicAdd(grads + (size_t)a.e_prime[e0 + j] * ld, eg);
    if (a.e_sub[e0 + j] != PCB_NONE) atomicAdd(grads + (size_t)a.e_sub[e0 + j] * ld, eg);
  }
  KLD_T_EXIT();
}

// Gradient with respect to q's log-parameters, Adam descent and the re-normalisation in one pass for
// the fused step.  The normalised groups partition the parameters: blocks [0, sum_blocks) take one
// warp per sum node, the blocks after them the leaves (one thread per leaf with up to four
// categories, else one warp per leaf).  A sum edge's gradient is pg * (exp(a) * (kld(children) + a - b)
// + exp(a)) (queries/kld.jl:258-300 with merge_params, misc.jl:710-754), a leaf parameter's is
// g * (a - b + 1) (kld.jl:502-547); neither is stored.  Both parameter sets, both moments and the edge
// lists are fetched before the wait on the push kernels; groups of up to 128 stay in registers
// between the update and the scaling.
struct AdamArgs {
  float* theta; const float* theta_p; const float* klds; const float* grads; float* m; float* v;
  float lr, b1, b2, eps;
  const int* t_dev;
  uint32_t n_groups, sum_blocks, n_inputs, leaf_thread_mode, ld;
  uint64_t P;
  const uint32_t* grp_node; const uint4* s_node; const uint32_t* e_prime; const uint32_t* e_sub;
  const uint32_t* in_node; const uint32_t* in_cats; const uint64_t* in_poff;
};

__device__ __forceinline__ void adam_update(float& thv, float& mv, float& vv, float gi, float lr, float b1, float b2,
                                            float eps, float c1, float c2) {
  mv = b1 * mv + (1.0f - b1) * gi;
  vv = b2 * vv + (1.0f - b2) * gi * gi;
  const float m_hat = mv / c1, v_hat = vv / c2;
  thv += -lr * (m_hat / (sqrtf(v_hat) + eps));
}

template <bool SUM>
__device__ __forceinline__ void adam_group_warp(const AdamArgs& a, uint32_t node, uint32_t e0, uint32_t cnt, uint64_t off,
                                                uint32_t lane) {
  constexpr int R = 4;
  const bool renorm = !(SUM && cnt == 1);   // single-edge sum nodes are left alone (adam.jl:113)
  float th[R], mi[R], vi[R], dif[R];
  uint32_t pr[R], sb[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t j = lane + 32 * r;
    th[r] = mi[r] = vi[r] = dif[r] = 0.0f; pr[r] = sb[r] = PCB_NONE;
    if (j < cnt) {
      th[r] = a.theta[off + j]; mi[r] = a.m[off + j]; vi[r] = a.v[off + j];
      dif[r] = th[r] - a.theta_p[off + j];
      if (SUM) { pr[r] = a.e_prime[e0 + j]; sb[r] = a.e_sub[e0 + j]; }
    }
    keep(th[r]); keep(mi[r]); keep(vi[r]); keep(dif[r]);
    if (SUM) { keep(pr[r]); keep(sb[r]); }
  }
  pcb_grid_dep_wait();
  const float t = (float)*a.t_dev;
  const float pg = a.grads[(size_t)node * a.ld];
  float ck[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {   // the children's values of a sum group, all gathers in flight at once
    ck[r] = 0.0f;
    if (SUM) {
      const uint32_t a0 = pr[r] != PCB_NONE ? pr[r] : node, a1 = sb[r] != PCB_NONE ? sb[r] : a0;
      const float k0 = a.klds[(size_t)a0 * a.ld], k1 = a.klds[(size_t)a1 * a.ld];
      ck[r] = k0 + (sb[r] != PCB_NONE ? k1 : 0.0f);
    }
  }
  const float c1 = 1.0f - powf(a.b1, t), c2 = 1.0f - powf(a.b2, t);
  auto grad_of = [&](float av, float d, float kids) {
    if (!SUM) return pg * (d + 1.0f);
    const float ea = expf(av);
    return pg * (ea * (kids + d) + ea);
  };
  float total = 0.0f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t j = lane + 32 * r;
    if (j < cnt) {
      adam_update(th[r], mi[r], vi[r], grad_of(th[r], dif[r], ck[r]), a.lr, a.b1, a.b2, a.eps, c1, c2);
      a.m[off + j] = mi[r];
      a.v[off + j] = vi[r];
      total += expf(th[r]);
    }
  }
  for (uint32_t j = lane + 32 * R; j < cnt; j += 32) {   // the rare wide group goes through memory
    float tv = a.theta[off + j], mv = a.m[off + j], vv = a.v[off + j];
    float kids = 0.0f;
    if (SUM) {
      kids = a.klds[(size_t)a.e_prime[e0 + j] * a.ld];
      if (a.e_sub[e0 + j] != PCB_NONE) kids += a.klds[(size_t)a.e_sub[e0 + j] * a.ld];
    }
    adam_update(tv, mv, vv, grad_of(tv, tv - a.theta_p[off + j], kids), a.lr, a.b1, a.b2, a.eps, c1, c2);
    a.m[off + j] = mv; a.v[off + j] = vv; a.theta[off + j] = tv;
    total += expf(tv);
  }
  total = warp_sum(total);
  const float ls = renorm ? logf(total) : 0.0f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t j = lane + 32 * r;
    if (j < cnt) a.theta[off + j] = th[r] - ls;
  }
  if (renorm)
    for (uint32_t j = lane + 32 * R; j < cnt; j += 32) a.theta[off + j] -= ls;
}

__global__ void __launch_bounds__(256) adam_renorm_kernel(AdamArgs a) {
  KLD_T_ENTER();
  const uint32_t lane = threadIdx.x & 31;
  if (blockIdx.x < a.sum_blocks) {
    const uint32_t w = (blockIdx.x * 256 + threadIdx.x) >> 5;
    if (w >= a.n_groups) return;
    const uint32_t node = a.grp_node[w];
    const uint4 sn = a.s_node[node];
    adam_group_warp<true>(a, node, sn.x, sn.y, sn.z, lane);
  } else if (!a.leaf_thread_mode) {
    const uint32_t i = ((blockIdx.x - a.sum_blocks) * 256 + threadIdx.x) >> 5;
    if (i >= a.n_inputs) return;
    const uint64_t off = a.in_poff[i];
    if (off >= a.P) return;
    adam_group_warp<false>(a, a.in_node[i], 0, a.in_cats[i], off, lane);
  } else {
    // leaves with up to four categories: one thread each
    const uint32_t i = (blockIdx.x - a.sum_blocks) * 256 + threadIdx.x;
    if (i >= a.n_inputs) return;
    const uint64_t off = a.in_poff[i];
    if (off >= a.P) return;
    const uint32_t C = a.in_cats[i], node = a.in_node[i];
    float th[4], mi[4], vi[4], dif[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      th[k] = mi[k] = vi[k] = dif[k] = 0.0f;
      if (k < C) {
        th[k] = a.theta[off + k]; mi[k] = a.m[off + k]; vi[k] = a.v[off + k];
        dif[k] = th[k] - a.theta_p[off + k];
      }
      keep(th[k]); keep(mi[k]); keep(vi[k]); keep(dif[k]);
    }
    pcb_grid_dep_wait();
    const float t = (float)*a.t_dev;
    const float g = a.grads[(size_t)node * a.ld];
    const float c1 = 1.0f - powf(a.b1, t), c2 = 1.0f - powf(a.b2, t);
    float total = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < C) {
        adam_update(th[k], mi[k], vi[k], g * (dif[k] + 1.0f), a.lr, a.b1, a.b2, a.eps, c1, c2);
        a.m[off + k] = mi[k];
        a.v[off + k] = vi[k];
        total += expf(th[k]);
      }
    const float ls = logf(total);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < C) a.theta[off + k] = th[k] - ls;
  }
  KLD_T_EXIT();
}
}

#ifdef PCB_DIAG
// diagnostic builds only: the stamps of the last 256 kernels of the chain and the slot counter
extern "C" int32_t pcb_debug_kld_trace(unsigned long long* out, unsigned int* slot, int reset) {
  PCB_CUDA(cudaDeviceSynchronize());
  PCB_CUDA(cudaMemcpyFromSymbol(out, g_kld_trace, sizeof(unsigned long long) * 3 * 256));
  PCB_CUDA(cudaMemcpyFromSymbol(slot, g_kld_slot, sizeof(unsigned int)));
  if (reset) { unsigned int z = 0; PCB_CUDA(cudaMemcpyToSymbol(g_kld_slot, &z, sizeof(z))); }
  return PCB_OK;
}
#endif

static int32_t kld_adam_body(pcb_circuit* c, pcb_workspace* ws, float* theta_q, const float* theta_p, float* m_dev,
                             float* v_dev, float lr, float beta1, float beta2, float eps, float* kld_out, cudaStream_t st) {
  pcb_stream s = (pcb_stream)st;
  // the leaf kernel, first of the chain, counts the step and clears the node gradients
  ws->kld_bump = ws->kld_t_dev;
  int32_t r = pcb_kld(c, ws, theta_q, theta_p, 1, kld_out, s);
  ws->kld_bump = nullptr;
  if (r != PCB_OK) return r;
  for (uint32_t t = c->n_steps; t >= 1; --t) {
    KldLayer a = kld_layer(c, ws, theta_q, theta_p, 1, t);
    a.nodes = c->st_up + c->h_st_up_off[t];
    a.count = c->h_st_up_off[t + 1] - c->h_st_up_off[t];
    uint32_t R = 1, K = 1;
    pcb_step_extent(c, t, R, K);
    PCB_CUDA(kld_launch_warps(c, kld1_push_kernel, a, a.nblk, R, st));
  }
  if (c->P) {
    AdamArgs a;
    a.theta = theta_q; a.theta_p = theta_p; a.klds = ws->klds; a.grads = ws->grads; a.m = m_dev; a.v = v_dev;
    a.lr = lr; a.b1 = beta1; a.b2 = beta2; a.eps = eps; a.t_dev = ws->kld_t_dev;
    a.n_groups = c->n_groups; a.sum_blocks = (c->n_groups + 7) / 8; a.n_inputs = c->n_inputs;
    a.leaf_thread_mode = c->max_cats <= 4; a.ld = ws->ldS; a.P = c->P;
    a.grp_node = c->grp_node; a.s_node = c->s_node; a.e_prime = c->e_prime; a.e_sub = c->e_sub;
    a.in_node = c->in_node; a.in_cats = c->in_cats; a.in_poff = c->in_poff;
    const uint32_t leaf_blocks = a.leaf_thread_mode ? (c->n_inputs + 255) / 256 : (c->n_inputs + 7) / 8;
    ++c->prof.launches[PCB_K_KLD];
    PCB_CUDA(pcb_launch_pdl(adam_renorm_kernel, dim3(a.sum_blocks + leaf_blocks), dim3(256), 0, st, c->pdl, a));
  }
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

extern "C" int32_t pcb_kld_adam_step(pcb_circuit* c, pcb_workspace* ws, float* theta_q_dev, const float* theta_p_dev,
                                     float* m_dev, float* v_dev, int32_t t, float lr, float beta1, float beta2,
                                     float eps, float* kld_out_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws && theta_q_dev && theta_p_dev && m_dev && v_dev, "null argument");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  PCB_REQUIRE(t >= 1, "Adam step count starts at 1");
  PCB_CUDA(cudaSetDevice(c->device));
  int32_t st0 = pcb_ws_ensure_sets(ws, 1, PCB_WS_NODES);
  if (st0 != PCB_OK) return st0;
  cudaStream_t st = (cudaStream_t)s;
  if (!ws->kld_t_dev) {
    PCB_CUDA(cudaMalloc((void**)&ws->kld_t_dev, sizeof(int)));
    ws->kld_t_host = -1;
  }
  // the graph increments the device word itself; it is set from the host only when the caller's
  // count does not continue the last call's
  cudaStream_t gs = st;
  const bool legacy = st == nullptr || st == cudaStreamLegacy;
  if (legacy) {
    if (!c->gstream) {
      PCB_CUDA(cudaStreamCreateWithFlags(&c->gstream, cudaStreamNonBlocking));
      PCB_CUDA(cudaEventCreateWithFlags(&c->ev_g0, cudaEventDisableTiming));
      PCB_CUDA(cudaEventCreateWithFlags(&c->ev_g1, cudaEventDisableTiming));
    }
    gs = c->gstream;
    PCB_CUDA(cudaEventRecord(c->ev_g0, st));
    PCB_CUDA(cudaStreamWaitEvent(gs, c->ev_g0, 0));
  }
  auto leave = [&]() -> int32_t {
    if (legacy) { PCB_CUDA(cudaEventRecord(c->ev_g1, gs)); PCB_CUDA(cudaStreamWaitEvent(st, c->ev_g1, 0)); }
    return PCB_OK;
  };
  if (ws->kld_t_host != t - 1) set_step_kernel<<<1, 1, 0, gs>>>(ws->kld_t_dev, t - 1);
  ws->kld_t_host = t;

  pcb_workspace::KldKey key;
  memset(&key, 0, sizeof(key));
  key.q = theta_q_dev; key.p = theta_p_dev; key.m = m_dev; key.v = v_dev; key.out = kld_out_dev; key.stream = (void*)st;
  key.lr = lr; key.b1 = beta1; key.b2 = beta2; key.eps = eps;
  auto plain = [&]() -> int32_t {
    int32_t r = kld_adam_body(c, ws, theta_q_dev, theta_p_dev, m_dev, v_dev, lr, beta1, beta2, eps, kld_out_dev, gs);
    if (r != PCB_OK) return r;
    return leave();
  };
  if (!c->graph_enabled || c->prof.on) return plain();
  if (ws->kld_exec && !memcmp(&key, &ws->kld_exec_key, sizeof(key))) {
    PCB_CUDA(cudaGraphLaunch(ws->kld_exec, gs));
    for (int k = 0; k < PCB_K_COUNT; ++k) c->prof.launches[k] += ws->kld_launches[k];
    ws->have_kld = true; ws->kld_S = 1;
    return leave();
  }
  const bool capture = ws->have_kld_key && !memcmp(&key, &ws->kld_last_key, sizeof(key));
  ws->kld_last_key = key;
  ws->have_kld_key = true;
  if (!capture) return plain();
  if (ws->kld_exec) { cudaGraphExecDestroy(ws->kld_exec); ws->kld_exec = nullptr; }
  uint64_t before[PCB_K_COUNT];
  for (int k = 0; k < PCB_K_COUNT; ++k) before[k] = c->prof.launches[k];
  PCB_CUDA(cudaStreamBeginCapture(gs, cudaStreamCaptureModeRelaxed));
  int32_t body = kld_adam_body(c, ws, theta_q_dev, theta_p_dev, m_dev, v_dev, lr, beta1, beta2, eps, kld_out_dev, gs);
  cudaGraph_t graph = nullptr;
  cudaError_t ce = cudaStreamEndCapture(gs, &graph);
  if (body == PCB_OK && ce == cudaSuccess && graph) ce = cudaGraphInstantiate(&ws->kld_exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (body != PCB_OK || ce != cudaSuccess || !ws->kld_exec) {
    ws->kld_exec = nullptr;
    cudaGetLastError();
    c->graph_enabled = false;   // this chain does not capture: stay with plain launches
    for (int k = 0; k < PCB_K_COUNT; ++k) c->prof.launches[k] = before[k];
    if (body != PCB_OK) return body;
    return plain();
  }
  for (int k = 0; k < PCB_K_COUNT; ++k) ws->kld_launches[k] = c->prof.launches[k] - before[k];
  ws->kld_exec_key = key;
  PCB_CUDA(cudaGraphLaunch(ws->kld_exec, gs));
  return leave();
}
