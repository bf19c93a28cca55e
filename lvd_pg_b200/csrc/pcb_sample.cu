// pcb_sample.cu — top-down sampling.
//
//  * pcb_sample_hard: Gumbel-max walk.  At a sum node the lanes of a warp split the edges, the
//    arg-max of key = logp + g(u) (lowest index on ties) picks the edge; a product node passes all
//    its children on; a leaf does the same arg-max over its categories.  The keys that decide are
//    fp64 values of the shared host/device routine of include/pcb200_gumbel.h; an fp32 evaluation
//    with an error bound first removes the entries that cannot win (race, warp_select64).  One CTA per
//    sample takes the pending work of a round in parallel (sample_hard_cta_kernel, sample_hard_nodes_kernel); one warp per
//    sample with a stack (sample_hard_kernel) serves very wide circuits and the entry point that
//    allocates nothing.
//    This is the temperature -> 0 limit of the reference's relaxed sampler
//    (VariationalJuice.jl/src/queries/sample.jl:8-148,233-296), fed with caller-supplied
//    uniforms instead of the in-kernel rand(Float32) of sample.jl:45.
//  * pcb_sample_soft: the relaxed sampler itself — gumbel_params_down_kernel (sample.jl:8-58),
//    gumbel_sample_down_kernel (:60-148), gumbel_input_sample_down_kernel (:233-296).
#include <algorithm>
#include <mutex>

#include "../../include/pcb200_gumbel.h"
#include "pcb_internal.h"

namespace {

struct Shape2 {
  dim3 block, grid;
};
Shape2 shape_for(uint32_t S, uint32_t items) {
  const uint32_t bx = std::min(S, 32u), by = 128 / bx;   // consecutive threads take consecutive words
  Shape2 s;
  s.block = dim3(bx, by, 1);
  s.grid = dim3((items + by - 1) / by, (S + bx - 1) / bx, 1);
  return s;
}

__device__ __forceinline__ void warp_argmax(double& key, uint32_t& idx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double ok = __shfl_xor_sync(0xffffffffu, key, o);
    uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (oi != 0xffffffffu && (idx == 0xffffffffu || ok > key || (ok == key && oi < idx))) {
      key = ok;
      idx = oi;
    }
  }
}

// Arg-max of Gumbel keys with the same result as the fp64 arg-max above, bit for bit, at a fraction of its cost.  The
// key logp - log(-log x) is largest where the race time r = -log x * exp(-logp) is smallest; every entry's r is formed
// in fp32 with a relative bound eps on its distance from the exact one, and an entry whose lower bound lies above the
// smallest upper bound cannot win.  Almost always a single candidate is left and is the answer; otherwise the fp64
// keys of the candidates alone decide (lowest index on ties: an entry that dropped out takes no part in a tie).
// Bound: x = u (1 - 1e-6) + 1e-6 carries a relative error <= 2.4e-7, __logf an absolute error <= 3.6e-7 on [0.5, 2] and
// three ulp elsewhere, so inner = -log x is off by 6e-7 / inner + 4e-7; __expf by 2.4e-7 + 1.2e-7 |logp|, the product by
// 6e-8; eps is four times the sum.  Entries with inner below 1e-4 or exp(-logp) below 1e-30 have no bounds and always
// stay candidates (lower bound 0, upper bound infinity).  Where exp(-logp) or the product leaves the fp32 range the upper
// bound is infinity and the lower one that of 3e38.
__device__ __forceinline__ void race(float lp, float u, float& lo, float& hi) {
  const float inner = -__logf(fmaf(u, 0.999999f, 1e-6f)), inv = __expf(-lp), r = inner * fminf(inv, 3e38f), least = fminf(r, 3e38f);
  const float eps = __fdividef(2.4e-6f, inner) + 3.2e-6f + 5e-7f * fminf(fabsf(lp), 100.0f);
  const bool none = inner < 1e-4f || inv < 1e-30f;
  lo = none ? 0.0f : least - least * eps;
  hi = none || !(inv < 3e38f) ? INFINITY : r + r * eps;
}

__device__ __noinline__ uint32_t warp_exact64(float lp0, float u0, bool c0, float lp1, float u1, bool c1, uint32_t lane) {
  double best = 0.0;
  uint32_t bi = 0xffffffffu;
  if (c0) { best = pcb_gumbel_key(lp0, u0); bi = lane; }
  if (c1) {
    const double key = pcb_gumbel_key(lp1, u1);
    if (bi == 0xffffffffu || key > best) { best = key; bi = lane + 32; }
  }
  warp_argmax(best, bi);
  return bi;
}

// up to 64 entries, `lane` and `lane + 32` (v0, v1: they exist)
__device__ __forceinline__ uint32_t warp_select64(float lp0, float u0, bool v0, float lp1, float u1, bool v1, uint32_t lane,
                                                  bool exact) {
  float lo0 = INFINITY, hi0 = INFINITY, lo1 = INFINITY, hi1 = INFINITY;
  race(lp0, u0, lo0, hi0);
  race(lp1, u1, lo1, hi1);
  // non-negative floats order like their bits; an entry that does not exist, or is not a number, is the largest word
  const uint32_t best = __reduce_min_sync(0xffffffffu, min(v0 ? __float_as_uint(hi0) : 0xffffffffu, v1 ? __float_as_uint(hi1) : 0xffffffffu));
  const float top = __uint_as_float(best);
  bool c0 = v0 && (exact || lo0 <= top), c1 = v1 && (exact || lo1 <= top);
  uint32_t b0 = __ballot_sync(0xffffffffu, c0), b1 = __ballot_sync(0xffffffffu, c1);
  if (__popc(b0) + __popc(b1) == 1) return b0 ? (uint32_t)__ffs(b0) - 1u : 32u + (uint32_t)__ffs(b1) - 1u;
  if (!(b0 | b1)) { c0 = v0; c1 = v1; }   // nothing comparable
  return warp_exact64(lp0, u0, c0, lp1, u1, c1, lane);
}

// any number of entries: the bounds are formed twice rather than kept
template <typename LogP>
__device__ __forceinline__ uint32_t warp_select(LogP lp, const float* us, uint32_t n, uint32_t lane, bool exact) {
  uint32_t best = 0xffffffffu;
  for (uint32_t j = lane; j < n; j += 32) {
    float lo, hi;
    race(lp(j), us[j], lo, hi);
    best = min(best, __float_as_uint(hi));
  }
  const float top = __uint_as_float(__reduce_min_sync(0xffffffffu, best));
  uint32_t left = 0, last = 0;
  for (uint32_t j = lane; j < n; j += 32) {
    float lo, hi;
    race(lp(j), us[j], lo, hi);
    if (!exact && lo <= top) { ++left; last = j; }
  }
  const uint32_t total = __reduce_add_sync(0xffffffffu, left);
  if (total == 1) return __shfl_sync(0xffffffffu, last, __ffs(__ballot_sync(0xffffffffu, left)) - 1);
  double key = 0.0;
  uint32_t bi = 0xffffffffu;
  for (uint32_t j = lane; j < n; j += 32) {
    float lo, hi;
    race(lp(j), us[j], lo, hi);
    if (total && !(lo <= top)) continue;
    const double k = pcb_gumbel_key(lp(j), us[j]);
    if (bi == 0xffffffffu || k > key) { key = k; bi = j; }
  }
  warp_argmax(key, bi);
  return bi;
}

// status word: 0 ok, 1 stack overflow, 2 iteration limit (malformed circuit)
__global__ void sample_hard_kernel(uint32_t S, const float* __restrict__ params, uint32_t Sp,
                                   const float* __restrict__ u_sum, const float* __restrict__ u_leaf, uint32_t R,
                                   uint32_t kmax, uint32_t cmax, uint32_t V, uint32_t N,
                                   const uint8_t* __restrict__ kind, const uint32_t* __restrict__ n_estart,
                                   const uint32_t* __restrict__ n_ecount, const uint32_t* __restrict__ n_pid0,
                                   const uint32_t* __restrict__ n_region, const uint32_t* __restrict__ e_prime,
                                   const uint32_t* __restrict__ e_sub, const uint32_t* __restrict__ node2input,
                                   const uint32_t* __restrict__ in_var, const uint32_t* __restrict__ in_cats,
                                   const uint64_t* __restrict__ in_poff, uint64_t P,
                                   const float* __restrict__ theta, uint32_t* __restrict__ stack_all,
                                   uint32_t stack_cap, int32_t* __restrict__ x_out, int32_t* __restrict__ status,
                                   uint32_t smem_stack, const uint4* __restrict__ s_node,
                                   const uint4* __restrict__ s_leaf, bool exact) {
  extern __shared__ uint32_t sstack[];   // [warps per block][stack_cap] when smem_stack is set
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (s >= S) return;
  const size_t ps = Sp == 1 ? 0 : s, pld = Sp;
  // the walk pops and pushes once per visited node: with the stack in shared memory those are not
  // global round trips on the walk's dependent chain
  uint32_t* stack = smem_stack ? sstack + (size_t)(threadIdx.x >> 5) * stack_cap : stack_all + (size_t)s * stack_cap;
  for (uint32_t v = lane; v < V; v += 32) x_out[s + (size_t)S * v] = -1;
  uint32_t sp = 1;
  if (lane == 0) stack[0] = N - 1;
  __syncwarp();
  const uint32_t max_iter = 4u * N + 8u;
  for (uint32_t it = 0; sp > 0; ++it) {
    if (it >= max_iter) {
      if (lane == 0) atomicMax(status, 2);
      break;
    }
    uint32_t n = stack[--sp];
    __syncwarp();
    const uint4 nm = s_node[n];             // one load instead of kind / edge range / parameter id / region
    const uint8_t kd = (uint8_t)(nm.w & 3u);
    if (kd == PCB_INPUT) {
      uint32_t C = nm.y & 0xffffu, var = nm.y >> 16;
      uint64_t off = nm.x;
      if (nm.x == 0xffffffffu) {   // a leaf whose record did not fit the node's own
        const uint4 lm = s_leaf[nm.z];
        C = lm.z; var = lm.w;
        off = (uint64_t)lm.x | ((uint64_t)lm.y << 32);
      }
      const float* us = u_leaf + ((size_t)s * V + var) * cmax;
      uint32_t bi;
      // fixed leaves keep their log-probs in the circuit, not in the caller's parameter matrix
      if (C <= 64) {
        const bool v0 = lane < C, v1 = lane + 32 < C;
        auto lpa = [&](uint32_t c) { return off < P ? params[ps + pld * (off + c)] : theta[off + c]; };
        bi = warp_select64(v0 ? lpa(lane) : 0.0f, v0 ? us[lane] : 0.0f, v0, v1 ? lpa(lane + 32) : 0.0f,
                           v1 ? us[lane + 32] : 0.0f, v1, lane, exact);
      } else {
        bi = warp_select([&](uint32_t c) { return off < P ? params[ps + pld * (off + c)] : theta[off + c]; }, us, C, lane, exact);
      }
      if (lane == 0) x_out[s + (size_t)S * var] = (int32_t)bi;
    } else if (kd == PCB_PRODUCT) {
      uint32_t e0 = nm.x, cnt = nm.y;
      // count pushes first so that every lane keeps the same stack pointer
      uint32_t pushes = 0;
      for (uint32_t j = lane; j < cnt; j += 32) pushes += e_sub[e0 + j] != PCB_NONE ? 2 : 1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) pushes += __shfl_xor_sync(0xffffffffu, pushes, o);
      if (sp + pushes > stack_cap) {
        if (lane == 0) atomicMax(status, 1);
        break;
      }
      if (lane == 0) {
        uint32_t q = sp;
        for (uint32_t j = 0; j < cnt; ++j) {
          stack[q++] = e_prime[e0 + j];
          uint32_t sb = e_sub[e0 + j];
          if (sb != PCB_NONE) stack[q++] = sb;
        }
      }
      sp += pushes;
      __syncwarp();
    } else {
      uint32_t e0 = nm.x, cnt = nm.y, pid0 = nm.z;
      const float* us = u_sum + ((size_t)s * R + (nm.w >> 2)) * kmax;
      uint32_t bi;
      // the children of this lane's first two edges are fetched with the parameters, not after the
      // arg-max: one dependent load less on the walk's chain
      uint32_t pr0 = PCB_NONE, sb0 = PCB_NONE, pr1 = PCB_NONE, sb1 = PCB_NONE;
      if (lane < cnt) { pr0 = e_prime[e0 + lane]; sb0 = e_sub[e0 + lane]; }
      if (lane + 32 < cnt) { pr1 = e_prime[e0 + lane + 32]; sb1 = e_sub[e0 + lane + 32]; }
      if (cnt <= 64) {
        const bool v0 = lane < cnt, v1 = lane + 32 < cnt;
        bi = warp_select64(v0 ? params[ps + pld * (size_t)(pid0 + lane)] : 0.0f, v0 ? us[lane] : 0.0f, v0,
                           v1 ? params[ps + pld * (size_t)(pid0 + lane + 32)] : 0.0f, v1 ? us[lane + 32] : 0.0f, v1, lane, exact);
      } else {
        bi = warp_select([&](uint32_t j) { return params[ps + pld * (size_t)(pid0 + j)]; }, us, cnt, lane, exact);
      }
      uint32_t pr, sb;
      if (bi < 64) {
        const uint32_t src = bi & 31u;
        const uint32_t a = __shfl_sync(0xffffffffu, bi < 32 ? pr0 : pr1, src);
        const uint32_t b = __shfl_sync(0xffffffffu, bi < 32 ? sb0 : sb1, src);
        pr = a; sb = b;
      } else {
        pr = e_prime[e0 + bi]; sb = e_sub[e0 + bi];
      }
      uint32_t pushes = sb != PCB_NONE ? 2 : 1;
      if (sp + pushes > stack_cap) {
        if (lane == 0) atomicMax(status, 1);
        break;
      }
      if (lane == 0) {
        stack[sp] = pr;
        if (sb != PCB_NONE) stack[sp + 1] = sb;
      }
      sp += pushes;
      __syncwarp();
    }
  }
}

// The same walk with one CTA per sample: the pending nodes of a sample are roots of sub-circuits over disjoint scopes,
// so they are independent.  Pending work is a list of EDGES (two lists in shared memory, at most one entry per
// variable): a warp takes a piece of the round's list with one edge per lane, and the lanes fetch the children and their
// records together.  Leaves of few categories are decided by their lanes, each on its own; a product's edges go to the
// next round's list; the sum nodes of the piece are taken one after another by the whole warp, the parameters and noise
// of the next one on their way, and the edges they select reach the list with one counter update.  The selection is the
// same computation as in the one-warp walk, so the samples are the same bit for bit.  Bound: instruction issue (62%
// of the slots at 4096 samples) and the loads a visit depends on.  A warp per node, leaves included, with keys from two
// logarithms and a maximum by five shuffles: 4096 samples of 784 variables x 64 latents 1573 us, now 495 us (both alone
// on the GPU); the noise it must read (470 MB) is 72 us of HBM.
// CW: warps per sample.  One warp fills its lanes best and has nobody to wait for; where the samples alone do not fill
// the GPU, more warps shorten the walk of each.
constexpr uint32_t LANE_CATS = 8;               // categories up to which a leaf is decided by one lane
constexpr uint32_t ROOT_ENTRY = 0xffffffffu;    // the list entry that stands for the root

// one lane's leaf: C categories, at most LANE_CATS
__device__ __noinline__ uint32_t lane_exact(const float* lp, size_t pld, const float* us, uint32_t C, uint32_t keep) {
  double best = 0.0;
  uint32_t bi = 0xffffffffu;
  for (uint32_t c = 0; c < C; ++c) {
    if (!((keep >> c) & 1u)) continue;
    const double key = pcb_gumbel_key(lp[pld * c], us[c]);
    if (bi == 0xffffffffu || key > best) { best = key; bi = c; }
  }
  return bi;
}
__device__ __forceinline__ uint32_t lane_select(const float* lp, size_t pld, const float* us, uint32_t C, bool exact) {
  float lo[LANE_CATS], top = __uint_as_float(0x7f800000u);
  bool any = false;
#pragma unroll
  for (uint32_t c = 0; c < LANE_CATS; ++c) {
    float hi = INFINITY;
    lo[c] = INFINITY;
    if (c < C) {
      race(lp[pld * c], us[c], lo[c], hi);
      if (hi <= top) { top = hi; any = true; }
    }
  }
  uint32_t keep = 0;
#pragma unroll
  for (uint32_t c = 0; c < LANE_CATS; ++c)
    if (c < C && (exact || (any && lo[c] <= top))) keep |= 1u << c;
  if (__popc(keep) == 1) return (uint32_t)__ffs(keep) - 1u;
  return lane_exact(lp, pld, us, C, keep ? keep : (1u << C) - 1u);
}

template <uint32_t CW>
__global__ void __launch_bounds__(CW * 32, CW == 1 ? 32 : 40 / CW) sample_hard_cta_kernel(
    uint32_t S, const float* __restrict__ params, uint32_t Sp, const float* __restrict__ u_sum,
    const float* __restrict__ u_leaf, uint32_t R, uint32_t kmax, uint32_t cmax, uint32_t V, uint32_t N,
    const uint32_t* __restrict__ e_prime, const uint32_t* __restrict__ e_sub, uint64_t P, const float* __restrict__ theta,
    uint32_t cap, int32_t* __restrict__ x_out, int32_t* __restrict__ status, const uint4* __restrict__ s_node,
    const uint4* __restrict__ s_leaf, bool exact) {
  extern __shared__ uint32_t lists[];   // [2][cap]
  __shared__ uint32_t count[2];
  const uint32_t s = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t ps = Sp == 1 ? 0 : s, pld = Sp;
  if (threadIdx.x == 0) { lists[0] = ROOT_ENTRY; count[0] = 1; count[1] = 0; }
  __syncthreads();
  uint32_t cur = 0;
  for (uint32_t round = 0;; ++round) {
    const uint32_t n_cur = count[cur];
    if (n_cur == 0 || n_cur > cap) break;   // more than the list holds: the status word says so
    if (round > N + 8u) {   // a circuit is at most N levels deep
      if (threadIdx.x == 0) atomicMax(status, 2);
      break;
    }
    __syncthreads();                       // every thread has read the count
    if (threadIdx.x == 0) count[cur] = 0;  // this list is the next round's target after the one being filled
    uint32_t* const out = lists + (cur ^ 1u) * cap;
    uint32_t* const out_n = &count[cur ^ 1u];
    const uint32_t per = min(32u, (n_cur + CW - 1) / CW);   // edges of a warp's piece
    for (uint32_t base = warp * per; base < n_cur; base += CW * per) {
      const bool has = lane < per && base + lane < n_cur;
      const uint32_t entry = has ? lists[cur * cap + base + lane] : 0u;
      uint32_t prime = PCB_NONE, sub = PCB_NONE;
      if (has) {
        if (entry == ROOT_ENTRY) prime = N - 1;
        else { prime = e_prime[entry]; sub = e_sub[entry]; }
      }
#pragma unroll 1
      for (uint32_t half = 0; half < 2; ++half) {
        const uint32_t n = half ? sub : prime;
        const uint4 nm = n != PCB_NONE ? s_node[n] : make_uint4(0, 0, 0, 3u);
        const uint32_t kd = nm.w & 3u;
        if (kd == PCB_INPUT) {
          uint32_t C = nm.y & 0xffffu, var = nm.y >> 16;
          uint64_t off = nm.x;
          if (nm.x == 0xffffffffu) {
            const uint4 lm = s_leaf[nm.z];
            C = lm.z; var = lm.w;
            off = (uint64_t)lm.x | ((uint64_t)lm.y << 32);
          }
          if (C <= LANE_CATS) {
            // fixed leaves keep their log-probs in the circuit, not in the caller's parameter matrix
            const float* lp = off < P ? params + ps + pld * off : theta + off;
            x_out[s + (size_t)S * var] = (int32_t)lane_select(lp, off < P ? pld : 1, u_leaf + ((size_t)s * V + var) * cmax, C, exact);
          }
        } else if (kd == PCB_PRODUCT) {
          const uint32_t pos = atomicAdd(out_n, nm.y);
          if (pos + nm.y > cap) atomicMax(status, 1);
          else for (uint32_t j = 0; j < nm.y; ++j) out[pos + j] = nm.x + j;
        }
        // leaves of many categories: a warp each
        const uint32_t my_cats = kd != PCB_INPUT ? 0u : nm.x == 0xffffffffu ? s_leaf[nm.z].z : nm.y & 0xffffu;
        for (uint32_t m = __ballot_sync(0xffffffffu, my_cats > LANE_CATS); m; m &= m - 1) {
          const uint32_t src = (uint32_t)__ffs(m) - 1u;
          const uint32_t ex = __shfl_sync(0xffffffffu, nm.x, src), ey = __shfl_sync(0xffffffffu, nm.y, src), ez = __shfl_sync(0xffffffffu, nm.z, src);
          uint32_t C = ey & 0xffffu, var = ey >> 16;
          uint64_t off = ex;
          if (ex == 0xffffffffu) {
            const uint4 lm = s_leaf[ez];
            C = lm.z; var = lm.w;
            off = (uint64_t)lm.x | ((uint64_t)lm.y << 32);
          }
          const float* us = u_leaf + ((size_t)s * V + var) * cmax;
          auto lpa = [&](uint32_t c) { return off < P ? params[ps + pld * (off + c)] : theta[off + c]; };
          const uint32_t bi = warp_select(lpa, us, C, lane, exact);
          if (lane == 0) x_out[s + (size_t)S * var] = (int32_t)bi;
        }
        // sum nodes, the operands of the next one in flight
        uint32_t m = __ballot_sync(0xffffffffu, kd == PCB_SUM);
        if (!m) continue;
        const uint32_t sums = m, mine = __popc(m & ((1u << lane) - 1u));
        uint32_t picked = 0;
        float lp0 = 0.f, u0 = 0.f, lp1 = 0.f, u1 = 0.f;
        auto fetch = [&](uint32_t src) {
          const uint32_t cnt = __shfl_sync(0xffffffffu, nm.y, src), pid = __shfl_sync(0xffffffffu, nm.z, src);
          const uint32_t reg = __shfl_sync(0xffffffffu, nm.w, src) >> 2;
          const float* us = u_sum + ((size_t)s * R + reg) * kmax;
          const float* pp = params + ps + pld * (size_t)pid;
          if (lane < cnt) { lp0 = pp[pld * lane]; u0 = __ldcs(us + lane); }
          if (lane + 32 < cnt) { lp1 = pp[pld * (lane + 32)]; u1 = __ldcs(us + lane + 32); }
        };
        fetch((uint32_t)__ffs(m) - 1u);
        while (m) {
          const uint32_t src = (uint32_t)__ffs(m) - 1u;
          m &= m - 1;
          const uint32_t cnt = __shfl_sync(0xffffffffu, nm.y, src);
          const float a0 = lp0, b0 = u0, a1 = lp1, b1 = u1;
          if (m) fetch((uint32_t)__ffs(m) - 1u);
          uint32_t bi;
          if (cnt <= 64) {
            bi = warp_select64(a0, b0, lane < cnt, a1, b1, lane + 32 < cnt, lane, exact);
          } else {
            const uint32_t pid = __shfl_sync(0xffffffffu, nm.z, src), reg = __shfl_sync(0xffffffffu, nm.w, src) >> 2;
            bi = warp_select([&](uint32_t j) { return params[ps + pld * (size_t)(pid + j)]; }, u_sum + ((size_t)s * R + reg) * kmax, cnt, lane, exact);
          }
          if (lane == src) picked = nm.x + bi;
        }
        uint32_t pos = 0;
        if (lane == 0) pos = atomicAdd(out_n, (uint32_t)__popc(sums));
        pos = __shfl_sync(0xffffffffu, pos, 0);
        if (pos + __popc(sums) > cap) { if (lane == 0) atomicMax(status, 1); }
        else if ((sums >> lane) & 1u) out[pos + mine] = picked;
      }
    }
    __syncthreads();   // the next list is complete
    cur ^= 1u;
  }
}

// The same walk for deep circuits, whose rounds have fewer pending nodes than warps: a round's latency is all that counts.
// Pending work is a list of NODES (at most one per variable): the children of a sum node's edges come with its parameters
// and need no load of their own, and the two children of an edge go to different warps.  Edge lists against this way, 256
// samples: chain of 300 variables x 64 latents 906 -> 489 us, image trees of 768 x 16 latents 359 -> 293, 1500 x 32 705 -> 510.
// The children cost 512 bytes of L2 reads per visit, so wide circuits keep the edge lists (784 variables
// x 64 latents, 2000 samples 373 against 492 us).
template <uint32_t CW>
__global__ void __launch_bounds__(CW * 32, 32 / CW) sample_hard_nodes_kernel(
    uint32_t S, const float* __restrict__ params, uint32_t Sp, const float* __restrict__ u_sum,
    const float* __restrict__ u_leaf, uint32_t R, uint32_t kmax, uint32_t cmax, uint32_t V, uint32_t N,
    const uint32_t* __restrict__ e_prime, const uint32_t* __restrict__ e_sub, uint64_t P, const float* __restrict__ theta,
    uint32_t cap, int32_t* __restrict__ x_out, int32_t* __restrict__ status, const uint4* __restrict__ s_node,
    const uint4* __restrict__ s_leaf, bool exact) {
  extern __shared__ uint32_t lists[];   // [2][cap]
  __shared__ uint32_t count[2];
  const uint32_t s = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t ps = Sp == 1 ? 0 : s, pld = Sp;
  if (threadIdx.x == 0) { lists[0] = N - 1; count[0] = 1; count[1] = 0; }
  __syncthreads();
  uint32_t cur = 0;
  for (uint32_t round = 0;; ++round) {
    const uint32_t n_cur = count[cur];
    if (n_cur == 0 || n_cur > cap) break;   // more than the list holds: the status word says so
    if (round > N + 8u) {   // a circuit is at most N levels deep
      if (threadIdx.x == 0) atomicMax(status, 2);
      break;
    }
    __syncthreads();                       // every thread has read the count
    if (threadIdx.x == 0) count[cur] = 0;  // this list is the next round's target after the one being filled
    uint32_t* const out = lists + (cur ^ 1u) * cap;
    uint32_t* const out_n = &count[cur ^ 1u];
    const uint32_t per = min(32u, (n_cur + CW - 1) / CW);   // nodes of a warp's piece
    for (uint32_t base = warp * per; base < n_cur; base += CW * per) {
      const bool has = lane < per && base + lane < n_cur;
      const uint4 nm = has ? s_node[lists[cur * cap + base + lane]] : make_uint4(0, 0, 0, 3u);
      const uint32_t kd = nm.w & 3u;
      if (kd == PCB_INPUT) {
        uint32_t C = nm.y & 0xffffu, var = nm.y >> 16;
        uint64_t off = nm.x;
        if (nm.x == 0xffffffffu) {
          const uint4 lm = s_leaf[nm.z];
          C = lm.z; var = lm.w;
          off = (uint64_t)lm.x | ((uint64_t)lm.y << 32);
        }
        if (C <= LANE_CATS) {
          // fixed leaves keep their log-probs in the circuit, not in the caller's parameter matrix
          const float* lp = off < P ? params + ps + pld * off : theta + off;
          x_out[s + (size_t)S * var] = (int32_t)lane_select(lp, off < P ? pld : 1, u_leaf + ((size_t)s * V + var) * cmax, C, exact);
        }
      } else if (kd == PCB_PRODUCT) {
        for (uint32_t j = 0; j < nm.y; ++j) {
          const uint32_t pr = e_prime[nm.x + j], sb = e_sub[nm.x + j], kids = sb != PCB_NONE ? 2u : 1u;
          const uint32_t pos = atomicAdd(out_n, kids);
          if (pos + kids > cap) { atomicMax(status, 1); break; }
          out[pos] = pr;
          if (kids == 2) out[pos + 1] = sb;
        }
      }
      // leaves of many categories: a warp each
      const uint32_t my_cats = kd != PCB_INPUT ? 0u : nm.x == 0xffffffffu ? s_leaf[nm.z].z : nm.y & 0xffffu;
      for (uint32_t m = __ballot_sync(0xffffffffu, my_cats > LANE_CATS); m; m &= m - 1) {
        const uint32_t src = (uint32_t)__ffs(m) - 1u;
        const uint32_t ex = __shfl_sync(0xffffffffu, nm.x, src), ey = __shfl_sync(0xffffffffu, nm.y, src), ez = __shfl_sync(0xffffffffu, nm.z, src);
        uint32_t C = ey & 0xffffu, var = ey >> 16;
        uint64_t off = ex;
        if (ex == 0xffffffffu) {
          const uint4 lm = s_leaf[ez];
          C = lm.z; var = lm.w;
          off = (uint64_t)lm.x | ((uint64_t)lm.y << 32);
        }
        const float* us = u_leaf + ((size_t)s * V + var) * cmax;
        auto lpa = [&](uint32_t c) { return off < P ? params[ps + pld * (off + c)] : theta[off + c]; };
        const uint32_t bi = warp_select(lpa, us, C, lane, exact);
        if (lane == 0) x_out[s + (size_t)S * var] = (int32_t)bi;
      }
      // sum nodes, the operands of the next one and the children of its edges in flight
      uint32_t m = __ballot_sync(0xffffffffu, kd == PCB_SUM);
      if (!m) continue;
      const uint32_t sums = m, below = (1u << lane) - 1u;
      uint32_t prime = PCB_NONE, sub = PCB_NONE;
      float lp0 = 0.f, u0 = 0.f, lp1 = 0.f, u1 = 0.f;
      uint32_t pr0 = 0, sb0 = 0, pr1 = 0, sb1 = 0;
      auto fetch = [&](uint32_t src) {
        const uint32_t cnt = __shfl_sync(0xffffffffu, nm.y, src), pid = __shfl_sync(0xffffffffu, nm.z, src);
        const uint32_t reg = __shfl_sync(0xffffffffu, nm.w, src) >> 2, e0 = __shfl_sync(0xffffffffu, nm.x, src);
        const float* us = u_sum + ((size_t)s * R + reg) * kmax;
        const float* pp = params + ps + pld * (size_t)pid;
        if (lane < cnt) { lp0 = pp[pld * lane]; u0 = __ldcs(us + lane); pr0 = e_prime[e0 + lane]; sb0 = e_sub[e0 + lane]; }
        if (lane + 32 < cnt) {
          lp1 = pp[pld * (lane + 32)]; u1 = __ldcs(us + lane + 32);
          pr1 = e_prime[e0 + lane + 32]; sb1 = e_sub[e0 + lane + 32];
        }
      };
      fetch((uint32_t)__ffs(m) - 1u);
      while (m) {
        const uint32_t src = (uint32_t)__ffs(m) - 1u;
        m &= m - 1;
        const uint32_t cnt = __shfl_sync(0xffffffffu, nm.y, src);
        const float a0 = lp0, b0 = u0, a1 = lp1, b1 = u1;
        const uint32_t p0 = pr0, q0 = sb0, p1 = pr1, q1 = sb1;
        if (m) fetch((uint32_t)__ffs(m) - 1u);
        uint32_t bi;
        if (cnt <= 64) {
          bi = warp_select64(a0, b0, lane < cnt, a1, b1, lane + 32 < cnt, lane, exact);
        } else {
          const uint32_t pid = __shfl_sync(0xffffffffu, nm.z, src), reg = __shfl_sync(0xffffffffu, nm.w, src) >> 2;
          bi = warp_select([&](uint32_t j) { return params[ps + pld * (size_t)(pid + j)]; }, u_sum + ((size_t)s * R + reg) * kmax, cnt, lane, exact);
        }
        const uint32_t pr = __shfl_sync(0xffffffffu, bi < 32 ? p0 : p1, bi & 31u), sb = __shfl_sync(0xffffffffu, bi < 32 ? q0 : q1, bi & 31u);
        if (lane == src) {
          prime = bi < 64 ? pr : e_prime[nm.x + bi];
          sub = bi < 64 ? sb : e_sub[nm.x + bi];
        }
      }
      const uint32_t subs = __ballot_sync(0xffffffffu, sub != PCB_NONE), total = __popc(sums) + __popc(subs);
      uint32_t pos = 0;
      if (lane == 0) pos = atomicAdd(out_n, total);
      pos = __shfl_sync(0xffffffffu, pos, 0);
      if (pos + total > cap) { if (lane == 0) atomicMax(status, 1); }
      else if ((sums >> lane) & 1u) {
        pos += __popc(sums & below) + __popc(subs & below);
        out[pos] = prime;
        if (sub != PCB_NONE) out[pos + 1] = sub;
      }
    }
    __syncthreads();   // the next list is complete
    cur ^= 1u;
  }
}

// ---- relaxed sampling: exp((log p + gumbel) / T) of every sum edge, normalised per sum node ------------------
// The keys are formed in fp64 like the reference's (sample.jl:24-54 promotes through its Float64 literals), with
// logarithm and exponential by table and short polynomial (P. T. P. Tang, ACM TOMS 15 (1989) and 16 (1990)): the
// result is rounded to fp32 (6e-8), a hundred times the error of these series, and ten fp64 operations per logarithm
// replace the forty or more of one that is exact to the last bit.  Arguments outside the tables' range (u outside
// [0, 1), |z| >= 600, NaN) take the CUDA functions.  Instruction issue is the bound (66% of the slots, fp64 units at
// 28%): the checks of a pair of edges share one branch, the noise-free variant is a kernel of its own.
constexpr uint32_t SOFT_THREADS = 256;
// Every entry is there once for each lane of a half warp, so that lanes with different entries meet no bank twice (with
// one copy a lookup of 128 and 256 entries took three times the passes): 32 entries, and two more terms of the series.
constexpr uint32_t SOFT_COPIES = 16;
struct SoftTables {
  double rc[32][SOFT_COPIES], lg[32][SOFT_COPIES];   // 1/c and log c of 32 intervals of [sqrt(1/2), sqrt 2)
  double ex[32][SOFT_COPIES];                        // 2^(i/32)
};

__device__ __forceinline__ void soft_tables_fill(SoftTables* t) {
  const uint32_t i = threadIdx.x & 31;
  const double mid = __hiloint2double((int)(0x3fe6a09eu + (i << 15) + (1u << 14)), 0);
  // the interval around one keeps c = 1: log x is then the polynomial in x - 1 alone, relatively exact there
  const double rcp = i == 18 ? 1.0 : 1.0 / mid, lg = -log(rcp), ex = exp2((double)i / 32.0);
  for (uint32_t k = threadIdx.x >> 5; k < SOFT_COPIES; k += blockDim.x >> 5) { t->rc[i][k] = rcp; t->lg[i][k] = lg; t->ex[i][k] = ex; }
  __syncthreads();
}

// log of a positive normal double: |r| <= 2^-6 and the series ends after r^5, a relative 2e-10 at most
__device__ __forceinline__ double soft_log(double x, const SoftTables* t) {
  const int hi = __double2hiint(x), tmp = hi - 0x3fe6a09e, e = tmp >> 20;
  const double m = __hiloint2double(hi - (e << 20), __double2loint(x));
  const uint32_t i = (tmp >> 15) & 31, copy = threadIdx.x % SOFT_COPIES;
  const double r = fma(m, t->rc[i][copy], -1.0);
  const double q = fma(r, fma(r, fma(r, fma(r, 0.2, -0.25), 1.0 / 3.0), -0.5), 1.0);
  const double ed = __hiloint2double(0x43300000, e ^ (int)0x80000000) - (4503599627370496.0 + 2147483648.0);   // (double)e
  return fma(ed, 0.69314718055994530942, fma(r, q, t->lg[i][copy]));
}

// exp(z) rounded to fp32, |z| < 600: |r| <= ln2 / 64, the series ends after r^4, a relative 2e-12
__device__ __forceinline__ float soft_exp(double z, const SoftTables* t) {
  const double shift = 6755399441055744.0;   // 1.5 * 2^52: the sum's low word is the rounded integer
  const double s = fma(z, 32.0 / 0.69314718055994530942, shift);
  const int n = __double2loint(s);
  const double r = fma(s - shift, -0.69314718055994530942 / 32.0, z);
  const double p = fma(fma(fma(fma(r, 1.0 / 24.0, 1.0 / 6.0), r, 0.5), r, 1.0), r, 1.0) * t->ex[n & 31][threadIdx.x % SOFT_COPIES];
  return (float)__hiloint2double(__double2hiint(p) + ((n >> 5) << 20), __double2loint(p));
}

// the tables serve u in [0, 1), |z| < 600 and temperatures down to 1/512 (their noise is off by up to 3.6e-11, which the
// temperature divides: 1.9e-8 there, a third of the fp32 rounding of the weight); `ok` is cleared for anything else
constexpr double SOFT_TABLE_INV_T = 512.0;
__device__ __forceinline__ double soft_z_max(double inv_t) { return inv_t <= SOFT_TABLE_INV_T ? 600.0 : 0.0; }
template <bool NOISE>
__device__ __forceinline__ float soft_weight_fast(float logp, float u, double inv_t, double z_max, const SoftTables* t, bool& ok) {
  double g = 0.0;
  if (NOISE) {
    g = -soft_log(-soft_log(fma((double)u, 1.0 - 1e-6, 1e-6), t), t);
    ok = ok && __float_as_uint(u) < 0x3f800000u;
  }
  const double z = ((double)logp + g) * inv_t;
  ok = ok && fabs(z) < z_max;
  return soft_exp(z, t);
}
template <bool NOISE>
__device__ __noinline__ float soft_weight_any(float logp, float u, double inv_t) {
  double g = 0.0;
  if (NOISE) g = -log(-log(fma((double)u, 1.0 - 1e-6, 1e-6)));
  return (float)exp(((double)logp + g) * inv_t);
}
template <bool NOISE>
__device__ __forceinline__ float soft_weight(float logp, float u, double inv_t, double z_max, const SoftTables* t) {
  bool ok = true;
  const float e = soft_weight_fast<NOISE>(logp, u, inv_t, z_max, t, ok);
  return ok ? e : soft_weight_any<NOISE>(logp, u, inv_t);
}

// Threads are laid out (set, edge) with the set fastest, `rows` sum nodes per pass of a block; a thread keeps its up
// to eight edges in registers between the sum and the division, wider nodes go through memory.
template <bool NOISE>
__global__ void __launch_bounds__(SOFT_THREADS, 4) soft_params_kernel(
    float* __restrict__ w, uint32_t ld, uint32_t S, uint32_t St, uint32_t rows, const float* __restrict__ params,
    uint32_t Sp, const float* __restrict__ u, double inv_t, const uint32_t* __restrict__ grp_node, uint32_t n_groups,
    const uint32_t* __restrict__ n_pid0, const uint32_t* __restrict__ n_ecount) {
  __shared__ SoftTables tab;
  __shared__ float red[SOFT_THREADS];
  soft_tables_fill(&tab);
  const double z_max = soft_z_max(inv_t);
  const uint32_t s0 = blockIdx.y * St, sw = min(St, S - s0), J = SOFT_THREADS / St, JG = J / rows;
  const uint32_t q = threadIdx.x / St, s = threadIdx.x % St, r = q / JG, jg = q % JG;
  const bool lane_on = q < JG * rows && s < sw;
  const size_t ps = Sp == 1 ? 0 : s0 + s;
  for (uint32_t g0 = blockIdx.x * rows; g0 < n_groups; g0 += gridDim.x * rows) {
    const bool on = lane_on && g0 + r < n_groups;
    uint32_t pid0 = 0, cnt = 0;
    if (on) {
      const uint32_t n = grp_node[g0 + r];
      pid0 = n_pid0[n]; cnt = n_ecount[n];
    }
    const float* pp = params + ps + (size_t)Sp * pid0;
    const float* pu = NOISE ? u + s0 + s + (size_t)S * pid0 : nullptr;
    float* pw = w + (size_t)pid0 * ld + s0 + s;
    float x[8], y[8], sum = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      const uint32_t j = jg + k * JG;
      x[k] = j < cnt ? pp[(size_t)Sp * j] : 0.0f;
      y[k] = NOISE && j < cnt ? __ldcs(pu + (size_t)S * j) : 0.5f;
    }
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
      if (jg + k * JG < cnt) { x[k] = soft_weight<NOISE>(x[k], y[k], inv_t, z_max, &tab); sum += x[k]; }
    for (uint32_t j = jg + 8 * JG; j < cnt; j += JG) {
      const float e = soft_weight<NOISE>(pp[(size_t)Sp * j], NOISE ? pu[(size_t)S * j] : 0.5f, inv_t, z_max, &tab);
      pw[(size_t)ld * j] = e;
      sum += e;
    }
    red[threadIdx.x] = sum;
    __syncthreads();
    float total = 0.0f;
    if (on)
      for (uint32_t k = 0; k < JG; ++k) total += red[(r * JG + k) * St + s];
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
      if (jg + k * JG < cnt) pw[(size_t)ld * (jg + k * JG)] = x[k] / total;
    for (uint32_t j = jg + 8 * JG; j < cnt; j += JG) pw[(size_t)ld * j] /= total;
  }
}

// The same from row-major sets and noise ([S, P] and [S, edges] as a row-major host framework holds them): lanes over a
// node's edges, warps over the sets; the weights turn through shared memory into the [edge][set] order of the walk below.
// The next node's values are fetched while this one's are worked on.  A transposition of both matrices ahead of the
// column kernel cost 140 us at 24 x 1.7 M edges; this kernel takes 253 us (333 with tables that lanes share and without
// the prefetch, 312 with two branches an edge and a division in place of the product with a reciprocal in fp64), the
// column kernel 285 without the transpositions.
constexpr uint32_t SOFT_ROWS_K = 256;   // edges of a node that the tile holds
template <bool NOISE>
__global__ void __launch_bounds__(SOFT_THREADS, 3) soft_params_rows_kernel(
    float* __restrict__ w, uint32_t ld, uint32_t S, const float* __restrict__ params, uint64_t ss,
    const float* __restrict__ u, uint64_t us, double inv_t, const uint32_t* __restrict__ grp_node, uint32_t n_groups,
    const uint32_t* __restrict__ n_pid0, const uint32_t* __restrict__ n_ecount) {
  __shared__ SoftTables tab;
  __shared__ double inv_tot[32];
  extern __shared__ float soft_tile[];   // [edges of the widest node][33]
  soft_tables_fill(&tab);
  const double z_max = soft_z_max(inv_t);
  const uint32_t s0 = blockIdx.y * 32, sw = min(32u, S - s0), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float x[4][2], y[4][2], xn[4][2], yn[4][2];   // 64 edges of up to four sets a warp, and those of the next node
  const float* const mine = params + (s0 + warp) * ss + lane;   // this lane's edge of the warp's first set; further sets
  const float* const noise = u + (s0 + warp) * us + lane;       // eight rows on
  auto fetch = [&](float (&x)[4][2], float (&y)[4][2], uint32_t pid, uint32_t n) {   // n edges from pid
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      if (warp + 8 * k >= sw) break;
      const float* const px = mine + 8 * k * ss + pid;
      const float* const py = noise + 8 * k * us + pid;
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) {
        const bool in = lane + 32 * h < n;
        x[k][h] = in ? px[32 * h] : 0.0f;
        if (NOISE) y[k][h] = in ? __ldcs(py + 32 * h) : 0.5f;
      }
    }
  };
  uint32_t pid0 = 0, cnt = 0, pid1 = 0, cnt1 = 0;   // of this node and of the next one
  if (blockIdx.x < n_groups) { const uint32_t n = grp_node[blockIdx.x]; pid0 = n_pid0[n]; cnt = n_ecount[n]; }
  if (blockIdx.x + gridDim.x < n_groups) { const uint32_t n = grp_node[blockIdx.x + gridDim.x]; pid1 = n_pid0[n]; cnt1 = n_ecount[n]; }
  fetch(x, y, pid0, cnt);
  for (uint32_t g = blockIdx.x; g < n_groups; g += gridDim.x) {
    const uint32_t g2 = g + 2 * gridDim.x;
    const uint32_t n2 = g2 < n_groups ? grp_node[g2] : 0;
    fetch(xn, yn, pid1, cnt1);
    const uint32_t pid2 = g2 < n_groups ? n_pid0[n2] : 0, cnt2 = g2 < n_groups ? n_ecount[n2] : 0;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    for (uint32_t j0 = 0; j0 < cnt; j0 += 64) {
      if (j0) fetch(x, y, pid0 + j0, cnt - j0);
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
        if (warp + 8 * k >= sw) break;
        bool ok = true;
        float e[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) e[h] = soft_weight_fast<NOISE>(x[k][h], y[k][h], inv_t, z_max, &tab, ok);
        if (!ok)
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) e[h] = soft_weight<NOISE>(x[k][h], y[k][h], inv_t, z_max, &tab);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h)
          if (j0 + lane + 32 * h < cnt) {
            soft_tile[(j0 + lane + 32 * h) * 33 + warp + 8 * k] = e[h];
            sum[k] += e[h];
          }
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      if (warp + 8 * k >= sw) break;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
      if (lane == 0) inv_tot[warp + 8 * k] = 1.0 / (double)sum[k];
    }
    __syncthreads();
    const uint32_t step_j = SOFT_THREADS / sw, step_s = SOFT_THREADS % sw;   // 256 elements further in [edge][set] order
    uint32_t j = threadIdx.x / sw, s = threadIdx.x % sw;
    float* const out = w + (size_t)pid0 * ld + s0;
    while (j < cnt) {
      out[j * ld + s] = (float)((double)soft_tile[j * 33 + s] * inv_tot[s]);   // the quotient, rounded once
      j += step_j; s += step_s;
      if (s >= sw) { s -= sw; ++j; }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h) { x[k][h] = xn[k][h]; y[k][h] = yn[k][h]; }
    pid0 = pid1; cnt = cnt1; pid1 = pid2; cnt1 = cnt2;
  }
}

// One launch per step, from the root down: the dense blocks of the step above hand their probability to their children
// (and to the nodes that fused products multiply), the other nodes of the step pull from their parents (all parents were completed by earlier
// launches).  The weights of a CTA are copied into shared memory before the wait on the preceding launch, one private
// slot per thread and row; after it the parents' values are staged in one batch.  784 variables x 64 latents x 24
// samples: 993 -> 155 us over 20 layers (one thread walked all parents of a child before); 139 us over the 12 steps.
constexpr uint32_t SOFT_SLOTS = 40, SOFT_STAGE = 8 * SOFT_THREADS;

struct SoftLayer {
  float* td; const float* w;
  uint32_t ld, S, St, JC, per_blk, dense_ctas, slots;
  const PcbDenseBlock* blk; const uint32_t* src_list;
  const uint32_t* nodes; uint32_t count, root;
  const uint32_t* in_off; const PcbInEntry* in_ent;
};

__global__ void __launch_bounds__(SOFT_THREADS) soft_down_kernel(SoftLayer a) {
  extern __shared__ float park[];
  __shared__ float red[SOFT_THREADS];
  pcb_grid_dep_launch();
  const uint32_t s0 = blockIdx.y * a.St, sw = min(a.St, a.S - s0), J = SOFT_THREADS / a.St;
  const uint32_t q = threadIdx.x / a.St, s = threadIdx.x % a.St;
  if (blockIdx.x < a.dense_ctas) {
    const PcbDenseBlock b = a.blk[blockIdx.x / a.per_blk];
    const uint32_t JC = a.JC, IG = J / JC;
    const uint32_t jj = q % JC, ig = q / JC, j = blockIdx.x % a.per_blk * JC + jj;
    const bool on = ig < IG && s < sw && j < b.K;
    const float* base = a.w + ((size_t)b.pid0 + (on ? j : 0)) * a.ld + s0 + (on ? s : 0);
    const size_t step = (size_t)b.K * a.ld;
    float* const mine = park + threadIdx.x;
    float* const stage = park + (size_t)a.slots * SOFT_THREADS;
    if (on)
      for (uint32_t i = ig, m = 0; i < b.R && m < a.slots; i += IG, ++m) pcb_copy4_async(mine + m * SOFT_THREADS, base + i * step);
    pcb_grid_dep_wait();
    const uint32_t ci = SOFT_STAGE / a.St;
    float acc = 0.0f;
    uint32_t i = ig, m = 0;
    for (uint32_t c0 = 0; c0 < b.R; c0 += ci) {
      const uint32_t n = min(ci, b.R - c0);
      const float* tp = a.td + (size_t)(b.p0 + c0) * a.ld + s0 + s;
      float v[8];
      for (uint32_t g0 = q; g0 < n; g0 += 8 * J) {
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) v[k] = q < J && s < sw && g0 + k * J < n ? tp[(size_t)(g0 + k * J) * a.ld] : 0.0f;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
          if (q < J && s < sw && g0 + k * J < n) stage[(g0 + k * J) * a.St + s] = v[k];
      }
      if (c0 == 0) pcb_copies_wait();
      __syncthreads();
      if (on)
        for (; i < c0 + n; i += IG, ++m)
          acc += stage[(i - c0) * a.St + s] * (m < a.slots ? mine[m * SOFT_THREADS] : base[i * step]);
      if (c0 + ci < b.R) __syncthreads();
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    if (on && ig == 0) {
      float t = 0.0f;
      for (uint32_t k = 0; k < IG; ++k) t += red[threadIdx.x + k * JC * a.St];
      const uint32_t nsrc = b.src != PCB_NONE ? a.src_list[b.src] : 0;
      if (!nsrc) a.td[(size_t)(b.c0 + j) * a.ld + s0 + s] = t;
      for (uint32_t x = 0; x < nsrc; ++x) a.td[(size_t)(a.src_list[b.src + 1 + x] + j) * a.ld + s0 + s] = t;   // what the product hands on
      if (b.d0 != PCB_NONE) a.td[(size_t)(b.d0 + j) * a.ld + s0 + s] = t;
    }
    return;
  }
  const uint32_t k = (blockIdx.x - a.dense_ctas) * J + q;
  pcb_grid_dep_wait();
  if (q >= J || k >= a.count || s >= sw) return;
  const uint32_t n = a.nodes[k], i0 = a.in_off[n], i1 = a.in_off[n + 1];
  float acc = (i0 == i1 && n == a.root) ? 1.0f : 0.0f;
  for (uint32_t x = i0; x < i1; ++x) {
    const PcbInEntry en = a.in_ent[x];
    float tp = a.td[(size_t)en.parent * a.ld + s0 + s];
    if (en.pid != PCB_NONE) tp *= a.w[(size_t)en.pid * a.ld + s0 + s];
    acc += tp;
  }
  a.td[(size_t)n * a.ld + s0 + s] = acc;
}

__global__ void soft_leaf_kernel(const float* __restrict__ td, uint32_t ld, uint32_t S,
                                 const float* __restrict__ params, uint64_t ss, uint64_t pld, uint32_t n_inputs, uint32_t V,
                                 const uint32_t* __restrict__ in_node, const uint32_t* __restrict__ in_var,
                                 const uint32_t* __restrict__ in_cats, const uint64_t* __restrict__ in_poff,
                                 uint64_t P, const float* __restrict__ theta, float* __restrict__ out) {
  uint32_t i = blockIdx.x * blockDim.y + threadIdx.y;
  uint32_t s = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n_inputs || s >= S) return;
  const size_t ps = s * ss;   // parameter p of set s lies at s * ss + p * pld
  float tp = td[(size_t)in_node[i] * ld + s];
  uint32_t C = in_cats[i], var = in_var[i];
  uint64_t off = in_poff[i];
  for (uint32_t k = 0; k < C; ++k) {
    // fixed leaves keep their log-probs in the circuit, not in the caller's parameter matrix
    float lp = off < P ? params[ps + pld * (off + k)] : theta[off + k];
    atomicAdd(out + s + (size_t)S * (var + (size_t)V * k), tp * expf(lp));
  }
}

}  // namespace

extern "C" int32_t pcb_sample_hard(pcb_circuit* c, pcb_workspace* ws, const float* params_dev, uint32_t Sp,
                                   const float* u_sum_dev, const float* u_leaf_dev, uint32_t S, int32_t* x_out_dev,
                                   pcb_stream s) {
  PCB_REQUIRE(c && ws && params_dev && u_leaf_dev && x_out_dev, "null argument");
  PCB_REQUIRE(u_sum_dev || c->n_regions == 0, "u_sum missing");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  PCB_REQUIRE(S >= 1 && (Sp == 1 || Sp == S), "params must hold 1 or S parameter sets");
  PCB_CUDA(cudaSetDevice(c->device));
  // one CTA per sample keeps its lists in shared memory; only the one-warp walk of a very wide circuit
  // (or on request) needs stacks in global memory
  const bool cta_walk = (size_t)2 * (c->V + 2) * 4 <= 40 * 1024 && !c->sample_walk_warp;
  int32_t st0 = pcb_ws_ensure_sets(ws, S, cta_walk ? 0 : PCB_WS_STACK);
  if (st0 != PCB_OK) return st0;
  cudaStream_t st = (cudaStream_t)s;
  int32_t* status = ws->sample_status;
  PCB_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), st));
  if (cta_walk) {
    // one CTA per sample, its warps sharing the rounds of pending nodes
    PCB_CUDA(cudaMemsetAsync(x_out_dev, 0xff, (size_t)S * c->V * sizeof(int32_t), st));   // -1: a variable the walk does not reach
    ++c->prof.launches[PCB_K_SAMPLE];
    auto walk = [&](auto* kernel, uint32_t warps) {
      kernel<<<S, warps * 32, (size_t)2 * ws->stack_cap * 4, st>>>(
          S, params_dev, Sp, u_sum_dev, u_leaf_dev, c->n_regions, c->max_group, c->max_cats, c->V, c->N, c->e_prime, c->e_sub,
          c->P, c->theta, ws->stack_cap, x_out_dev, status, c->s_node, c->s_leaf, c->sample_exact_keys);
    };
    // Warps per sample by the samples that an SM holds at a time, of the call's or of those whose lists fit: 784 variables x
    // 64 latents, us with 1 / 2 / 4 / 8: 4096 samples 512 / 629 / 664 / 912, 2048 samples 412 / 367 / 407 / 494, 1024 samples
    // 396 / 295 / 243 / 320, 512 samples 376 / 269 / 199 / 187.  3072 variables leave nine: 3500 samples of an image tree
    // 13.9 ms with one warp each, 6.4 ms with several.  Up to sixteen variables per layer a circuit counts as deep.
    const uint32_t resident = std::min(S / 148, (uint32_t)(227 * 1024 / (2 * ws->stack_cap * 4 + 1088)));
    const bool deep = c->V <= 16 * c->L;
    if (resident >= 16) walk(sample_hard_cta_kernel<1>, 1);
    else if (resident >= 10) deep ? walk(sample_hard_nodes_kernel<2>, 2) : walk(sample_hard_cta_kernel<2>, 2);
    else if (resident >= (deep ? 4u : 5u)) deep ? walk(sample_hard_nodes_kernel<4>, 4) : walk(sample_hard_cta_kernel<4>, 4);   // CTAs of eight warps per SM
    else deep ? walk(sample_hard_nodes_kernel<8>, 8) : walk(sample_hard_cta_kernel<8>, 8);
    PCB_CUDA(cudaGetLastError());
    int32_t h0 = 0;
    PCB_CUDA(cudaMemcpyAsync(&h0, status, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    PCB_CUDA(cudaStreamSynchronize(st));
    if (h0 == 1) return pcb_fail(PCB_ERR_TOO_LARGE, "sampling walk overflowed its lists (circuit not decomposable?)");
    if (h0 == 2) return pcb_fail(PCB_ERR_INVALID, "sampling walk exceeded its round limit (malformed circuit)");
    return PCB_OK;
  }
  uint32_t warps_per_block = 4;
  while (warps_per_block > 1 && (size_t)warps_per_block * ws->stack_cap * 4 > 48 * 1024) warps_per_block /= 2;
  const size_t sm = (size_t)warps_per_block * ws->stack_cap * 4;
  const uint32_t smem_stack = sm <= 48 * 1024 ? 1u : 0u;
  ++c->prof.launches[PCB_K_SAMPLE];
  sample_hard_kernel<<<(S + warps_per_block - 1) / warps_per_block, warps_per_block * 32, smem_stack ? sm : 0, st>>>(
      S, params_dev, Sp, u_sum_dev, u_leaf_dev, c->n_regions, c->max_group, c->max_cats, c->V, c->N, c->kind,
      c->n_estart, c->n_ecount, c->n_pid0, c->n_region, c->e_prime, c->e_sub, c->node2input, c->in_var, c->in_cats,
      c->in_poff, c->P, c->theta, ws->stack, ws->stack_cap, x_out_dev, status, smem_stack, c->s_node, c->s_leaf,
      c->sample_exact_keys);
  PCB_CUDA(cudaGetLastError());
  int32_t h = 0;
  PCB_CUDA(cudaMemcpyAsync(&h, status, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  PCB_CUDA(cudaStreamSynchronize(st));
  if (h == 1) return pcb_fail(PCB_ERR_TOO_LARGE, "sampling walk overflowed its stack (circuit not decomposable?)");
  if (h == 2) return pcb_fail(PCB_ERR_INVALID, "sampling walk exceeded its iteration limit (malformed circuit)");
  return PCB_OK;
}

static int32_t sample_soft_impl(pcb_circuit* c, pcb_workspace* ws, const float* params_dev, uint32_t Sp,
                                const float* u_dev, float temperature, uint32_t S, float* out_dev, bool rows, pcb_stream s) {
  PCB_REQUIRE(c && ws && params_dev && out_dev, "null argument");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  PCB_REQUIRE(S >= 1 && (Sp == 1 || Sp == S), "params must hold 1 or S parameter sets");
  PCB_REQUIRE(temperature > 0.0f, "temperature must be positive");
  PCB_CUDA(cudaSetDevice(c->device));
  int32_t st0 = pcb_ws_ensure_sets(ws, S, PCB_WS_NODES | PCB_WS_EDGES);
  if (st0 != PCB_OK) return st0;
  cudaStream_t st = (cudaStream_t)s;
  const uint32_t ld = ws->ldS;
  ws->have_kld = false;  // the node gradients' rows hold the probabilities
  float* td = ws->grads;
  const uint32_t St = std::min(S, 32u), J = SOFT_THREADS / St, tiles = (S + St - 1) / St;
  PCB_CUDA(cudaMemsetAsync(out_dev, 0, (size_t)S * c->V * c->max_cats * sizeof(float), st));
  if (c->n_groups) {
    // about eight edges per thread: sum nodes that share a pass of a block
    const uint32_t pass = std::max(1u, std::min(J, J * 8 / std::max(1u, c->max_group)));
    const uint32_t passes = (c->n_groups + pass - 1) / pass;
    ++c->prof.launches[PCB_K_SAMPLE];
    if (rows)
      (u_dev ? soft_params_rows_kernel<true> : soft_params_rows_kernel<false>)<<<
          dim3(std::min(c->n_groups, std::max(1u, 148 * 3 / tiles)), tiles), SOFT_THREADS, c->max_group * 33 * sizeof(float), st>>>(
          ws->eprob, ld, S, params_dev, Sp == 1 ? 0 : c->P, u_dev, c->n_inner, 1.0 / (double)temperature, c->grp_node,
          c->n_groups, c->n_pid0, c->n_ecount);
    else (u_dev ? soft_params_kernel<true> : soft_params_kernel<false>)<<<dim3(std::min(passes, std::max(1u, 148 * 4 / tiles)), tiles), SOFT_THREADS, 0, st>>>(
        ws->eprob, ld, S, St, pass, params_dev, Sp, u_dev, 1.0 / (double)temperature, c->grp_node, c->n_groups,
        c->n_pid0, c->n_ecount);
  }
  static PcbPerDeviceOnce once;
  PCB_CUDA(once.run([&]() {
    return cudaFuncSetAttribute(soft_down_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)((SOFT_SLOTS * SOFT_THREADS + SOFT_STAGE) * sizeof(float)));
  }));
  bool chained = false;   // the first launch waits for the weights in full, the others for the launch before them
  SoftLayer a;
  a.td = td; a.w = ws->eprob; a.ld = ld; a.S = S; a.St = St; a.root = c->N - 1; a.in_off = c->in_off; a.in_ent = c->in_ent;
  a.src_list = c->src_list;
  for (int64_t t = c->n_steps; t >= 0; --t) {   // the blocks of step t + 1 and the other nodes of step t
    const uint32_t blocks = pcb_step_blocks(c, (uint32_t)t + 1);
    a.blk = blocks ? c->dense + c->h_dense_off[t + 1] : nullptr;
    a.nodes = c->st_down + c->h_st_down_off[t];
    a.count = c->h_st_down_off[t + 1] - c->h_st_down_off[t];
    if (!blocks && !a.count) continue;
    uint32_t R = 1, K = 1;
    pcb_step_extent(c, (uint32_t)t + 1, R, K);
    a.JC = std::min({std::max(1u, 64 / St), J, K});   // children of a CTA: runs of 256 bytes of weights
    a.per_blk = (K + a.JC - 1) / a.JC;
    a.slots = std::min(SOFT_SLOTS, (R + J / a.JC - 1) / (J / a.JC));
    a.dense_ctas = blocks * a.per_blk;
    ++c->prof.launches[PCB_K_SAMPLE];
    PCB_CUDA(pcb_launch_pdl(soft_down_kernel, dim3(a.dense_ctas + (a.count + J - 1) / J, tiles), dim3(SOFT_THREADS),
                            blocks ? (a.slots * SOFT_THREADS + SOFT_STAGE) * sizeof(float) : 0, st,
                            c->pdl && chained, a));
    chained = true;
  }
  if (c->n_inputs) {
    Shape2 sh = shape_for(S, c->n_inputs);
    ++c->prof.launches[PCB_K_SAMPLE];
    soft_leaf_kernel<<<sh.grid, sh.block, 0, st>>>(td, ld, S, params_dev, rows ? (Sp == 1 ? 0 : c->P) : (Sp == 1 ? 0 : 1), rows ? 1 : Sp, c->n_inputs, c->V, c->in_node, c->in_var,
                                                   c->in_cats, c->in_poff, c->P, c->theta, out_dev);
  }
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

extern "C" int32_t pcb_sample_soft(pcb_circuit* c, pcb_workspace* ws, const float* params_dev, uint32_t Sp,
                                   const float* u_dev, float temperature, uint32_t S, float* out_dev, pcb_stream s) {
  return sample_soft_impl(c, ws, params_dev, Sp, u_dev, temperature, S, out_dev, false, s);
}

extern "C" int32_t pcb_sample_soft_rows(pcb_circuit* c, pcb_workspace* ws, const float* params_dev, uint32_t Sp,
                                        const float* u_dev, float temperature, uint32_t S, float* out_dev, pcb_stream s) {
  PCB_REQUIRE(c && c->max_group <= SOFT_ROWS_K, "row-major sets: at most 256 edges per sum node");
  return sample_soft_impl(c, ws, params_dev, Sp, u_dev, temperature, S, out_dev, true, s);
}

// ---- conditioned top-down probabilities ------------------------------------------------------------------
// conditioned_td_prob (queries/td_prob.jl:161-291): the top-down pass with the circuit's own weights in
// which a marked inner node does not take what its parents send but node_probs[s, z_var, z_cat]; the
// leaves then spread their probability over their categories (gumbel_input_sample_down with the
// circuit's leaf parameters, queries/sample.jl:233-336).  As in the reference nothing starts at the
// root: an unmarked node without parents has probability 0.
namespace {
__global__ void cond_td_down_kernel(float* __restrict__ td, uint32_t ld, uint32_t S, const float* __restrict__ theta,
                                    const uint32_t* __restrict__ nodes, uint32_t count, const uint8_t* __restrict__ kind,
                                    const uint32_t* __restrict__ in_off, const PcbInEntry* __restrict__ in_ent,
                                    const int32_t* __restrict__ marked_var, const int32_t* __restrict__ marked_cat,
                                    const float* __restrict__ node_probs, uint32_t Z1) {
  uint32_t i = blockIdx.x * blockDim.y + threadIdx.y;
  uint32_t s = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= count || s >= S) return;
  const uint32_t n = nodes[i];
  float acc = 0.0f;
  if (kind[n] != PCB_INPUT && marked_var[n] > 0) {
    acc = node_probs[s + (size_t)S * ((uint32_t)(marked_var[n] - 1) + (size_t)Z1 * (uint32_t)(marked_cat[n] - 1))];
  } else {
    for (uint32_t x = in_off[n]; x < in_off[n + 1]; ++x) {
      const PcbInEntry en = in_ent[x];
      float tp = td[(size_t)en.parent * ld + s];
      if (en.pid != PCB_NONE) tp *= expf(__ldg(theta + en.pid));
      acc += tp;
    }
  }
  td[(size_t)n * ld + s] = acc;
}
}  // namespace

extern "C" int32_t pcb_cond_td_prob(pcb_circuit* c, pcb_workspace* ws, const int32_t* marked_var_dev,
                                    const int32_t* marked_cat_dev, const float* node_probs_dev, uint32_t S, uint32_t Z1,
                                    float* out_dev, pcb_stream s) {
  PCB_REQUIRE(c && ws && marked_var_dev && marked_cat_dev && node_probs_dev && out_dev, "null argument");
  PCB_REQUIRE(ws->c == c, "workspace belongs to another circuit");
  PCB_REQUIRE(S >= 1 && Z1 >= 1, "empty input");
  PCB_CUDA(cudaSetDevice(c->device));
  int32_t st0 = pcb_ws_ensure_sets(ws, S, PCB_WS_NODES);
  if (st0 != PCB_OK) return st0;
  cudaStream_t st = (cudaStream_t)s;
  const uint32_t ld = ws->ldS;
  ws->have_kld = false;   // the gradient rows are reused for the top-down probabilities
  float* td = ws->grads;
  PCB_CUDA(cudaMemsetAsync(out_dev, 0, (size_t)S * c->V * c->max_cats * sizeof(float), st));
  for (int64_t lay = c->L; lay >= 0; --lay) {
    uint32_t o0 = c->h_down_all_off[lay], o1 = c->h_down_all_off[lay + 1];
    if (o1 == o0) continue;
    Shape2 sh = shape_for(S, o1 - o0);
    ++c->prof.launches[PCB_K_SAMPLE];
    cond_td_down_kernel<<<sh.grid, sh.block, 0, st>>>(td, ld, S, c->theta, c->down_all + o0, o1 - o0, c->kind, c->in_off,
                                                      c->in_ent, marked_var_dev, marked_cat_dev, node_probs_dev, Z1);
  }
  if (c->n_inputs) {
    Shape2 sh = shape_for(S, c->n_inputs);
    ++c->prof.launches[PCB_K_SAMPLE];
    soft_leaf_kernel<<<sh.grid, sh.block, 0, st>>>(td, ld, S, c->theta, 0, 1, c->n_inputs, c->V, c->in_node, c->in_var,
                                                   c->in_cats, c->in_poff, c->P, c->theta, out_dev);
  }
  PCB_CUDA(cudaGetLastError());
  return PCB_OK;
}

// ---- hard sampling without any allocation --------------------------------------------------------------
// Some hosts of this library must not see it allocate device memory.  Julia's CUDA.jl, which is
// where the reference lives, keeps nearly all free device memory in its own pool, so a
// cudaMalloc issued behind its back can fail with memory "free" from Julia's point of view, and
// it synchronises the whole device under the caller's running streams; a serving loop that has
// already handed every byte to its own arena is in the same position.  pcb_sample_hard needs a
// workspace and grows it on demand; this variant keeps the per-sample walk stacks (and the
// status word the bounded walk reports to) in a fixed array that is part of the library image
// instead, so every GPU that loads the library holds PCB_STATIC_SAMPLE_WORDS * 4 bytes (4 MiB)
// of it until the process exits.
//
// The array is shared by all calls on a device and keeps whatever the last call left in it:
// stacks are written before they are read and the status word is cleared on the stream at the
// start of every call, but two calls whose kernels overlap on the GPU (different streams) race.
// A circuit with at most 12 286 variables keeps one warp's stack within 48 KB of shared memory and
// then only the status word of the array is used; larger circuits walk on the array itself.
// Like pcb_sample_hard the call ends by reading the status word back and waiting for the stream,
// so it cannot be made while that stream is being captured.
#define PCB_STATIC_SAMPLE_WORDS (1u << 20)
static __device__ __align__(256) uint32_t g_static_sample_scratch[PCB_STATIC_SAMPLE_WORDS + 64];

namespace {
constexpr int kMaxDevices = 64;
uint32_t* g_scratch_addr[kMaxDevices] = {nullptr};  // device address of the array, per device
std::mutex g_scratch_mutex;                          // host threads may make their first calls together

// In host code the array's name is only a handle for the runtime, not a device pointer: the
// address a kernel may use comes from cudaGetSymbolAddress, asked once per device while that
// device is current.
int32_t static_scratch(int device, uint32_t** out) {
  PCB_REQUIRE(device >= 0 && device < kMaxDevices, "device index beyond the static scratch table");
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_addr[device]) {
    uint32_t* p = nullptr;
    PCB_CUDA(cudaGetSymbolAddress((void**)&p, g_static_sample_scratch));
    g_scratch_addr[device] = p;
  }
  *out = g_scratch_addr[device];
  return PCB_OK;
}
}  // namespace

extern "C" int32_t pcb_sample_hard_static(pcb_circuit* c, const float* params_dev, uint32_t Sp,
                                          const float* u_sum_dev, const float* u_leaf_dev, uint32_t S,
                                          int32_t* x_out_dev, pcb_stream s) {
  PCB_REQUIRE(c && params_dev && u_leaf_dev && x_out_dev, "null argument");
  PCB_REQUIRE(u_sum_dev || c->n_regions == 0, "u_sum missing");
  PCB_REQUIRE(S >= 1 && (Sp == 1 || Sp == S), "params must hold 1 or S parameter sets");
  const uint64_t stack_cap = (uint64_t)c->V + 2;
  if ((uint64_t)S * stack_cap > PCB_STATIC_SAMPLE_WORDS)
    return pcb_fail(PCB_ERR_TOO_LARGE,
                    "pcb_sample_hard_static: S * (num_vars + 2) = " + std::to_string((uint64_t)S * stack_cap) +
                        " exceeds the static scratch of " + std::to_string(PCB_STATIC_SAMPLE_WORDS) +
                        " words; sample in smaller groups or use pcb_sample_hard");
  PCB_CUDA(cudaSetDevice(c->device));
  uint32_t* scratch = nullptr;
  int32_t st0 = static_scratch(c->device, &scratch);   // first call on a device resolves the symbol
  if (st0 != PCB_OK) return st0;
  cudaStream_t st = (cudaStream_t)s;
  int32_t* status = reinterpret_cast<int32_t*>(scratch + PCB_STATIC_SAMPLE_WORDS);
  PCB_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), st));
  uint32_t warps_per_block = 4;
  while (warps_per_block > 1 && (size_t)warps_per_block * stack_cap * 4 > 48 * 1024) warps_per_block /= 2;
  const size_t sm = (size_t)warps_per_block * stack_cap * 4;
  const uint32_t smem_stack = sm <= 48 * 1024 ? 1u : 0u;   // else the walk stacks stay in the static scratch
  ++c->prof.launches[PCB_K_SAMPLE];
  sample_hard_kernel<<<(S + warps_per_block - 1) / warps_per_block, warps_per_block * 32, smem_stack ? sm : 0, st>>>(
      S, params_dev, Sp, u_sum_dev, u_leaf_dev, c->n_regions, c->max_group, c->max_cats, c->V, c->N, c->kind,
      c->n_estart, c->n_ecount, c->n_pid0, c->n_region, c->e_prime, c->e_sub, c->node2input, c->in_var, c->in_cats,
      c->in_poff, c->P, c->theta, scratch, (uint32_t)stack_cap, x_out_dev, status, smem_stack, c->s_node, c->s_leaf,
      c->sample_exact_keys);
  PCB_CUDA(cudaGetLastError());
  int32_t h = 0;
  PCB_CUDA(cudaMemcpyAsync(&h, status, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  PCB_CUDA(cudaStreamSynchronize(st));
  if (h == 1) return pcb_fail(PCB_ERR_TOO_LARGE, "sampling walk overflowed its stack (circuit not decomposable?)");
  if (h == 2) return pcb_fail(PCB_ERR_INVALID, "sampling walk exceeded its iteration limit (malformed circuit)");
  return PCB_OK;
}
