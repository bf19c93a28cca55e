// pcb_mi.cu — pairwise mutual information of categorical columns (the input of Chow-Liu structure
// learning, the step before the circuit exists).
//
// Reference (paths relative to VariationalJuice.jl/src): pairwise_marginal_kernel, single_marginal_kernel,
// single_and_pairwise_marginal, pairwise_MI_chunked — utils/information.jl:3-157.  The reference
// counts co-occurrences with one global atomic per (example, variable pair), copies the [V, V, C, C]
// table to the host in chunks and forms MI there.
//
// Here the co-occurrence table is what it is algebraically: onehot(X)^T * onehot(X), a
// (V*C) x (V*C) x rows contraction of 0/1 bytes with 32-bit integer sums (tcgen05.mma.kind::i8, exact for every
// count), and it never leaves the SM.  A persistent CTA per SM walks the tiles of 128 x 256 (variable, category)
// rows on or above the diagonal:
//   * two groups of eight producer warps build the one-hot operands (K-major, 128-byte swizzle, 128 examples per
//     stage) in shared memory from the uint8 columns, a stage each at a time.  Up to 32 categories a thread turns 16
//     examples into the 16-byte pieces of four rows at a time (13 logic operations per four rows and word).  From 64
//     on an operand is almost all zeros: a warp takes the 128 examples of one variable, four per lane, clears the
//     bytes that the stage's last use had set and sets the new ones (byte stores to random rows conflict about three
//     ways, so below 64 categories whole lines are cheaper: 32 categories 28.7 against 22.9 ms).
//   * one thread issues the MMAs into one of two 128 x 256 accumulators (all 512 columns of tensor memory);
//   * eight epilogue warps turn the counts of the other accumulator into sum p log(p / (p_a p_b)) per variable pair
//     (the pseudocount spread over the table as in the reference) under the next tile's contraction.  The logarithm
//     of a smoothed count is looked up while all rows + 1 of them fit in shared memory (MAX_TABLE); with more rows every
//     cell takes a logf.
// Bound: no single unit.  Issue slots are 66% busy (producers and epilogue), the tensor pipe is active 38% of the time, the
// MMAs read 48 KB of shared memory per stage next to the byte stores.  3072 variables x 32 categories x 4096 rows, this
// kernel alone: 283 -> 22.9 ms, the whole call 23.6 - 26.2 ms with the clock (64 categories and more: 15.5 - 17.6 ms).
#include <algorithm>
#include <string>

#include "pcb_internal.h"
#include "pcb_tc.cuh"

namespace {

using namespace pcbtc;

constexpr uint32_t TM = 128, TN = 256;         // (variable, category) rows of the two operand tiles
constexpr uint32_t KCH = 128;                  // examples per stage: one 128-byte swizzled row of bytes
constexpr uint32_t A_BYTES = TM * KCH, STAGE_BYTES = (TM + TN) * KCH;
constexpr uint32_t STAGES = 3;
constexpr uint32_t NPW = 8, NPG = 2, NEW = 8;  // producer warps of a stage, their groups, epilogue warps
constexpr uint32_t MMA_WARP = NPW * NPG;
constexpr uint32_t NTHREADS = (MMA_WARP + 1 + NEW) * 32;
constexpr uint32_t SCATTER_CATS = 64;          // categories from which the operands are written byte by byte
static_assert((TM + TN) / SCATTER_CATS <= NPW, "one warp per variable of a stage");
constexpr uint32_t PREV_BYTES = STAGES * NPW * 128;  // the bytes that a stage holds, as the rows that were set
constexpr uint32_t MAX_TABLE = 8192;           // rows up to which probability and logarithm of all counts fit in shared memory
constexpr uint32_t SMEM_BASE = 1024 + STAGES * STAGE_BYTES + PREV_BYTES + 256;

__device__ __forceinline__ uint32_t idesc_u8(uint32_t m, uint32_t n) {
  // D s32, A and B u8, both K-major
  return (2u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void umma_u8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}

// counts of every (variable, category), then log of the smoothed marginal
__global__ void mi_hist_kernel(const uint8_t* __restrict__ data, uint64_t rows, uint32_t V, uint32_t C,
                               unsigned int* __restrict__ counts) {
  __shared__ unsigned int h[256];
  const uint32_t v = blockIdx.x;
  for (uint32_t i = threadIdx.x; i < C; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (uint64_t n = blockIdx.y * blockDim.x + threadIdx.x; n < rows; n += (uint64_t)gridDim.y * blockDim.x) {
    const uint32_t x = data[(size_t)v * rows + n];
    if (x < C) atomicAdd(h + x, 1u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < C; i += blockDim.x)
    if (h[i]) atomicAdd(counts + (size_t)v * C + i, h[i]);
}
// a category that never occurs and is not smoothed gets 0: it only meets cells whose count is 0 as well
__global__ void mi_logp_kernel(const unsigned int* __restrict__ counts, uint32_t n, float smooth, float z,
                               float* __restrict__ logp) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float p = ((float)counts[i] + smooth) / z;
  logp[i] = p > 0.0f ? logf(p) : 0.0f;
}

struct MiArgs {
  const uint8_t* data;    // [rows, V] column-major
  uint64_t rows;
  uint32_t V, C, lc, tm, tn, tiles, table;   // lc: log2 C; tm, tn: operand tiles; table: entries of the logarithm table or 0
  const float* logp;      // [V * C] log marginals
  float pair_smooth, z;   // pseudocount / C^2, rows + pseudocount
  float* mi;              // [V, V]
  int* status;
};

// column tj holds the tiles ti = 0 .. min(2 tj + 1, tm - 1)
__device__ __forceinline__ void tile_of(uint32_t idx, uint32_t& ti, uint32_t& tj) {
  tj = (uint32_t)((sqrtf(1.0f + 4.0f * (float)idx) - 1.0f) * 0.5f);
  while ((uint64_t)tj * (tj + 1) > idx) --tj;
  while ((uint64_t)(tj + 1) * (tj + 2) <= idx) ++tj;
  ti = idx - tj * (tj + 1);
}

// four consecutive examples of a column; `valid`: which of them exist
__device__ __forceinline__ uint32_t load4(const uint8_t* col, uint64_t n, uint64_t rows, bool aligned, uint32_t& valid) {
  valid = n >= rows ? 0u : rows - n >= 4 ? 15u : (1u << (uint32_t)(rows - n)) - 1u;
  if (valid == 15u && aligned) return __ldg(reinterpret_cast<const uint32_t*>(col + n));
  uint32_t w = 0;
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k)
    if ((valid >> k) & 1u) w |= (uint32_t)__ldg(col + n + k) << (8 * k);
  return w;
}
// sixteen, 255 past the end; where the address is odd, from the aligned words that hold a byte of the column
__device__ __forceinline__ uint4 load16(const uint8_t* col, uint64_t n, uint64_t rows, bool aligned16) {
  if (aligned16 && n + 16 <= rows) return __ldg(reinterpret_cast<const uint4*>(col + n));
  uint32_t w[5] = {0u, 0u, 0u, 0u, 0u};
  const uintptr_t at = reinterpret_cast<uintptr_t>(col + n), base = at & ~uintptr_t(3);
  const uint32_t here = n >= rows ? 0u : (uint32_t)min((uint64_t)16, rows - n), sh = (uint32_t)(at & 3) * 8;
#pragma unroll
  for (uint32_t k = 0; k < 5; ++k)
    if (here && base + 4 * k < at + here) w[k] = __ldg(reinterpret_cast<const uint32_t*>(base + 4 * k));
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    w[k] = __funnelshift_r(w[k], w[k + 1], sh);
    const uint32_t left = here > 4 * k ? min(4u, here - 4 * k) : 0u;
    if (left < 4) w[k] |= 0xffffffffu << (8 * left);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// byte of (tile row, example) in a K-major tile of 128-byte rows, 128-byte swizzle
__device__ __forceinline__ uint32_t byte_off(uint32_t row, uint32_t n) {
  return row * 128u + (((n >> 4) ^ (row & 7u)) << 4) + (n & 15u);
}
// per byte of x: o_r = 1 where the byte is r, for the two (four) rows r of a group
__device__ __forceinline__ void two_rows(uint32_t x, uint32_t& o0, uint32_t& o1) {
  const uint32_t m = (~(((x >> 1) & 0x7f7f7f7fu) + 0x7f7f7f7fu) >> 7) & 0x01010101u;   // bytes below two
  o1 = x & m;
  o0 = m & ~x;
}
__device__ __forceinline__ void four_rows(uint32_t x, uint32_t& o0, uint32_t& o1, uint32_t& o2, uint32_t& o3) {
  const uint32_t m = (~(((x >> 2) & 0x3f3f3f3fu) + 0x7f7f7f7fu) >> 7) & 0x01010101u;   // bytes below four
  const uint32_t lo = x & m, hi = (x >> 1) & m;
  o0 = m & ~(lo | hi);
  o1 = lo & ~hi;
  o2 = hi & ~lo;
  o3 = lo & hi;
}

// LANES: categories, 32 at most (lanes of the accumulator that share a variable); SCATTER: the operands are written
// byte by byte (64 categories and more, six variables per stage at most)
template <uint32_t LANES, bool SCATTER>
__global__ void __launch_bounds__(NTHREADS, 1) mi_tile_kernel(MiArgs a) {
  constexpr uint32_t SEG = LANES < 16 ? LANES : 16;   // columns of a 16-column piece that share a variable
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint32_t* prev = reinterpret_cast<uint32_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + PREV_BYTES);   // [STAGES] operands written
  uint64_t* empty = full + STAGES;                     // [STAGES] the MMAs that read a stage are done
  uint64_t* accfull = empty + STAGES;                  // [2] counts of a tile complete
  uint64_t* accempty = accfull + 2;                    // [2] counts of a tile read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accempty + 2);
  float2* table = reinterpret_cast<float2*>(smem + STAGES * STAGE_BYTES + PREV_BYTES + 256);

  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (uint32_t s = 0; s < STAGES; ++s) { mbar_init(&full[s], NPW); mbar_init(&empty[s], 1); }
    for (uint32_t s = 0; s < 2; ++s) { mbar_init(&accfull[s], 1); mbar_init(&accempty[s], NEW); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (uint32_t i = tid; i < STAGES * STAGE_BYTES / 16; i += NTHREADS) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
  for (uint32_t i = tid; i < a.table; i += NTHREADS) {
    const float p = ((float)i + a.pair_smooth) / a.z;
    table[i] = make_float2(p, p > 0.0f ? logf(p) : 0.0f);
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t nchunks = (uint32_t)((a.rows + KCH - 1) / KCH);
  const uint32_t total_rows = a.V * a.C;
  bool ok = true;

  if (warp < MMA_WARP) {
    // =========================== producers =======================================================
    const bool aligned = ((reinterpret_cast<uintptr_t>(a.data) | a.rows) & 3) == 0;
    const bool aligned16 = ((reinterpret_cast<uintptr_t>(a.data) | a.rows) & 15) == 0;
    // group g of producers takes the stages it = g, g + NPG, ...: two stages are written at a time.  The data of a
    // group's next stage is on its way while this one is written.
    const uint32_t wg = warp % NPW, ptid = wg * 32 + lane;
    const uint64_t total = (uint64_t)((a.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) * nchunks;
    uint32_t ti = 0, tj = 0, i1 = warp / NPW, t1 = blockIdx.x;
    bool moved = true;
    // scatter: unit wg of a stage is one variable of the A tile (wg < ua) or of the B tile; with more categories than
    // tile rows the tile covers a part of the variable's categories
    const uint32_t ua = max(1u, TM >> a.lc), ub = max(1u, TN >> a.lc);
    const bool on_a = wg < ua;
    const uint32_t size = on_a ? TM : TN, local = (on_a ? wg : wg - ua) << a.lc;   // first tile row of the variable
    uint32_t first = 0, w = 0, valid = 0;
    // full: item m of a thread is 16 examples (k8) of the four rows 4 * (m * 32 + ptid / 8); with two categories those
    // are two variables
    constexpr uint32_t ITEMS = SCATTER ? 1 : (TM + TN) / 4 * 8 / (NPW * 32), VARS = LANES == 2 ? 2 : 1;
    const uint32_t k8 = ptid & 7u;
    uint4 x[ITEMS][VARS];
    auto fetch = [&]() {
      while (i1 >= nchunks) { i1 -= nchunks; t1 += gridDim.x; moved = true; }
      if (t1 >= a.tiles) return;
      if (moved) { tile_of(t1, ti, tj); moved = false; }
      const uint64_t n0 = (uint64_t)i1 * KCH;
      if constexpr (SCATTER) {
        const uint32_t v = ((on_a ? ti * TM : tj * TN) + local) >> a.lc;
        w = valid = 0;
        first = (on_a ? ti * TM : tj * TN) & (a.C - 1);
        if (wg < ua + ub && v < a.V) w = load4(a.data + (size_t)v * a.rows, n0 + 4 * lane, a.rows, aligned, valid);
      } else {
        const uint64_t n = n0 + 16 * k8;
#pragma unroll
        for (uint32_t m = 0; m < ITEMS; ++m)
#pragma unroll
          for (uint32_t y = 0; y < VARS; ++y) {
            const uint32_t row = 4 * (m * (NPW * 4) + (ptid >> 3)) + 2 * y;
            const uint32_t r = row < TM ? ti * TM + row : tj * TN + (row - TM);
            x[m][y] = r < total_rows ? load16(a.data + (size_t)(r >> a.lc) * a.rows, n, a.rows, aligned16)
                                     : make_uint4(~0u, ~0u, ~0u, ~0u);
          }
      }
    };
    fetch();
    for (uint64_t it = warp / NPW; it < total && ok; it += NPG) {
      const uint32_t s = (uint32_t)(it % STAGES), ph = (uint32_t)(it / STAGES) & 1u;
      uint8_t* st = smem + s * STAGE_BYTES;
      const bool got = lane != 0 || mbar_wait(&empty[s], ph ^ 1u, a.status);
      ok = __all_sync(0xffffffffu, got);
      if (!ok) break;
      if constexpr (SCATTER) {
        const uint32_t word = w, mask = valid, base = first;
        i1 += NPG;
        fetch();
        if (wg < ua + ub) {
          uint8_t* op = on_a ? st : st + A_BYTES;
          uint32_t* const pw = prev + (s * NPW + wg) * 32 + lane;
          // this lane owns the bytes of its four examples in the rows of this variable: it clears the ones it set in
          // the stage's last use (an example without a byte is kept as the variable's first row)
          if (it >= STAGES) {
            const uint32_t old = *pw;
#pragma unroll
            for (uint32_t b = 0; b < 4; ++b) op[byte_off((old >> (8 * b)) & 255u, 4 * lane + b)] = 0;
          }
          uint32_t now = 0;
#pragma unroll
          for (uint32_t b = 0; b < 4; ++b) {
            const uint32_t c = (word >> (8 * b)) & 255u, row = local + c - base;
            const bool set = ((mask >> b) & 1u) && c < a.C && c >= base && row < size;
            if (set) op[byte_off(row, 4 * lane + b)] = 1;
            now |= (set ? row : local) << (8 * b);
          }
          *pw = now;
        }
      } else {
#pragma unroll
        for (uint32_t m = 0; m < ITEMS; ++m) {
          const uint32_t row = 4 * (m * (NPW * 4) + (ptid >> 3));
          uint4 o[4];
          if constexpr (LANES == 2) {
            two_rows(x[m][0].x, o[0].x, o[1].x); two_rows(x[m][0].y, o[0].y, o[1].y);
            two_rows(x[m][0].z, o[0].z, o[1].z); two_rows(x[m][0].w, o[0].w, o[1].w);
            two_rows(x[m][VARS - 1].x, o[2].x, o[3].x); two_rows(x[m][VARS - 1].y, o[2].y, o[3].y);
            two_rows(x[m][VARS - 1].z, o[2].z, o[3].z); two_rows(x[m][VARS - 1].w, o[2].w, o[3].w);
          } else {
            const uint32_t cat = (row & (LANES - 1)) * 0x01010101u;   // tiles start at a multiple of the categories
            four_rows(x[m][0].x ^ cat, o[0].x, o[1].x, o[2].x, o[3].x); four_rows(x[m][0].y ^ cat, o[0].y, o[1].y, o[2].y, o[3].y);
            four_rows(x[m][0].z ^ cat, o[0].z, o[1].z, o[2].z, o[3].z); four_rows(x[m][0].w ^ cat, o[0].w, o[1].w, o[2].w, o[3].w);
          }
          uint8_t* op = row < TM ? st : st + A_BYTES;
          const uint32_t tr = row < TM ? row : row - TM;
#pragma unroll
          for (uint32_t r = 0; r < 4; ++r) *reinterpret_cast<uint4*>(op + byte_off(tr + r, 16 * k8)) = o[r];
        }
        i1 += NPG;
        fetch();
      }
      fence_proxy_async();   // generic-proxy writes -> visible to the tensor core
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
    }
  } else if (warp == MMA_WARP) {
    // =========================== MMA issuer ======================================================
    if (lane == 0) {
      const uint32_t idesc = idesc_u8(TM, TN);
      uint32_t it = 0, tc = 0;
      for (uint32_t t = blockIdx.x; t < a.tiles && ok; t += gridDim.x, ++tc) {
        const uint32_t buf = tc & 1u;
        ok = mbar_wait(&accempty[buf], ((tc >> 1) & 1u) ^ 1u, a.status);
        if (!ok) break;
        tc_fence_after();
        for (uint32_t i = 0; i < nchunks; ++i, ++it) {
          const uint32_t s = it % STAGES;
          ok = mbar_wait(&full[s], (it / STAGES) & 1u, a.status);
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = make_desc(smem_u32(smem + s * STAGE_BYTES)), db = make_desc(smem_u32(smem + s * STAGE_BYTES + A_BYTES));
#pragma unroll
          for (uint32_t ks = 0; ks < KCH / 32; ++ks)   // 32 examples = 32 bytes along the swizzled row
            umma_u8(tmem_base + buf * TN, da + ks * 2u, db + ks * 2u, idesc, (i | ks) ? 1u : 0u);
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(&accfull[buf]);
      }
    }
    __syncwarp();
  } else {
    // =========================== epilogue ========================================================
    const uint32_t quad = warp & 3u, half = (warp - MMA_WARP - 1) >> 2;   // a warp reads the 32 lanes its number selects
    uint32_t tc = 0;
    for (uint32_t t = blockIdx.x; t < a.tiles && ok; t += gridDim.x, ++tc) {
      uint32_t ti, tj;
      tile_of(t, ti, tj);
      const uint32_t buf = tc & 1u;
      const bool got = lane != 0 || mbar_wait(&accfull[buf], (tc >> 1) & 1u, a.status);
      ok = __all_sync(0xffffffffu, got);
      if (!ok) break;
      tc_fence_after();
      const uint32_t ra = ti * TM + quad * 32 + lane, v1 = ra >> a.lc;
      const bool va = ra < total_rows;
      const float lpa = va ? a.logp[ra] : 0.0f;
      float run = 0.0f;   // the pair's sum over the columns so far
#pragma unroll 1
      for (uint32_t c0 = 0; c0 < TN / 2; c0 += 16) {
        uint32_t count[16];
        const uint32_t col = tj * TN + half * (TN / 2) + c0;
        float4 lb[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) lb[k] = __ldg(reinterpret_cast<const float4*>(a.logp + col) + k);   // padded to whole tiles
        tmem_ld16(tmem_base + ((quad * 32u) << 16) + buf * TN + half * (TN / 2) + c0, count);
        const float* lpb = reinterpret_cast<const float*>(lb);
#pragma unroll
        for (uint32_t g = 0; g < 16; g += SEG) {
          const uint32_t cg = col + g, v2 = cg >> a.lc;
          const bool vcol = cg < total_rows;
          float part = 0.0f;
          if (a.table) {
#pragma unroll
            for (uint32_t k = 0; k < SEG; ++k) {
              const float2 e = table[count[g + k]];
              part = fmaf(e.x, e.y - lpa - lpb[g + k], part);
            }
          } else {
#pragma unroll
            for (uint32_t k = 0; k < SEG; ++k) {
              const float p = ((float)count[g + k] + a.pair_smooth) / a.z;
              part = fmaf(p, (p > 0.0f ? logf(p) : 0.0f) - lpa - lpb[g + k], part);
            }
          }
          if (SEG == 16) {   // the next columns may share v2
            run += part;
            if (((cg + 16) & (a.C - 1)) && c0 + 16 < TN / 2) continue;
            part = run;
            run = 0.0f;
          }
          if (!va) part = 0.0f;
#pragma unroll
          for (uint32_t o = LANES >> 1; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
          if ((lane & (LANES - 1)) == 0 && va && vcol && v1 <= v2) {
            float* const out = a.mi + (size_t)v1 * a.V + v2;
            float* const mirror = a.mi + (size_t)v2 * a.V + v1;
            if (a.C <= 32) {   // the pair lies in this warp alone
              *out = part;
              *mirror = part;
            } else {
              atomicAdd(out, part);
              if (v1 != v2) atomicAdd(mirror, part);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&accempty[buf]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Scratch comes stream-ordered from a pool of the library's own that keeps at most 4 MB between calls: an allocation
// and a release by the driver cost 0.8 ms per call, more than the whole call on a hundred variables.
cudaError_t mi_pool(int dev, cudaMemPool_t* pool) {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  std::lock_guard<std::mutex> g(mu);
  cudaMemPool_t& p = pools[dev & 63];
  if (!p) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaError_t e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) { p = nullptr; return e; }
    uint64_t keep = 4ull << 20;
    e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) return e;
  }
  *pool = p;
  return cudaSuccess;
}

}  // namespace

extern "C" int32_t pcb_pairwise_mi(const uint8_t* data_dev, uint64_t num_rows, uint32_t num_vars, uint32_t num_cats,
                                   float pseudocount, float* mi_dev, pcb_stream s) {
  PCB_REQUIRE(data_dev && mi_dev, "null argument");
  PCB_REQUIRE(num_rows >= 1 && num_rows < (1ull << 24), "row count must be below 2^24 (counts are exact in fp32 up to there)");
  PCB_REQUIRE(num_vars >= 1 && num_cats >= 2 && num_cats <= 256 && (num_cats & (num_cats - 1)) == 0,
              "the number of categories must be a power of two between 2 and 256");
  PCB_REQUIRE(pseudocount >= 0.0f, "negative pseudocount");
  int dev = 0, major = 0, sms = 0;
  PCB_CUDA(cudaGetDevice(&dev));
  PCB_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
  PCB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (major != 10)
    return pcb_fail(PCB_ERR_INVALID, "pairwise MI needs an sm_100 device (tcgen05)");
  cudaStream_t st = (cudaStream_t)s;
  const uint32_t VC = num_vars * num_cats;
  MiArgs a;
  a.data = data_dev; a.rows = num_rows; a.V = num_vars; a.C = num_cats; a.mi = mi_dev;
  a.lc = 0;
  while ((1u << a.lc) < num_cats) ++a.lc;
  a.tm = (VC + TM - 1) / TM; a.tn = (VC + TN - 1) / TN;
  const uint64_t tiles = (uint64_t)a.tn * (a.tn - 1) + a.tm;   // the last column ends at the last row tile
  if (tiles > 0x7fffffffull) return pcb_fail(PCB_ERR_INVALID, "pairwise MI: too many tiles for one launch");
  a.tiles = (uint32_t)tiles;
  a.table = num_rows <= MAX_TABLE ? (uint32_t)num_rows + 1 : 0;
  a.pair_smooth = pseudocount / ((float)num_cats * (float)num_cats);
  a.z = (float)num_rows + pseudocount;
  const uint32_t pad = pcb_round_up(VC, TN);
  uint32_t* scratch = nullptr;   // counts, log marginals (both padded to whole tiles), status
  cudaMemPool_t pool = nullptr;
  PCB_CUDA(mi_pool(dev, &pool));
  PCB_CUDA(cudaMallocFromPoolAsync((void**)&scratch, ((size_t)2 * pad + 1) * sizeof(uint32_t), pool, st));
  float* logp = reinterpret_cast<float*>(scratch + pad);
  a.logp = logp;
  a.status = reinterpret_cast<int*>(scratch + (size_t)2 * pad);
  cudaMemsetAsync(scratch, 0, ((size_t)2 * pad + 1) * sizeof(uint32_t), st);
  if (num_cats > 32) cudaMemsetAsync(mi_dev, 0, (size_t)num_vars * num_vars * sizeof(float), st);
  mi_hist_kernel<<<dim3(num_vars, (uint32_t)std::min<uint64_t>(64, (num_rows + 4095) / 4096)), 256, 0, st>>>(data_dev, num_rows, num_vars,
                                                                                                           num_cats, scratch);
  mi_logp_kernel<<<(VC + 255) / 256, 256, 0, st>>>(scratch, VC, pseudocount / (float)num_cats, a.z, logp);
  static PcbPerDeviceOnce once;
  auto kernel = num_cats == 2 ? mi_tile_kernel<2, false> : num_cats == 4 ? mi_tile_kernel<4, false>
              : num_cats == 8 ? mi_tile_kernel<8, false> : num_cats == 16 ? mi_tile_kernel<16, false>
              : num_cats < SCATTER_CATS ? mi_tile_kernel<32, false> : mi_tile_kernel<32, true>;
  cudaError_t ce = once.run([] {
    const int most = (int)(SMEM_BASE + (MAX_TABLE + 1) * sizeof(float2));
    for (auto k : {mi_tile_kernel<2, false>, mi_tile_kernel<4, false>, mi_tile_kernel<8, false>, mi_tile_kernel<16, false>,
                   mi_tile_kernel<32, false>, mi_tile_kernel<32, true>}) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  });
  if (ce == cudaSuccess) {
    kernel<<<std::min(a.tiles, (uint32_t)sms), NTHREADS, SMEM_BASE + a.table * sizeof(float2), st>>>(a);
    ce = cudaGetLastError();
  }
  int h = 0;
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(&h, a.status, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(scratch, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  if (ce != cudaSuccess) return pcb_fail(PCB_ERR_CUDA, std::string("pairwise MI: ") + cudaGetErrorString(ce));
  if (h != 0) return pcb_fail(PCB_ERR_CUDA, "pairwise MI: a kernel gave up a bounded wait");
  return PCB_OK;
}
