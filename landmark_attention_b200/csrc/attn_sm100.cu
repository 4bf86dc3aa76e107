// Fused landmark attention for sm_100a: TMA-fed tcgen05 MMAs with TMEM accumulators.
//
// Shape contract: bf16 / fp16, head dim up to 128 (a multiple of 8), landmark block 64, any Lq, Lk - Lq a multiple of 64.
// Rows past the end of a sequence and features past the head dim are zeros that TMA fills in: no padded copies exist
// (the copies took 86 of 146 us at Lq = 1999, H = 32, D = 128 and 104 of 237 us at D = 64), and what is computed for them
// is dropped at the stores.  Head dims up to 64 have instances with half the products.
//
// Forward, one or two tiles of 128 query rows per CTA; rows 0-63 of a tile belong to landmark block `own0`, rows 64-127 to
// `own0 + 1`.
//   1. Pre-pass: S_lm = Q . K_lm^T against the landmark keys only (every 64th key, fetched with a strided 5-D TMA box)
//      gives each row the maximum landmark score of its earlier blocks.  Together with the row maximum of the
//      own (diagonal) block, which is processed first, this is the FINAL maximum of the outer softmax, so the O
//      accumulator in TMEM is never rescaled.
//   2. Main loop over key blocks n = own0+1 ... 0:  S = Q . K_n^T (N = 64);  the softmax threads read S from TMEM,
//      form the block's weights  p_j = softmax_inside_block(s)_j * exp(l_n - m)  (own block: exp(s_j - m), causal),
//      write them in 16 bits over the TMEM columns their S came from, and O += P . V_n takes P from there as the A operand
//      and V as an MN-major operand straight from its row-major TMA tile.
//   3. Epilogue: O / l -> global, plus the statistics L = l, M = m the backward pass needs.
// Reference semantics: llama/ltriton/flash_landmark_attention.py:6-122.
//
// Backward is recompute-based and atomic-free (bit-reproducible), in two launches:
//   a. dQ (sm100_bwd_dq_kernel): persistent; a unit is (128 query rows, batch*head).  Its prologue computes
//      delta = rowsum(O * dO) from the O and dO tiles (:125-149, without the 1/L pre-scaling) and stores it for (b).
//      Then, per key block: S = Q K^T, dP = dO V^T -> dS (written over the V tile, which dP no longer needs) ->
//      dQ += dS K with K as an MN-major operand.  Two softmax warpgroups take alternate blocks.
//   b. dK/dV (sm100_bwd_dkv_kernel): persistent; a unit is a pair of adjacent key blocks of one head, held in shared
//      memory while the query tiles that see them stream through.  Per tile: S, dP of both blocks into TMEM (N = 128);
//      the softmax threads rebuild P and dS (16 bits, [128 q x 64 k] swizzled tiles); dV += P^T dO and dK += dS^T Q with the
//      pair's 128 keys as M; P, dS, dO and Q are consumed as MN-major operands from their row-major tiles.
//   Per tile pair: earlier block  dS_j = g s_j (dP_j - nD) scale,  dS_landmark = g (nD - delta) scale,  P_j = g s_j,
//   with s = softmax inside the block, g = exp(l_n - M) / L, nD = sum_j s_j dP_j;  own block: p = exp(S - M) / L,
//   dS = p (dP - delta) scale.                                                                      (:152-305)
#include <atomic>
#include <mutex>
#include "common.cuh"
#include "attn_params.h"
#include "sm100_ptx.cuh"

namespace lmk {

__device__ int g_lmk_status = 0;   // first bounded wait that expired (0 = none); see lmk_device_status()


namespace {

using namespace ptx;

constexpr int kBlk = 64;
constexpr int kQTile = 128;
constexpr uint32_t kTileBytes = 16384;   // one [128 x 64] or two [64 x 64] 16-bit tiles
constexpr uint32_t kHalfTile = 8192;
constexpr float kLog2e = 1.4426950408889634f;

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  if (kBf16) {
    __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&t);
  } else {
    __half2 t = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&t);
  }
}

// write one row (64 16-bit values, given as 32 packed words) of a [128 x 64] K-major 128B-swizzled tile
__device__ __forceinline__ void store_row_sw128(uint32_t tile_base, int row, const uint32_t (&w)[32]) {
  const uint32_t row_addr = tile_base + row * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint32_t addr = row_addr + ((c ^ (row & 7)) << 4);
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[4 * c]), "r"(w[4 * c + 1]),
                 "r"(w[4 * c + 2]), "r"(w[4 * c + 3])
                 : "memory");
  }
}

// Row reductions with four independent chains: one softmax thread has little other work in flight, so a single
// 63-deep dependent chain of max / add would expose the ALU latency on every step.
// row_max: NaN where a value is NaN.
template <int N>
__device__ __forceinline__ float row_max(const float (&v)[64]) {
  float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j + 1 < N; j += 2) m[j / 2 % 4] = max3_nan(m[j / 2 % 4], v[j], v[j + 1]);
  return max3_nan(max3_nan(m[0], m[1], N % 2 ? v[N - 1] : -INFINITY), m[2], m[3]);
}
// Shift of the exponentials of an earlier block, -(row maximum) * c.  Some of them are polynomials, which make finite numbers of
// NaN and infinities (ex2_poly2): where the maximum is one of these the shift is NaN, and with it the exponentials between
// the polynomials, their sum, and everything that is divided by it.
__device__ __forceinline__ float block_shift(const float (&v)[64], float c) {
  const float mx = row_max<63>(v);
  return fmaf(mx, 0.f, -mx * c);
}
__device__ __forceinline__ float row_max_upto(const float (&v)[64], int last) {
  float a = -INFINITY, b = -INFINITY, c = -INFINITY, d = -INFINITY;
#pragma unroll
  for (int j = 0; j < 64; j += 4) {
    a = fmaxf(a, j <= last ? v[j] : -INFINITY);
    b = fmaxf(b, j + 1 <= last ? v[j + 1] : -INFINITY);
    c = fmaxf(c, j + 2 <= last ? v[j + 2] : -INFINITY);
    d = fmaxf(d, j + 3 <= last ? v[j + 3] : -INFINITY);
  }
  return fmaxf(fmaxf(a, b), fmaxf(c, d));
}
template <int N>
__device__ __forceinline__ float row_sum(const float (&v)[64]) {
  float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
#pragma unroll
  for (int j = 0; j + 3 < N; j += 4) {
    a += v[j];
    b += v[j + 1];
    c += v[j + 2];
    d += v[j + 3];
  }
#pragma unroll
  for (int j = N & ~3; j < N; ++j) a += v[j];
  return (a + b) + (c + d);
}

// ---------------------------------------------------------------------------------------------- other landmark patterns
// Instances with kIrr take landmark groups of any length up to 64 keys: a regular pattern with blocks below 64, or landmarks
// anywhere, given as one flag per (batch row, key).  The key tiles are then the GROUPS: tile n is the 64 keys that end with
// the group's landmark (TMA has no alignment rule for rows; rows in front of the sequence read as zeros), so the landmark
// is in column 63 as in the block-64 pattern and the first c0 columns, which belong to the group before, are hidden.  Each key
// belongs to one tile, softmax inside a group never leaves a tile, and the kernels stay single-pass: 51-key groups use 80 % of
// the columns and still take half the time of two passes over aligned tiles.  The keys behind the last landmark form the
// last tile, which ends at a position of its own.
// Rows whose groups do not fit (longer than 64 keys, or so short that tiles would be mostly empty) are left to the two-pass
// kernels of attn_mask_sm100.cu: the forward kernel marks them in R, the backward ones find them in the plan.
constexpr int kIrrMaxTiles = 65;                    // 64 landmarks and the open group
constexpr int kIrrMaxKeys = 64 * kIrrMaxTiles;
// The single pass works on 64 columns a group, however short the group is.  Measured (us, forward + backward, single-pass /
// two-pass kernels): B16 H8 T512, groups of 10 keys 525 / 625, 16 365 / 593, 51 183 / 361; B2 H8 T512, of 10 182 / 209,
// 51 98 / 122; B16 H8 T256, of 8 258 / 228, 10 219 / 225, 16 159 / 216.  The line (16 keys a group, counted 256 keys longer than
// the row is) falls at 8 keys for 256 and at 11 for 512: groups of 8 to 11 keys of longer rows would gain from a lower one.
constexpr int kIrrMinMeanGroup = 16;

struct IrrArgs {
  const uint8_t* flags = nullptr;      // [B, Lk] or null: the regular pattern with `block`
  int64_t stride = 0;
  int block = 0, G = 0;
  const int* plan = nullptr;           // backward, flags only: see irr_plan_kernel
  float* R = nullptr;                  // log2 of the row's normaliser instead of L and M (always with flags; forward otherwise)
};

// landmark positions and per-key landmark counts of one batch row, in shared memory
struct IrrSmem {
  uint64_t kmask[kIrrMaxTiles + 1];    // bit j of word w: key 64 w + j is a landmark
  int gbase[kIrrMaxTiles + 1];         // landmarks before word w
  int ends[kIrrMaxTiles + 1];          // position of column 63 of tile n
  int n_lm;
  int fallback;
};
__device__ __forceinline__ int irr_group(const IrrSmem& t, int pos) {          // landmarks strictly before pos
  return t.gbase[pos >> 6] + __popcll(t.kmask[pos >> 6] & ((1ull << (pos & 63)) - 1ull));
}
// All threads of the CTA; contains __syncthreads().
__device__ __forceinline__ void irr_build(IrrSmem& t, const uint8_t* flags, int Lk, int G) {
  const int words = (Lk + 63) / 64, warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int w = warp; w < words; w += warps) {
    const int k0 = w * 64 + lane;
    const unsigned lo = __ballot_sync(0xffffffffu, k0 < Lk && flags[k0] != 0);
    const unsigned hi = __ballot_sync(0xffffffffu, k0 + 32 < Lk && flags[k0 + 32] != 0);
    if (lane == 0) t.kmask[w] = (uint64_t)lo | ((uint64_t)hi << 32);
  }
  if (threadIdx.x == 0) t.fallback = 0;
  __syncthreads();
  if (warp == 0) {                     // exclusive prefix sums of the words' counts, three words a lane
    int c[3], sum = 0;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int w = lane * 3 + e;
      c[e] = w < words ? __popcll(t.kmask[w]) : 0;
      sum += c[e];
    }
    int inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    int run = inc - sum;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int w = lane * 3 + e;
      if (w < words) t.gbase[w] = run;
      run += c[e];
    }
    if (lane == 31) t.n_lm = run;
  }
  __syncthreads();
  const int n_lm = t.n_lm;
  const bool too_many = irr_group(t, Lk - 1) > min(G, kIrrMaxTiles - 1) || kIrrMinMeanGroup * (n_lm + 1) > Lk + 256;
  if (threadIdx.x < words && !too_many) {
    uint64_t m = t.kmask[threadIdx.x];
    int n = t.gbase[threadIdx.x];
    while (m) {
      const int j = __ffsll((long long)m) - 1;
      t.ends[n++] = threadIdx.x * 64 + j;
      m &= m - 1;
    }
  }
  if (threadIdx.x == 0) {
    if (!too_many) t.ends[n_lm] = Lk;
    else t.fallback = 1;
  }
  __syncthreads();
  if (!too_many && threadIdx.x <= n_lm && t.ends[threadIdx.x] - (threadIdx.x ? t.ends[threadIdx.x - 1] : -1) > 64)
    if (threadIdx.x < n_lm || n_lm == 0 || t.ends[n_lm - 1] + 1 < Lk) t.fallback = 1;       // (an empty open group is no group)
  __syncthreads();
}

// The same table in global memory for the backward kernels, one record per batch row: [0] landmarks, [1] fallback, [2 ...]
// ends, then one byte per key with its group.
constexpr int kIrrPlanHead = 2 + kIrrMaxTiles + 1;
constexpr int kIrrPlanInts = kIrrPlanHead + (kIrrMaxKeys + 3) / 4;
__device__ __forceinline__ bool irr_plan_fallback(const int* plan, int b) {
  return ld_behind_wait(plan + (int64_t)b * kIrrPlanInts + 1) != 0;
}
__device__ __forceinline__ int irr_plan_end(const int* plan, int b, int n) {
  return ld_behind_wait(plan + (int64_t)b * kIrrPlanInts + 2 + n);
}
__device__ __forceinline__ int irr_plan_group(const int* plan, int b, int pos) {
  return ld_behind_wait(reinterpret_cast<const uint8_t*>(plan + (int64_t)b * kIrrPlanInts + kIrrPlanHead) + pos);
}
__global__ void __launch_bounds__(256) irr_plan_kernel(const uint8_t* flags, int64_t stride, int Lk, int G, int* plan) {
  grid_dep_wait();
  grid_dep_launch();
  __shared__ IrrSmem t;
  const int b = blockIdx.x;
  irr_build(t, flags + (int64_t)b * stride, Lk, G);
  int* p = plan + (int64_t)b * kIrrPlanInts;
  if (threadIdx.x == 0) {
    p[0] = t.n_lm;
    p[1] = t.fallback;
  }
  if (t.fallback) return;
  for (int n = threadIdx.x; n <= t.n_lm; n += blockDim.x) p[2 + n] = t.ends[n];
  uint8_t* own = reinterpret_cast<uint8_t*>(p + kIrrPlanHead);
  for (int k = threadIdx.x; k < Lk; k += blockDim.x) own[k] = (uint8_t)irr_group(t, k);
}

// Hides the columns of the group before (c0 of them, the same for the whole warp), eight at a time up to the last one: eight
// tests of their own, one a chunk, took 400 - 600 clk an item whatever c0 was (clock stamps, groups of 51), nested ones end with
// the chunk that needs them.
template <int kChunk = 0, typename GetFn>
__device__ __forceinline__ void irr_hide(GetFn col, int c0) {
  if constexpr (kChunk < 8) {
    if (c0 > 8 * kChunk) {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (8 * kChunk + e < c0) col(8 * kChunk + e) = -INFINITY;
      irr_hide<kChunk + 1>(col, c0);
    }
  }
}

// ---------------------------------------------------------------------------------------------- forward, two tiles
// Up to TWO adjacent 128-row query tiles per CTA (one CTA per SM): softmax warpgroup 0 owns tile A
// (rows 256u .. 256u+127), warpgroup 1 owns tile B (the next 128 rows).  Both tiles consume the same K/V stream, so
// every K/V block is fetched from L2 once per 256 query rows, and the two softmax pipelines overlap with each
// other and with the MMAs.  Tile A skips the two newest key blocks (they lie after its own blocks).
// With one tile a CTA uses half of the registers, TMEM and shared memory, so that two CTAs share an SM and each other's start
// and end.
template <int kTiles> constexpr int kFwdStages = kTiles == 2 ? 5 : 2;
template <int kTiles> constexpr int kFwdThreads = (4 * kTiles + 3) * 32;
enum { kErrFwd2Producer = 111, kErrFwd2Mma = 112, kErrFwd2Softmax = 113, kErrFwd2Epilogue = 114 };

// one in this many pairs of exponentials uses ex2_poly2, of degree 4 (calls at B1 H32 L2048: 32 -> 42.2 us, 16 -> 41.3, 8 -> 39.9;
// a cubic 39.8.  Further from the truth by less than a cubic in one pair of 64: 2.7e-6 / 8 against 7.5e-5 / 64 on average)
constexpr int kFwdPolyEvery = 8;

template <int kStages> struct Fwd2Smem {
  uint64_t q_full;
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t s_full[2][2];    // [tile][S buffer]
  uint64_t s_free[2][2];
  uint64_t p_ready[2][2];   // [tile][buffer]: a warp whose rows have little to do can be one item ahead of the others
  uint64_t o_full;
  uint32_t tmem_base;
};

template <bool kBf16, int kD, bool kIrr, int kTiles>
__global__ void __launch_bounds__(kFwdThreads<kTiles>, 3 - kTiles)
sm100_fwd2_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_klm,
                  void* o_ptr, float* L_ptr, float* M_ptr, int H, int Lq, int Lk, int D, int lm_box, float scale_log2,
                  const void* k_ptr, int64_t ks_b, int64_t ks_h, int64_t ks_row, IrrArgs irr) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  auto q_tile = [&](int w) { return base + (uint32_t)w * 32768u; };
  constexpr int kStages = kFwdStages<kTiles>, kSw = 4 * kTiles;        // softmax warps; the three roles follow them
  auto k_slot = [&](int s) { return base + kTiles * 32768u + (uint32_t)s * 32768u; };
  auto v_slot = [&](int s) { return base + kTiles * 32768u + (uint32_t)s * 32768u + 16384u; };
  Fwd2Smem<kStages>* sm = reinterpret_cast<Fwd2Smem<kStages>*>(smem_raw + (base - raw) + (kTiles + kStages) * 32768u);

  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int t_a = ((int)gridDim.y - 1 - (int)blockIdx.y) * kTiles;      // heaviest tiles first, across all heads
  const bool has_b = kTiles == 2 && (t_a + 1) * kQTile < Lq;            // the second tile has at least one row
  const int bh = blockIdx.x, b = bh / H, h = bh - b * H;
  const int prefix_blocks = (Lk - Lq) / kBlk;
  const int pos_a = Lk - Lq + t_a * kQTile;             // key position of tile A's first row
  IrrSmem* tab = reinterpret_cast<IrrSmem*>(sm + 1);
  if constexpr (kIrr) {
    grid_dep_wait();                                    // flags may come from the kernel in front
    if (irr.flags != nullptr) {
      irr_build(*tab, irr.flags + (int64_t)b * irr.stride, Lk, irr.G);
      if (tab->fallback) {                              // uniform; the two-pass kernel takes the tiles marked here
        if (tid < 2 && (tid == 0 || has_b)) irr.R[(int64_t)bh * Lq + (t_a + tid) * kQTile] = -INFINITY;
        return;
      }
    }
  }
  auto group_of = [&](int pos) { return irr.flags != nullptr ? irr_group(*tab, pos) : pos / irr.block; };
  auto end_of = [&](int n) { return irr.flags != nullptr ? (n < 0 ? -1 : tab->ends[n]) : (n + 1) * irr.block - 1; };
  const int own0_a = prefix_blocks + 2 * t_a;           // tile A: blocks own0_a, own0_a+1; tile B: +2, +3
  // newest tile that any row of tile A / of the CTA sees
  const int last_a = kIrr ? warp_uniform(group_of(min(pos_a + kQTile, Lk) - 1)) : own0_a + 1;
  const int n_last = kIrr ? warp_uniform(group_of(min(pos_a + (has_b ? 2 : 1) * kQTile, Lk) - 1))
                          : min(own0_a + (has_b ? 3 : 1), (Lk - 1) / kBlk);
  const int n_lm_tiles = (n_last + 63) / 64;            // landmarks 0 .. n_last-1
  const int total = n_lm_tiles + n_last + 1;
  // tile A takes part in every item but the main items of tile B's own blocks
  auto active = [&](int w, int i) { return w == 1 ? has_b : (i < n_lm_tiles || n_last - (i - n_lm_tiles) <= last_a); };

  if (tid == 0) {
    mbar_init(smem_u32(&sm->q_full), 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&sm->full[s]), 1);
      mbar_init(smem_u32(&sm->empty[s]), 1);
    }
    for (int w = 0; w < 2; ++w) {
      for (int s = 0; s < 2; ++s) {
        mbar_init(smem_u32(&sm->s_full[w][s]), 1);
        mbar_init(smem_u32(&sm->s_free[w][s]), 1);
        mbar_init(smem_u32(&sm->p_ready[w][s]), 128);
      }
    }
    mbar_init(smem_u32(&sm->o_full), 1);
    mbar_init_fence();
  }
  if (warp == kSw + 1) tmem_alloc(smem_u32(&sm->tmem_base), kTiles * 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)warp_uniform((int)sm->tmem_base);
  auto tmem_s = [&](int w, int sb) { return tmem + (uint32_t)(w * 128 + sb * 64); };
  auto tmem_o = [&](int w) { return tmem + kTiles * 128u + (uint32_t)w * 128u; };
  if constexpr (!kIrr) grid_dep_wait();      // only the set-up may overlap the kernel in front (see the launch; kIrr: above)
  grid_dep_launch();      // a dependent kernel (the backward pass, the next call) may do its set-up while this grid drains

  if (warp == kSw) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      prefetch_tensormap(&tm_q);
      prefetch_tensormap(&tm_k);
      prefetch_tensormap(&tm_v);
      prefetch_tensormap(&tm_klm);
      const uint32_t qb = smem_u32(&sm->q_full);
      mbar_arrive_expect_tx(qb, (has_b ? 2 : 1) * (kD / 64) * kTileBytes);
      for (int w = 0; w < (has_b ? 2 : 1); ++w)
        for (int c = 0; c < kD / 64; ++c)
          tma_load_4d(q_tile(w) + c * kTileBytes, &tm_q, qb, 64 * c, (t_a + w) * kQTile, h, b);
      for (int i = 0; i < total; ++i) {
        const int s = i % kStages;
        mbar_wait(smem_u32(&sm->empty[s]), ((i / kStages) & 1) ^ 1, &g_lmk_status, kErrFwd2Producer);
        const uint32_t fb = smem_u32(&sm->full[s]);
        if (kIrr && i < n_lm_tiles) continue;           // the softmax warps gather the landmark keys themselves
        if (i < n_lm_tiles) {
          mbar_arrive_expect_tx(fb, (uint32_t)(lm_box * kD * 2));
          for (int c = 0; c < kD / 64; ++c)
            tma_load_5d(k_slot(s) + c * kHalfTile, &tm_klm, fb, 64 * c, kBlk - 1, i * 64, h, b);
        } else {
          const int n = n_last - (i - n_lm_tiles);
          const int r0 = kIrr ? end_of(n) - 63 : n * kBlk;
          mbar_arrive_expect_tx(fb, 2 * (kD / 64) * kHalfTile);
          for (int c = 0; c < kD / 64; ++c) {
            tma_load_4d(k_slot(s) + c * kHalfTile, &tm_k, fb, 64 * c, r0, h, b);
            tma_load_4d(v_slot(s) + c * kHalfTile, &tm_v, fb, 64 * c, r0, h, b);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == kSw + 1) {
    // ------------------------------------------------------------------ MMA issuer 1: S = Q K^T
    // A second issuing warp takes the P V products: the S products of the next key block never queue behind a wait for the
    // softmax of the current one.
    constexpr uint32_t fmt = kBf16 ? 1u : 0u;
    constexpr uint32_t idesc_s = instr_desc_f16(fmt, 128, 64, 0, 0);
    mbar_wait(smem_u32(&sm->q_full), 0, &g_lmk_status, kErrFwd2Mma);
    const uint64_t dq0 = smem_desc_sw128(q_tile(0), 16, 1024);
    const uint64_t dk0 = smem_desc_sw128(k_slot(0), 16, 1024);
    int ks[2] = {0, 0};
    int s = 0;
    uint32_t ph = 0;
    for (int j = 0; j < total; ++j) {
      mbar_wait(smem_u32(&sm->full[s]), ph, &g_lmk_status, kErrFwd2Mma);
      const uint64_t dk = desc_advance(dk0, (uint32_t)s * 32768u);
#pragma unroll
      for (int w = 0; w < kTiles; ++w) {
        if (!active(w, j)) continue;
        const int k = ks[w]++, sb = k & 1;
        if (k >= 2) mbar_wait(smem_u32(&sm->s_free[w][sb]), ((k >> 1) & 1) ^ 1, &g_lmk_status, kErrFwd2Mma);
        tc_fence_after();
        const uint64_t dq = desc_advance(dq0, (uint32_t)w * 32768u);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kD / 16; ++kk)
            mma_f16_ss(tmem_s(w, sb), desc_advance(dq, kmajor_step(kk, kTileBytes)),
                       desc_advance(dk, kmajor_step(kk, kHalfTile)), idesc_s, kk > 0);
          mma_commit(smem_u32(&sm->s_full[w][sb]));
        }
      }
      if (++s == kStages) { s = 0; ph ^= 1; }
    }
    __syncwarp();
  } else if (warp == kSw + 2) {
    // ------------------------------------------------------------------ MMA issuer 2: O += P V
    constexpr uint32_t fmt = kBf16 ? 1u : 0u;
    constexpr uint32_t idesc_o = instr_desc_f16(fmt, 128, kD, 0, 1);
    const uint64_t dv0 = smem_desc_sw128(v_slot(0), kHalfTile, 1024);
    int kp[2] = {0, 0};
    bool o_started[2] = {false, false};
    int s = 0;
    for (int i = 0; i < total; ++i) {
      const uint64_t dv = desc_advance(dv0, (uint32_t)s * 32768u);
#pragma unroll
      for (int w = 0; w < kTiles; ++w) {
        if (!active(w, i)) continue;
        const int k = kp[w]++;
        mbar_wait(smem_u32(&sm->p_ready[w][k & 1]), (k >> 1) & 1, &g_lmk_status, kErrFwd2Mma);
        tc_fence_after();
        if (i >= n_lm_tiles) {
          // A = P straight from TMEM: the softmax threads wrote it over the first 32 columns of the S buffer it was
          // computed from (8 columns = 16 keys per K-step)
          const uint32_t tp = tmem_s(w, k & 1);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kBlk / 16; ++kk)
              mma_f16_ts(tmem_o(w), tp + kk * 8, desc_advance(dv, kk * 2048), idesc_o,
                         (o_started[w] || kk > 0) ? 1u : 0u);
          }
          o_started[w] = true;
        }
        if (elect_one()) mma_commit(smem_u32(&sm->s_free[w][k & 1]));      // the S / P buffer may take the next S product
      }
      // the stage is free once both P V products are done; each of them waited for its S product to be read
      if (elect_one()) mma_commit(smem_u32(&sm->empty[s]));
      if (++s == kStages) s = 0;
    }
    if (elect_one()) mma_commit(smem_u32(&sm->o_full));
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    const int w = warp >> 2;                       // 0: tile A, 1: tile B
    const int row = tid & 127;
    const int half = row >> 6;
    const int pos = min(pos_a + w * kQTile + row, Lk - 1);
    const int own = kIrr ? group_of(pos) : own0_a + 2 * w + half;
    const int vis = min(kIrr ? 63 - (end_of(own) - pos) : row & 63, kBlk - 2);
    // kIrr: newest and oldest own tile of the warp's rows; ends of the next tile that this warp takes and of the one before it
    const int own_max = kIrr ? __reduce_max_sync(0xffffffffu, own) : own;
    const int own_min = kIrr ? __reduce_min_sync(0xffffffffu, own) : own;
    int e_hi = 0, e_lo = 0;
    if constexpr (kIrr) {
      const int first = kTiles == 2 && w == 0 ? last_a : n_last;
      e_hi = end_of(first);
      e_lo = end_of(first - 1);
    }
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    float m2 = -INFINITY, l = 0.f;
    int k = 0;
    if (kIrr && n_lm_tiles > 0) {                  // landmark keys of tiles 0 .. n_last-1 -> rows of the first stage
      const uint16_t* kb = reinterpret_cast<const uint16_t*>(k_ptr) + b * ks_b + h * ks_h;
      for (int e = tid; e < n_last * (kD / 8); e += kSw * 32) {
        const int n = e / (kD / 8), c = e - n * (kD / 8);
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (c * 8 < D) x = *reinterpret_cast<const uint4*>(kb + (int64_t)end_of(n) * ks_row + c * 8);
        const uint32_t addr = k_slot(0) + (uint32_t)(c >> 3) * kHalfTile + (uint32_t)n * 128u +
                              (uint32_t)(((c & 7) ^ (n & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w) : "memory");
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync 1, %0;" ::"n"(kSw * 32) : "memory");
      if (tid == 0) mbar_arrive(smem_u32(&sm->full[0]));
    }
    for (int i = 0; i < total; ++i) {
      if (!active(w, i)) continue;
      const int sb = k & 1;
      mbar_wait(smem_u32(&sm->s_full[w][sb]), (k / 2) & 1, &g_lmk_status, kErrFwd2Softmax);
      tc_fence_after();
      if (kIrr) __syncwarp();
      float sv[64];
      {
        uint32_t ra[32], rb[32];
        tmem_ld_32x32b_x32(tmem_s(w, sb) + lane_base, ra);
        tmem_ld_32x32b_x32(tmem_s(w, sb) + 32 + lane_base, rb);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          sv[j] = __uint_as_float(ra[j]);
          sv[32 + j] = __uint_as_float(rb[j]);
        }
      }
      uint32_t wgt[32];
      bool write_p = false;
      if (i < n_lm_tiles) {
        m2 = fmaxf(m2, row_max_upto(sv, own - 1 - i * 64) * scale_log2);
      } else {
        const int n = n_last - (i - n_lm_tiles);
        write_p = true;
        // With kIrr the rows of a warp can stand differently to tile n; every branch is taken by whole warps all the same
        // (votes), because the TMEM accesses behind it have to be executed by all lanes together.
        bool later = n > own, mixed = false;
        if constexpr (kIrr) {
          const int c0 = warp_uniform(64 - (e_hi - e_lo));
          e_hi = e_lo;
          if (n > 0) e_lo = end_of(n - 2);
          later = n > own_max;
          if (!later) irr_hide([&](int j) -> float& { return sv[j]; }, c0);
          mixed = !later && (c0 == 63 || n >= own_min);      // (c0 == 63: a landmark without keys)
        }
        if (later) {
#pragma unroll
          for (int j = 0; j < 32; ++j) wgt[j] = 0u;
        } else if (kIrr && mixed) {
          const bool earlier = n < own;
          const int last = earlier ? kBlk - 2 : (n == own ? vis : -1);
          const float lm = sv[63];
#pragma unroll
          for (int j = 0; j < 64; ++j) sv[j] = j <= last ? sv[j] : -INFINITY;
          const float mx = row_max<63>(sv) * scale_log2;
          if (n == own) m2 = fmaxf(m2, mx);
          const float el = earlier ? ex2(fmaf(lm, scale_log2, -m2)) : 0.f;
          float shift = earlier ? mx : m2;
          shift = shift == -INFINITY ? 0.f : shift;                               // nothing visible
#pragma unroll
          for (int j = 0; j < 64; ++j) sv[j] = ex2(fmaf(sv[j], scale_log2, -shift));      // (hidden ones: 0)
          const float sum = row_sum<64>(sv);
          const float wg = earlier ? (sum > 0.f ? __fdividef(el, sum) : 0.f) : 1.f;
          l += earlier ? el : sum;
#pragma unroll
          for (int j = 0; j < 32; ++j) wgt[j] = pack2<kBf16>(sv[2 * j] * wg, sv[2 * j + 1] * wg);
        } else if (!kIrr && n == own) {
          m2 = fmaxf(m2, row_max_upto(sv, vis) * scale_log2);
#pragma unroll
          for (int j = 0; j < 64; ++j) sv[j] = (j <= vis) ? ex2(fmaf(sv[j], scale_log2, -m2)) : 0.f;
          l += row_sum<64>(sv);
#pragma unroll
          for (int j = 0; j < 32; ++j) wgt[j] = pack2<kBf16>(sv[2 * j], sv[2 * j + 1]);
        } else {
          const float nmx = block_shift(sv, scale_log2);
          const float el = ex2(fmaf(sv[63], scale_log2, -m2));
          const uint64_t c2 = pk2(scale_log2, scale_log2), n2 = pk2(nmx, nmx);
          uint64_t sp[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const uint64_t x = fma2(pk2(sv[2 * j], sv[2 * j + 1]), c2, n2);
            if (j % kFwdPolyEvery == 1) {
              sp[j] = ex2_poly2<4>(x);       // a share of the exponentials runs on the FMA pipe
            } else {
              float a, b;
              upk2(x, a, b);
              sp[j] = pk2(ex2(a), j == 31 ? 0.f : ex2(b));
            }
          }
          uint64_t s0 = sp[0], s1 = sp[1], s2 = sp[2], s3 = sp[3];
#pragma unroll
          for (int j = 4; j < 32; j += 4) {
            s0 = add2(s0, sp[j]);
            s1 = add2(s1, sp[j + 1]);
            s2 = add2(s2, sp[j + 2]);
            s3 = add2(s3, sp[j + 3]);
          }
          float dl, dh;
          upk2(add2(add2(s0, s1), add2(s2, s3)), dl, dh);
          l += el;
          const float wg = __fdividef(el, dl + dh);
          const uint64_t w2 = pk2(wg, wg);
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float a, b;
            upk2(mul2(sp[j], w2), a, b);
            wgt[j] = pack2<kBf16>(a, b);
          }
        }
      }
      if (write_p) {
        tmem_st_32x32b_x32(tmem_s(w, sb) + lane_base, wgt);     // P replaces S in place; the P V product reads it there
        tmem_st_wait();
      }
      tc_fence_before();
      mbar_arrive(smem_u32(&sm->p_ready[w][sb]));
      ++k;
    }
    // ------------------------------------------------------------------ epilogue
    mbar_wait(smem_u32(&sm->o_full), 0, &g_lmk_status, kErrFwd2Epilogue);
    tc_fence_after();
    const float inv = kIrr && l == 0.f ? 0.f : 1.f / l;
    const int grow = (t_a + w) * kQTile + row;
    const bool stored = grow < Lq && (w == 0 || has_b);
    uint4* orow = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(o_ptr) + ((int64_t)bh * Lq + grow) * D);
    if (w == 0 || has_b) {
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_o(w) + c * 32 + lane_base, r);
        tmem_ld_wait();
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          uint4 pk;
          pk.x = pack2<kBf16>(__uint_as_float(r[8 * v4 + 0]) * inv, __uint_as_float(r[8 * v4 + 1]) * inv);
          pk.y = pack2<kBf16>(__uint_as_float(r[8 * v4 + 2]) * inv, __uint_as_float(r[8 * v4 + 3]) * inv);
          pk.z = pack2<kBf16>(__uint_as_float(r[8 * v4 + 4]) * inv, __uint_as_float(r[8 * v4 + 5]) * inv);
          pk.w = pack2<kBf16>(__uint_as_float(r[8 * v4 + 6]) * inv, __uint_as_float(r[8 * v4 + 7]) * inv);
          if (stored && c * 32 + v4 * 8 < D) orow[c * 4 + v4] = pk;
        }
      }
    }
    if (stored) {
      if (irr.R != nullptr) {
        irr.R[(int64_t)bh * Lq + grow] = l > 0.f ? m2 + __log2f(l) : INFINITY;
      } else {
        L_ptr[(int64_t)bh * Lq + grow] = l;
        M_ptr[(int64_t)bh * Lq + grow] = m2 * (1.f / kLog2e);
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == kSw + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTiles * 256);
  }
}

// ---------------------------------------------------------------------------------------------- backward
// One (query row, key block) pair of the backward pass, in packed fp32 pairs and within 168 registers per thread (so
// that two softmax warpgroups fit next to the issuing warps).
//   kind 0: block after the row's own block -> zeros;  kind 1: own block (causal, landmark hidden);
//   kind 2: earlier block (grouped).
// one in this many pairs of exponentials uses ex2_poly2, a cubic (forward + backward, us: B4 H16 L1024 D64 2 -> 91.4, 3 -> 90.4,
// 4 -> 90.3, 64 -> 91.3; B1 H32 L8192 D128 2 -> 2590, 3 -> 2577, 4 -> 2566)
constexpr int kBwdPolyEvery = 4;

template <bool kBf16>
__device__ __forceinline__ uint32_t pack2p(uint64_t v) {
  float lo, hi;
  upk2(v, lo, hi);
  return pack2<kBf16>(lo, hi);
}

// With kIrr the rows of a warp can be of different kinds (groups end anywhere).  The TMEM accesses have to be executed by all lanes
// of a warp together, so nothing branches on `kind` there: mixed warps take one masked pass with per-row limits and shifts.
// M2L = (row max + log(row sum)) * log2(e): exp2(s * c - M2L) is the outer-softmax probability.
//
// bwd_weights: reads S from TMEM once and leaves the row's weights in sp (packed pairs) up to the row factor w: P = w * sp.
struct RowFactors {
  float rden = 0.f;       // grouped rows: 1 / sum of the in-block exponentials
  float g = 0.f;          // grouped rows: the landmark's outer-softmax probability
  float w = 1.f;          // g * rden, or 1 where sp holds probabilities
};
template <bool kIrr, typename AfterFn>
__device__ __forceinline__ RowFactors bwd_weights(uint64_t (&sp)[32], int c0, uint32_t ts, int kind, int vis, float c, float M2L,
                                                  AfterFn after_s) {
  float nmx = 0.f, lm2 = 0.f;
  if (kIrr) __syncwarp();
  {
    uint32_t ra[32], rb[32];
    tmem_ld_32x32b_x32(ts, ra);
    tmem_ld_32x32b_x32(ts + 32, rb);
    tmem_ld_wait();
    if constexpr (kIrr)               // the first c0 columns belong to the group before
      irr_hide([&](int j) -> float& { return reinterpret_cast<float&>(j < 32 ? ra[j] : rb[j - 32]); }, c0);
    if (kIrr || kind == 2) {
      float sv[64];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        sv[j] = __uint_as_float(ra[j]);
        sv[32 + j] = __uint_as_float(rb[j]);
      }
      nmx = block_shift(sv, c);
      lm2 = sv[63] * c;
      if (kIrr && c0 == 63) nmx = 0.f;      // no key but the landmark
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      sp[j] = pk2u(ra[2 * j], ra[2 * j + 1]);
      sp[16 + j] = pk2u(rb[2 * j], rb[2 * j + 1]);
    }
  }
  after_s();      // S is in registers: its buffer may take the next product
  RowFactors f;
  const uint64_t c2 = pk2(c, c);
  uint64_t s0 = 0ull, s1 = 0ull, s2 = 0ull, s3 = 0ull;
  // all rows of the warp are of kind 2 and the group has keys (votes: the branches below are taken by whole warps)
  const bool fast = kIrr && c0 != 63 && __all_sync(0xffffffffu, kind == 2);
  if (kIrr && !fast) {
    const int last = kind == 2 ? kBlk - 2 : (kind == 1 ? vis : -1);
    const float shift = kind == 2 ? nmx : -M2L;
    const uint64_t m2 = pk2(shift, shift);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float a, b;
      upk2(fma2(sp[j], c2, m2), a, b);
      sp[j] = pk2(2 * j <= last ? ex2(a) : 0.f, 2 * j + 1 <= last ? ex2(b) : 0.f);
      if (j % 4 == 0) s0 = add2(s0, sp[j]);
      if (j % 4 == 1) s1 = add2(s1, sp[j]);
      if (j % 4 == 2) s2 = add2(s2, sp[j]);
      if (j % 4 == 3) s3 = add2(s3, sp[j]);
    }
  } else if (!kIrr && kind == 0) {
#pragma unroll
    for (int j = 0; j < 32; ++j) sp[j] = 0ull;
  } else if (!kIrr && kind == 1) {
    const uint64_t m2 = pk2(-M2L, -M2L);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float a, b;
      upk2(fma2(sp[j], c2, m2), a, b);
      sp[j] = pk2(2 * j <= vis ? ex2(a) : 0.f, 2 * j + 1 <= vis ? ex2(b) : 0.f);
    }
  } else {
    const uint64_t n2 = pk2(nmx, nmx);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const uint64_t x = fma2(sp[j], c2, n2);
      if (j % kBwdPolyEvery == 1) {
        sp[j] = ex2_poly2<3>(x);         // a share of the exponentials runs on the FMA pipe
      } else {
        float a, b;
        upk2(x, a, b);
        sp[j] = pk2(ex2(a), j == 31 ? 0.f : ex2(b));
      }
    }
    s0 = sp[0], s1 = sp[1], s2 = sp[2], s3 = sp[3];
#pragma unroll
    for (int j = 4; j < 32; j += 4) {
      s0 = add2(s0, sp[j]);
      s1 = add2(s1, sp[j + 1]);
      s2 = add2(s2, sp[j + 2]);
      s3 = add2(s3, sp[j + 3]);
    }
  }
  if (kIrr || kind == 2) {
    float dl, dh;
    upk2(add2(add2(s0, s1), add2(s2, s3)), dl, dh);
    const bool grouped = !kIrr || kind == 2;       // the rest is selects
    f.rden = kIrr && (c0 == 63 || !grouped) ? 0.f : __fdividef(1.f, dl + dh);
    f.g = ex2(lm2 - M2L);
    f.w = grouped ? f.g * f.rden : 1.f;
  }
  return f;
}

// bwd_dscores: reads dP from TMEM once, arrives on free_bar, and leaves the row of dS, packed to 16 bits, in wd.
template <bool kBf16, bool kIrr>
__device__ __forceinline__ void bwd_dscores(uint32_t (&wd)[32], const uint64_t (&sp)[32], const RowFactors& f, uint32_t tdp,
                                            uint32_t free_bar, int kind, float scale, float delta) {
  uint64_t dp[32];
  if (kIrr) __syncwarp();
  if (!kIrr && kind == 0) {
#pragma unroll
    for (int j = 0; j < 32; ++j) dp[j] = 0ull;
  } else {
    uint32_t ra[32], rb[32];
    tmem_ld_32x32b_x32(tdp, ra);
    tmem_ld_32x32b_x32(tdp + 32, rb);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      dp[j] = pk2u(ra[2 * j], ra[2 * j + 1]);
      dp[16 + j] = pk2u(rb[2 * j], rb[2 * j + 1]);
    }
  }
  tc_fence_before();
  mbar_arrive(free_bar);
  float sub = delta, lm_ds = 0.f;
  if (kIrr || kind == 2) {
    uint64_t n0 = 0ull, n1 = 0ull, n2a = 0ull, n3 = 0ull;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      n0 = fma2(sp[j], dp[j], n0);
      n1 = fma2(sp[j + 1], dp[j + 1], n1);
      n2a = fma2(sp[j + 2], dp[j + 2], n2a);
      n3 = fma2(sp[j + 3], dp[j + 3], n3);
    }
    float ql, qh;
    upk2(add2(add2(n0, n1), add2(n2a, n3)), ql, qh);
    const float nd = (ql + qh) * f.rden;
    sub = !kIrr || kind == 2 ? nd : delta;
    lm_ds = f.g * (nd - delta) * scale;
  }
  // dS = P * (dP - sub) * scale = sp * fma(dP, w * scale, -sub * w * scale)
  const float sc = scale * f.w;
  const uint64_t sc2 = pk2(sc, sc);
  const float nss = -sub * sc;
  const uint64_t nss2 = pk2(nss, nss);
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    float d0, d1;
    upk2(mul2(sp[j], fma2(dp[j], sc2, nss2)), d0, d1);
    if (j == 31 && kind == 2) d1 = lm_ds;
    wd[j] = pack2<kBf16>(d0, d1);
  }
}

enum { kErrDkvProducer = 201, kErrDkvMma = 202, kErrDkvSoftmax = 203, kErrDkvEpilogue = 204,
       kErrDqProducer = 301, kErrDqMma = 302, kErrDqSoftmax = 303, kErrDqEpilogue = 304 };

// ---------------------------------------------------------------------------------------------- backward: dK, dV
// Thread roles (both backward kernels): warps 0-3 and 4-7 are two softmax warpgroups, warp 8 issues TMA loads, warp 9 issues
// the S / dP MMAs and owns the TMEM allocation, warp 10 issues the accumulating MMAs.  Two issuing warps keep the
// products of the next item from queueing behind a wait for the current one.  (Registers are granted to 4 warps at
// a time, so 9 to 12 warps all leave 168 registers per thread.)
constexpr int kBwdGroups = 2;                       // softmax warpgroups
constexpr int kBwdThreads = (kBwdGroups * 4 + 3) * 32;
constexpr int kSdpBufs = 2;                         // S / dP buffers in TMEM of the dQ kernel: 2 x (64 + 64) columns
template <int kD> constexpr int kDkvStages = kD == 128 ? 2 : 4;

template <int kStages> struct DkvSmem {
  uint64_t k_full, k_empty, v_full, v_empty;
  uint64_t q_full[kStages], q_empty[kStages];       // Q: until dK has read it
  uint64_t do_full[kStages], do_empty[kStages];     // dO: until dP and dV have read it
  uint64_t s_full, s_free;                          // S of both blocks (one N = 128 product); both warpgroups hold it in registers
  uint64_t dp_full, dp_free;
  uint64_t p_ready, p_free;                         // the P rows are in the weight tiles / dV has read them
  uint64_t ds_ready, ds_free;                       // likewise the dS rows that replace them, and dK
  uint64_t acc_full[2], acc_empty[2];               // [0] dV, [1] dK
  uint32_t tmem_base;
};

// Stores 32 accumulator columns of one TMEM lane per thread as 16-bit values.  Four neighbouring lanes exchange 16-byte
// chunks first, so that a warp's store covers 64 contiguous bytes of eight rows and not 16 bytes of thirty-two.
// row_off[j]: element offset of row j of the lane's four rows, or -1 for a row that is not stored.  An output of the C interface
// may start at any word: one off a 16-byte boundary is stored word by word.
template <bool kBf16>
__device__ __forceinline__ void store_acc_cols(void* out, const int64_t (&row_off)[4], const uint32_t (&r)[32], int col0, int D,
                                               int lane) {
  uint4 v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    v[e].x = pack2<kBf16>(__uint_as_float(r[8 * e + 0]), __uint_as_float(r[8 * e + 1]));
    v[e].y = pack2<kBf16>(__uint_as_float(r[8 * e + 2]), __uint_as_float(r[8 * e + 3]));
    v[e].z = pack2<kBf16>(__uint_as_float(r[8 * e + 4]), __uint_as_float(r[8 * e + 5]));
    v[e].w = pack2<kBf16>(__uint_as_float(r[8 * e + 6]), __uint_as_float(r[8 * e + 7]));
  }
  // transpose of the 4 x 4 matrix (lane of the four, chunk): swap the off-diagonal chunks of 2 x 2 blocks, then the blocks
  auto swap = [&](uint4& a, uint4& b, int step) {      // lower lane: b <-> partner's a
    const bool up = (lane & step) != 0;
    uint4 x = up ? a : b;
    x.x = __shfl_xor_sync(0xffffffffu, x.x, step);
    x.y = __shfl_xor_sync(0xffffffffu, x.y, step);
    x.z = __shfl_xor_sync(0xffffffffu, x.z, step);
    x.w = __shfl_xor_sync(0xffffffffu, x.w, step);
    a = up ? x : a;
    b = up ? b : x;
  };
  swap(v[0], v[1], 1);
  swap(v[2], v[3], 1);
  swap(v[0], v[2], 2);
  swap(v[1], v[3], 2);
  const int col = col0 + 8 * (lane & 3);
  if (col >= D) return;
  const bool wide = ((uintptr_t)out & 15) == 0;       // rows and columns are multiples of 16 bytes
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (row_off[j] < 0) continue;
    uint32_t* to = reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(out) + row_off[j] + col);
    if (wide) {
      *reinterpret_cast<uint4*>(to) = v[j];
    } else {
      to[0] = v[j].x;
      to[1] = v[j].y;
      to[2] = v[j].z;
      to[3] = v[j].w;
    }
  }
}

// Persistent; a work unit is a PAIR of adjacent 64-key blocks (a = 2c, b = 2c+1) of one (batch, head).  Both blocks
// stay in shared memory while the unit streams the query tiles that see them, so each Q/dO tile is fetched from
// L2 once per 128 keys.  All four products of an item are single ones over both blocks: S = Q K^T and dP = dO V^T with N = 128,
// dV += P^T dO and dK += dS^T Q with M = 128 keys and N = kD.  Warpgroup 0 rebuilds P and dS for block a, warpgroup 1 for block b.
// P is handed over as soon as S allows it, before dP is looked at; dS takes its place once dV has read it, and the next P takes
// dS's place once dK has read that: each of these waits has half an item of other work in front of it.
// Q and dO have barriers of their own, so dO's place is reloaded from the end of dV on and Q's from the end of dK on.
// The former arrangement (one P and one dS tile that the warpgroups took in turns, dV and dK as four products of N = 64, 448 KB of
// shared-memory traffic an item instead of 384, Q and dO handed over together, 128 features multiplied whatever kD is) against
// this one, forward + backward: B4 H16 L1024 D64 102.6 / 95.4 us, B1 H32 L2048 D128 201.7 / 197.7.
// CTA c takes units w = round * grid + c with the direction alternating per round (snake), heaviest pairs first.
// Loads, S/dP products and the softmax of the next unit start while the accumulators of the current one are drained.
template <bool kBf16, int kD, bool kWhole, bool kIrr>      // kWhole: whole tiles and D = kD
__global__ void __launch_bounds__(kBwdThreads, 1)
sm100_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                     const float* L_ptr, const float* M_ptr, const float* delta_ptr, void* dk_ptr, void* dv_ptr, int H, int BH,
                     int Lq, int Lk, int D_any, float scale, float scale_log2, int max_tiles, IrrArgs irr) {
  const int D = kWhole ? kD : D_any;
  constexpr int kStages = kDkvStages<kD>;
  constexpr uint32_t kOperand = (kD / 64) * kTileBytes;     // [128 rows x kD] as 64-feature sub-tiles of 16 KB
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  // K of the pair as one [128 keys x kD] K-major operand, block g's 64 rows at g * 8 KB inside each sub-tile; V likewise
  const uint32_t k_pair = base, v_pair = base + kOperand;
  auto q_slot = [&](int s) { return base + 2 * kOperand + (uint32_t)s * 2 * kOperand; };
  auto do_slot = [&](int s) { return base + 3 * kOperand + (uint32_t)s * 2 * kOperand; };
  const uint32_t w_tile = base + (2 + 2 * kStages) * kOperand;         // P, then dS: [128 q x 64 keys] of block a, then of b
  DkvSmem<kStages>* sm =
      reinterpret_cast<DkvSmem<kStages>*>(smem_raw + (base - raw) + (2 + 2 * kStages) * kOperand + 2 * kTileBytes);

  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int prefix_blocks = (Lk - Lq) / kBlk;
  const int n_tiles = (Lq + kQTile - 1) / kQTile;
  const int n_blocks = (Lk + kBlk - 1) / kBlk;
  const int n_pairs = ((kIrr ? max_tiles : n_blocks) + 1) / 2;
  const int n_units = n_pairs * BH;
  auto unit_of = [&](int r) {
    const int c = (r & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
    return r * (int)gridDim.x + c;
  };
  // kIrr: tile table of the unit's batch row (flags), or the regular pattern
  auto group_of = [&](int b, int pos) { return irr.flags != nullptr ? irr_plan_group(irr.plan, b, pos) : pos / irr.block; };
  auto end_of = [&](int b, int n) {
    return n < 0 ? -1 : (irr.flags != nullptr ? irr_plan_end(irr.plan, b, n) : (n + 1) * irr.block - 1);
  };
  auto tiles_of = [&](int b) { return kIrr ? group_of(b, Lk - 1) + 1 : n_blocks; };
  auto skipped = [&](int w) {
    if constexpr (!kIrr) return false;
    const int b = (w % BH) / H;
    return (irr.flags != nullptr && irr_plan_fallback(irr.plan, b)) || 2 * (w / BH) >= tiles_of(b);
  };
  auto unit_tq0 = [&](int w) {                       // first query tile that sees the pair
    const int pair = w / BH;
    if constexpr (kIrr) return max(end_of((w % BH) / H, 2 * pair - 1) + 1 - (Lk - Lq), 0) / kQTile;
    return 2 * pair > prefix_blocks ? (2 * pair - prefix_blocks) / 2 : 0;
  };

  if (tid == 0) {
    mbar_init(smem_u32(&sm->k_full), 1);
    mbar_init(smem_u32(&sm->k_empty), 1);
    mbar_init(smem_u32(&sm->v_full), 1);
    mbar_init(smem_u32(&sm->v_empty), 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&sm->q_full[s]), 1);
      mbar_init(smem_u32(&sm->q_empty[s]), 1);
      mbar_init(smem_u32(&sm->do_full[s]), 1);
      mbar_init(smem_u32(&sm->do_empty[s]), 2);       // dP and dV, issued by different warps
    }
    mbar_init(smem_u32(&sm->s_full), 1);
    mbar_init(smem_u32(&sm->s_free), 256);
    mbar_init(smem_u32(&sm->dp_full), 1);
    mbar_init(smem_u32(&sm->dp_free), 256);
    mbar_init(smem_u32(&sm->p_ready), 256);
    mbar_init(smem_u32(&sm->p_free), 1);
    mbar_init(smem_u32(&sm->ds_ready), 256);
    mbar_init(smem_u32(&sm->ds_free), 1);
    for (int g = 0; g < 2; ++g) {
      mbar_init(smem_u32(&sm->acc_full[g]), 1);
      mbar_init(smem_u32(&sm->acc_empty[g]), 128);
    }
    mbar_init_fence();
  }
  if (warp == kBwdGroups * 4 + 1) tmem_alloc(smem_u32(&sm->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)warp_uniform((int)sm->tmem_base);
  const uint32_t tmem_s = tmem, tmem_dp = tmem + 128u, tmem_dv = tmem + 256u, tmem_dk = tmem + 256u + kD;

  if (warp == kBwdGroups * 4) {
    if (lane == 0) {
      prefetch_tensormap(&tm_q);
      prefetch_tensormap(&tm_k);
      prefetch_tensormap(&tm_v);
      prefetch_tensormap(&tm_do);
      int it = 0, u = 0;
      for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
        if (skipped(w)) continue;
        const int pair = w / BH, bh = w - pair * BH, b = bh / H, h = bh - b * H;
        const int tq0 = unit_tq0(w), n_items = n_tiles - tq0;
        int key_row[2];
        for (int g = 0; g < 2; ++g) {       // a block past the end of the sequence reads as zeros
          const int n = 2 * pair + g;
          key_row[g] = kIrr ? (n < tiles_of(b) ? end_of(b, n) - 63 : Lk) : n * kBlk;
        }
        auto load_pair = [&](uint32_t dst, const CUtensorMap* tm, uint64_t* full, uint64_t* empty) {
          const uint32_t fb = smem_u32(full);
          mbar_wait(smem_u32(empty), (u & 1) ^ 1, &g_lmk_status, kErrDkvProducer);
          mbar_arrive_expect_tx(fb, kOperand);
          for (int g = 0; g < 2; ++g)
            for (int c = 0; c < kD / 64; ++c)
              tma_load_4d(dst + c * kTileBytes + g * kHalfTile, tm, fb, 64 * c, key_row[g], h, b);
        };
        auto load_rows = [&](uint32_t dst, const CUtensorMap* tm, uint64_t* full, uint64_t* empty, int tile) {
          const uint32_t fb = smem_u32(full);
          mbar_wait(smem_u32(empty), ((it / kStages) & 1) ^ 1, &g_lmk_status, kErrDkvProducer);
          mbar_arrive_expect_tx(fb, kOperand);
          for (int c = 0; c < kD / 64; ++c) tma_load_4d(dst + c * kTileBytes, tm, fb, 64 * c, tile * kQTile, h, b);
        };
        load_pair(k_pair, &tm_k, &sm->k_full, &sm->k_empty);
        for (int i = 0; i < n_items; ++i, ++it) {
          const int s = it % kStages;
          load_rows(q_slot(s), &tm_q, &sm->q_full[s], &sm->q_empty[s], tq0 + i);
          if (i == 0) load_pair(v_pair, &tm_v, &sm->v_full, &sm->v_empty);
          load_rows(do_slot(s), &tm_do, &sm->do_full[s], &sm->do_empty[s], tq0 + i);
        }
        ++u;
      }
    }
    __syncwarp();
  } else if (warp == kBwdGroups * 4 + 1) {
    // S = Q K^T and dP = dO V^T of both blocks of the pair at once, one query tile at a time.  The warpgroups hold S in
    // registers early in an item, so the next S product runs while they are still busy with dP.
    constexpr uint32_t fmt = kBf16 ? 1u : 0u;
    constexpr uint32_t idesc_s = instr_desc_f16(fmt, 128, 128, 0, 0);
    const uint64_t dk0 = smem_desc_sw128(k_pair, 16, 1024), dv0 = smem_desc_sw128(v_pair, 16, 1024);
    const uint64_t dq0 = smem_desc_sw128(q_slot(0), 16, 1024), ddo0 = smem_desc_sw128(do_slot(0), 16, 1024);
    int it = 0, u = 0;
    for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
      if (warp_uniform(skipped(w))) continue;
      const int n_items = n_tiles - warp_uniform(unit_tq0(w));
      mbar_wait(smem_u32(&sm->k_full), u & 1, &g_lmk_status, kErrDkvMma);
      for (int i = 0; i < n_items; ++i, ++it) {
        const int s = it % kStages;
        const uint64_t dq = desc_advance(dq0, (uint32_t)s * 2 * kOperand), ddo = desc_advance(ddo0, (uint32_t)s * 2 * kOperand);
        mbar_wait(smem_u32(&sm->q_full[s]), (it / kStages) & 1, &g_lmk_status, kErrDkvMma);
        if (it >= 1) mbar_wait(smem_u32(&sm->s_free), (it & 1) ^ 1, &g_lmk_status, kErrDkvMma);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kD / 16; ++kk)
            mma_f16_ss(tmem_s, desc_advance(dq, kmajor_step(kk, kTileBytes)), desc_advance(dk0, kmajor_step(kk, kTileBytes)),
                       idesc_s, kk > 0);
          mma_commit(smem_u32(&sm->s_full));
          if (i == n_items - 1) mma_commit(smem_u32(&sm->k_empty));
        }
        if (i == 0) mbar_wait(smem_u32(&sm->v_full), u & 1, &g_lmk_status, kErrDkvMma);
        mbar_wait(smem_u32(&sm->do_full[s]), (it / kStages) & 1, &g_lmk_status, kErrDkvMma);
        if (it >= 1) mbar_wait(smem_u32(&sm->dp_free), (it & 1) ^ 1, &g_lmk_status, kErrDkvMma);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kD / 16; ++kk)
            mma_f16_ss(tmem_dp, desc_advance(ddo, kmajor_step(kk, kTileBytes)), desc_advance(dv0, kmajor_step(kk, kTileBytes)),
                       idesc_s, kk > 0);
          mma_commit(smem_u32(&sm->dp_full));
          mma_commit(smem_u32(&sm->do_empty[s]));
          if (i == n_items - 1) mma_commit(smem_u32(&sm->v_empty));
        }
      }
      ++u;
    }
  } else if (warp == kBwdGroups * 4 + 2) {
    // dV += P^T dO and dK += dS^T Q.  A = P^T / dS^T: MN-major view of the two [128 q x 64 keys] tiles; B = dO / Q: MN-major view
    // of the row-major [128 q x kD] tile; a K-step is 16 query rows = 2048 bytes.  dV waits for dO itself: P may be there first.
    constexpr uint32_t fmt = kBf16 ? 1u : 0u;
    constexpr uint32_t idesc_t = instr_desc_f16(fmt, 128, kD, 1, 1);
    const uint64_t dq0t = smem_desc_sw128(q_slot(0), kTileBytes, 1024);
    const uint64_t ddo0t = smem_desc_sw128(do_slot(0), kTileBytes, 1024);
    const uint64_t dwt = smem_desc_sw128(w_tile, kTileBytes, 1024);
    int it = 0, u = 0;
    for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
      if (warp_uniform(skipped(w))) continue;
      const int n_items = n_tiles - warp_uniform(unit_tq0(w));
      for (int i = 0; i < n_items; ++i, ++it) {
        const int s = it % kStages;
        const uint64_t ddot = desc_advance(ddo0t, (uint32_t)s * 2 * kOperand), dqt = desc_advance(dq0t, (uint32_t)s * 2 * kOperand);
        mbar_wait(smem_u32(&sm->do_full[s]), (it / kStages) & 1, &g_lmk_status, kErrDkvMma);
        if (i == 0) mbar_wait(smem_u32(&sm->acc_empty[0]), (u & 1) ^ 1, &g_lmk_status, kErrDkvMma);
        mbar_wait(smem_u32(&sm->p_ready), it & 1, &g_lmk_status, kErrDkvMma);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kQTile / 16; ++kk)
            mma_f16_ss(tmem_dv, desc_advance(dwt, kk * 2048), desc_advance(ddot, kk * 2048), idesc_t, (i > 0 || kk > 0) ? 1u : 0u);
          mma_commit(smem_u32(&sm->p_free));
          mma_commit(smem_u32(&sm->do_empty[s]));
          if (i == n_items - 1) mma_commit(smem_u32(&sm->acc_full[0]));
        }
        if (i == 0) mbar_wait(smem_u32(&sm->acc_empty[1]), (u & 1) ^ 1, &g_lmk_status, kErrDkvMma);
        mbar_wait(smem_u32(&sm->ds_ready), it & 1, &g_lmk_status, kErrDkvMma);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kQTile / 16; ++kk)
            mma_f16_ss(tmem_dk, desc_advance(dwt, kk * 2048), desc_advance(dqt, kk * 2048), idesc_t, (i > 0 || kk > 0) ? 1u : 0u);
          mma_commit(smem_u32(&sm->ds_free));
          mma_commit(smem_u32(&sm->q_empty[s]));
          if (i == n_items - 1) mma_commit(smem_u32(&sm->acc_full[1]));
        }
      }
      ++u;
    }
  } else {
    const int g = warp >> 2;                       // warpgroup g owns block g of every pair, and drains dV (0) or dK (1) of both
    const int row = tid & 127;
    const int half = row >> 6;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t my_tile = w_tile + (uint32_t)g * kTileBytes;
    int it = 0, u = 0;
    auto stat_m = [&](int64_t i) { return ld_behind_wait((kIrr && irr.R != nullptr ? irr.R : M_ptr) + i); };
    auto stat_l = [&](int64_t i) { return kIrr && irr.R != nullptr ? 1.f : ld_behind_wait(L_ptr + i); };
    // What a unit needs from global memory, asked for while the unit before it drains: the tile table first (all entries at
    // once), then the row statistics of the first item.  Read one after the other at the start of a unit they took
    // 1500 - 2000 clk of it.
    // (rows past the end of the sequence have zero Q and dO tiles: whatever finite weights they get contribute nothing)
    int bh = -1, b = 0, pair = 0, tq0 = 0, tiles = n_blocks, e_m = 0, e_0 = 0, e_1 = 0;      // bh < 0: no unit left
    float nM = 0.f, nL = 1.f, nDelta = 0.f;
    int nOwn = 0;
    auto own_of = [&](int r) { return kIrr ? group_of(b, min(Lk - Lq + r, Lk - 1)) : 0; };
    auto fetch_rows = [&](int tq) {
      const int64_t grow = (int64_t)bh * Lq + (kWhole ? tq * kQTile + row : min(tq * kQTile + row, Lq - 1));
      nM = stat_m(grow);
      nL = stat_l(grow);
      nDelta = ld_behind_wait(delta_ptr + grow);
      nOwn = own_of(tq * kQTile + row);
    };
    int r = 0;
    auto fetch_unit = [&]() {                       // kIrr
      for (;; ++r) {
        const int w = unit_of(r);
        if (w >= n_units) {
          bh = -1;
          return;
        }
        pair = w / BH;
        bh = w - pair * BH;
        b = bh / H;
        const bool fallback = irr.flags != nullptr && irr_plan_fallback(irr.plan, b);
        tiles = tiles_of(b);
        e_m = end_of(b, 2 * pair - 1);              // (entries behind the last tile: inside the table, not used)
        e_0 = end_of(b, 2 * pair);
        e_1 = end_of(b, 2 * pair + 1);
        if (fallback || 2 * pair >= tiles) continue;
        tq0 = max(e_m + 1 - (Lk - Lq), 0) / kQTile;
        fetch_rows(tq0);
        ++r;
        return;
      }
    };
    auto run_unit = [&]() {
      const int n = 2 * pair + g, n_items = n_tiles - tq0;
      const int end = g == 0 ? e_0 : e_1;
      const int c0 = kIrr && n < tiles ? warp_uniform(64 - (end - (g == 0 ? e_m : e_0))) : 0;
      for (int i = 0; i < n_items; ++i, ++it) {
        const int tq = tq0 + i;
        const int own = kIrr ? nOwn : prefix_blocks + 2 * tq + half;
        const int vis = min(kIrr ? 63 - (end - (Lk - Lq + tq * kQTile + row)) : row & 63, kBlk - 2);      // used where n == own
        const bool row_valid = kWhole || tq * kQTile + row < Lq;
        const float M2L = !row_valid ? 0.f : (kIrr && irr.R != nullptr ? nM : fmaf(nM, kLog2e, __log2f(nL)));
        const float delta = row_valid ? nDelta : 0.f;
        if (i + 1 < n_items) fetch_rows(tq + 1);      // one item ahead, so that their latency is never exposed
        const int kind = n > own ? 0 : (n == own ? 1 : 2);
        mbar_wait(smem_u32(&sm->s_full), it & 1, &g_lmk_status, kErrDkvSoftmax);
        tc_fence_after();
        uint64_t sp[32];
        const RowFactors f = bwd_weights<kIrr>(sp, c0, tmem_s + (uint32_t)g * 64u + lane_base, kind, vis, scale_log2, M2L, [&]() {
          tc_fence_before();
          mbar_arrive(smem_u32(&sm->s_free));
        });
        uint32_t wd[32];
        {
          const uint64_t w2 = pk2(f.w, f.w);
#pragma unroll
          for (int j = 0; j < 32; ++j) wd[j] = pack2p<kBf16>(mul2(sp[j], w2));
        }
        if (it >= 1) mbar_wait(smem_u32(&sm->ds_free), (it & 1) ^ 1, &g_lmk_status, kErrDkvSoftmax);
        store_row_sw128(my_tile, row, wd);
        fence_proxy_async_smem();
        mbar_arrive(smem_u32(&sm->p_ready));
        mbar_wait(smem_u32(&sm->dp_full), it & 1, &g_lmk_status, kErrDkvSoftmax);
        tc_fence_after();
        bwd_dscores<kBf16, kIrr>(wd, sp, f, tmem_dp + (uint32_t)g * 64u + lane_base, smem_u32(&sm->dp_free), kind, scale, delta);
        mbar_wait(smem_u32(&sm->p_free), it & 1, &g_lmk_status, kErrDkvSoftmax);
        store_row_sw128(my_tile, row, wd);
        fence_proxy_async_smem();
        mbar_arrive(smem_u32(&sm->ds_ready));
      }
      // epilogue: TMEM lane = key of the pair
      int64_t off = -1;
      {
        const int n_r = 2 * pair + half;
        int key = n_r * kBlk + (row & 63);
        bool stored = key < Lk;
        if (kIrr) {
          key = (half == 0 ? e_0 : e_1) - 63 + (row & 63);
          stored = n_r < tiles && key > (half == 0 ? e_m : e_0) && key < Lk;       // the tile's own keys
        }
        if (stored) off = ((int64_t)bh * Lk + key) * D;
      }
      int64_t row_off[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) row_off[j] = __shfl_sync(0xffffffffu, off, (lane & ~3) + j);
      if constexpr (kIrr) fetch_unit();
      mbar_wait(smem_u32(&sm->acc_full[g]), u & 1, &g_lmk_status, kErrDkvEpilogue);
      tc_fence_after();
      if (kIrr) __syncwarp();
      const uint32_t t_acc = (g == 0 ? tmem_dv : tmem_dk) + lane_base;
      void* const out = g == 0 ? dv_ptr : dk_ptr;
#pragma unroll
      for (int c = 0; c < kD / 64; ++c) {
        uint32_t ra[32], rb[32];
        tmem_ld_32x32b_x32(t_acc + c * 64, ra);
        tmem_ld_32x32b_x32(t_acc + c * 64 + 32, rb);
        tmem_ld_wait();
        if (c == kD / 64 - 1) {
          tc_fence_before();
          mbar_arrive(smem_u32(&sm->acc_empty[g]));     // the next unit may start accumulating
        }
        store_acc_cols<kBf16>(out, row_off, ra, c * 64, D, lane);
        store_acc_cols<kBf16>(out, row_off, rb, c * 64 + 32, D, lane);
      }
      ++u;
    };
    if constexpr (kIrr) {
      grid_dep_wait();     // delta comes from the dQ kernel, which may still be running (see the launch)
      fetch_unit();
      while (bh >= 0) run_unit();
    } else {      // nothing but the statistics to ask for: holding them over the epilogue's stores costs more than it hides
      for (int k = 0, w = unit_of(0); w < n_units; w = unit_of(++k)) {
        pair = w / BH;
        bh = w - pair * BH;
        tq0 = unit_tq0(w);
        if (u == 0) grid_dep_wait();
        fetch_rows(tq0);
        run_unit();
      }
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == kBwdGroups * 4 + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------- backward: dQ
constexpr int kDqStages = 4;
// The dQ kernel has a fourth role: S = Q K^T and dP = dO V^T are issued by two different warps, so that neither waits behind the
// other one's buffer.
constexpr int kDqThreads = kBwdThreads + 32;

struct DqSmem {
  uint64_t qdo_full;
  uint64_t ops_ready;       // the unit's Q and dO rows sit in TMEM (written by the softmax warpgroups)
  uint64_t ops_free;        // the S / dP products of the unit have read them
  uint64_t delta_read;      // both softmax warpgroups are done with the Q, dO and O tiles in shared memory
  uint64_t full[kDqStages];
  uint64_t empty[kDqStages];
  uint64_t ds_ready[kDqStages];
  uint64_t s_full[kSdpBufs];       // S and dP are handed over separately: the next S product of a buffer runs while its
  uint64_t s_free[kSdpBufs];       // warpgroup is still busy with dP
  uint64_t dp_full[kSdpBufs];
  uint64_t dp_free[kSdpBufs];
  uint64_t acc_full[2];     // per draining warpgroup (the one that took the unit's last item)
  uint64_t acc_empty;
  uint32_t tmem_base;
};

// Persistent: one CTA per SM walks through the units (128 query rows, batch*head), heaviest tiles first, dealt to the
// CTAs in a snake.  The K/V stream, the S/dP products and the softmax of the next unit start while dQ of the current
// unit is drained by one warpgroup (the two warpgroups alternate); only the unit's first accumulating MMA waits for
// the drain.  All barrier phases derive from counters that run across units.
template <bool kBf16, int kD, bool kWhole, bool kIrr>
__global__ void __launch_bounds__(kDqThreads, 1)
sm100_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                    const __grid_constant__ CUtensorMap tm_o, const float* L_ptr, const float* M_ptr, float* delta_ptr,
                    void* dq_ptr, int H, int BH, int Lq, int Lk, int D_any, float scale, float scale_log2, IrrArgs irr) {
  const int D = kWhole ? kD : D_any;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t q_tile = base, do_tile = base + 32768u;
  auto k_slot = [&](int s) { return base + 65536u + (uint32_t)s * 32768u; };
  auto v_slot = [&](int s) { return base + 65536u + (uint32_t)s * 32768u + 16384u; };   // V block, later dS
  const uint32_t o_tile = base + 65536u + kDqStages * 32768u;      // forward output tile, only for delta
  DqSmem* sm = reinterpret_cast<DqSmem*>(smem_raw + (base - raw) + 65536u + kDqStages * 32768u + 32768u);

  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5), lane = tid & 31;
  const int n_tiles = (Lq + kQTile - 1) / kQTile;
  const int n_blocks = (Lk + kBlk - 1) / kBlk;
  const int prefix_blocks = (Lk - Lq) / kBlk;
  const int n_units = n_tiles * BH;
  auto unit_of = [&](int r) {
    const int c = (r & 1) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
    return r * (int)gridDim.x + c;
  };
  // unit w -> query tile (heaviest = last tile first) and number of key blocks it sees
  auto unit_tile = [&](int w) { return n_tiles - 1 - w / BH; };
  // kIrr: tile table and group of every key of the unit's batch row (flags), or the regular pattern
  auto skipped = [&](int w) { return kIrr && irr.flags != nullptr && irr_plan_fallback(irr.plan, (w % BH) / H); };
  auto group_of = [&](int b, int pos) { return irr.flags != nullptr ? irr_plan_group(irr.plan, b, pos) : pos / irr.block; };
  auto end_of = [&](int b, int n) { return irr.flags != nullptr ? irr_plan_end(irr.plan, b, n) : (n + 1) * irr.block - 1; };
  auto regular_items = [&](int t) { return kWhole ? prefix_blocks + 2 * t + 2 : min(prefix_blocks + 2 * t + 2, n_blocks); };

  auto unit_items = [&](int w) {
    const int t = unit_tile(w);
    if constexpr (kIrr) return group_of((w % BH) / H, min(Lk - Lq + (t + 1) * kQTile, Lk) - 1) + 1;
    return regular_items(t);
  };

  if (tid == 0) {
    mbar_init(smem_u32(&sm->qdo_full), 1);
    mbar_init(smem_u32(&sm->ops_ready), 256);
    mbar_init(smem_u32(&sm->ops_free), 2);          // the S issuer and the dP issuer
    mbar_init(smem_u32(&sm->delta_read), 256);
    for (int s = 0; s < kDqStages; ++s) {
      mbar_init(smem_u32(&sm->full[s]), 1);
      mbar_init(smem_u32(&sm->empty[s]), 1);
      mbar_init(smem_u32(&sm->ds_ready[s]), 128);
    }
    for (int s = 0; s < kSdpBufs; ++s) {
      mbar_init(smem_u32(&sm->s_full[s]), 1);
      mbar_init(smem_u32(&sm->s_free[s]), 128);
      mbar_init(smem_u32(&sm->dp_full[s]), 1);
      mbar_init(smem_u32(&sm->dp_free[s]), 128);
    }
    mbar_init(smem_u32(&sm->acc_full[0]), 1);
    mbar_init(smem_u32(&sm->acc_full[1]), 1);
    mbar_init(smem_u32(&sm->acc_empty), 128);
    mbar_init_fence();
  }
  if (warp == kBwdGroups * 4 + 1) tmem_alloc(smem_u32(&sm->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = (uint32_t)warp_uniform((int)sm->tmem_base);
  // TMEM: S buffers [0,128), dP buffers [128,256), dQ [256,384), Q rows [384,448), dO rows [448,512).  Q and dO are the
  // A operands of S = Q K^T and dP = dO V^T for every key block of the unit: held in TMEM they are not re-read from
  // shared memory 2 x 32 KB per block (half of the kernel's shared-memory operand traffic), and their shared-memory
  // tiles are free for the next unit's loads as soon as the prologue has copied them.
  const uint32_t tmem_s = tmem, tmem_dp = tmem + 128, tmem_dq = tmem + 256, tmem_q = tmem + 384, tmem_do = tmem + 448;
  // Everything above (barriers, TMEM) overlapped the tail of the kernel before this one in the stream; any of this
  // kernel's inputs may come from it, so nothing is read from global memory before this point.  The dK/dV kernel that
  // follows may start its CTAs as SMs free up: it only depends on this kernel for `delta`.
  grid_dep_wait();
  grid_dep_launch();

  if (warp == kBwdGroups * 4) {
    if (lane == 0) {
      prefetch_tensormap(&tm_q);
      prefetch_tensormap(&tm_k);
      prefetch_tensormap(&tm_v);
      prefetch_tensormap(&tm_do);
      prefetch_tensormap(&tm_o);
      int it = 0, u = 0;
      for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
        if (skipped(w)) continue;
        const int t = unit_tile(w), bh = w % BH, b = bh / H, h = bh - b * H;
        const int total = unit_items(w), n_last = total - 1;
        const uint32_t qb = smem_u32(&sm->qdo_full);
        mbar_wait(smem_u32(&sm->delta_read), (u & 1) ^ 1, &g_lmk_status, kErrDqProducer);
        mbar_arrive_expect_tx(qb, 3 * (kD / 64) * kTileBytes);
        for (int c = 0; c < kD / 64; ++c) {
          tma_load_4d(o_tile + c * kTileBytes, &tm_o, qb, 64 * c, t * kQTile, h, b);
          tma_load_4d(q_tile + c * kTileBytes, &tm_q, qb, 64 * c, t * kQTile, h, b);
          tma_load_4d(do_tile + c * kTileBytes, &tm_do, qb, 64 * c, t * kQTile, h, b);
        }
        int next_end = kIrr ? end_of(b, n_last) : 0;     // read one tile ahead: the table may be in global memory
        for (int i = 0; i < total; ++i, ++it) {
          const int s = it % kDqStages;
          const int n = n_last - i, r0 = kIrr ? next_end - 63 : n * kBlk;
          if (kIrr && n > 0) next_end = end_of(b, n - 1);
          mbar_wait(smem_u32(&sm->empty[s]), ((it / kDqStages) & 1) ^ 1, &g_lmk_status, kErrDqProducer);
          const uint32_t fb = smem_u32(&sm->full[s]);
          mbar_arrive_expect_tx(fb, 2 * (kD / 64) * kHalfTile);
          for (int c = 0; c < kD / 64; ++c) {
            tma_load_4d(k_slot(s) + c * kHalfTile, &tm_k, fb, 64 * c, r0, h, b);
            tma_load_4d(v_slot(s) + c * kHalfTile, &tm_v, fb, 64 * c, r0, h, b);
          }
        }
        ++u;
      }
    }
    __syncwarp();
  } else if (warp == kBwdGroups * 4 + 1 || warp == kBwdGroups * 4 + 3) {
    // warp +1 issues S = Q K^T, warp +3 issues dP = dO V^T; both walk through the same items and wait for the same
    // barriers (each is a waiter of its own on full / ops_ready and sees every phase)
    constexpr uint32_t fmt = kBf16 ? 1u : 0u;
    constexpr uint32_t idesc_s = instr_desc_f16(fmt, 128, 64, 0, 0);
    const bool is_s = warp == kBwdGroups * 4 + 1;
    const uint64_t db0 = smem_desc_sw128(is_s ? k_slot(0) : v_slot(0), 16, 1024);
    const uint32_t t_out = is_s ? tmem_s : tmem_dp, t_a = is_s ? tmem_q : tmem_do;
    int it = 0, u = 0;
    for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
      if (warp_uniform(skipped(w))) continue;
      const int total = warp_uniform(unit_items(w));
      for (int i = 0; i < total; ++i, ++it) {
        const int s = it % kDqStages, sb = it % kSdpBufs;
        mbar_wait(smem_u32(&sm->full[s]), (it / kDqStages) & 1, &g_lmk_status, kErrDqMma);
        if (it >= kSdpBufs)
          mbar_wait(smem_u32(is_s ? &sm->s_free[sb] : &sm->dp_free[sb]), ((it / kSdpBufs) & 1) ^ 1, &g_lmk_status, kErrDqMma);
        // the unit's rows come last: waited for in front of the other two they cost the unit another 1000 clk
        if (i == 0) mbar_wait(smem_u32(&sm->ops_ready), u & 1, &g_lmk_status, kErrDqMma);
        tc_fence_after();
        const uint64_t db = desc_advance(db0, (uint32_t)s * 32768u);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kD / 16; ++kk)      // A from TMEM: 8 columns = 16 features per K-step
            mma_f16_ts(t_out + sb * 64, t_a + kk * 8, desc_advance(db, kmajor_step(kk, kHalfTile)), idesc_s, kk > 0);
          mma_commit(smem_u32(is_s ? &sm->s_full[sb] : &sm->dp_full[sb]));
        }
      }
      if (elect_one()) mma_commit(smem_u32(&sm->ops_free));        // the next unit's Q / dO rows may be written
      ++u;
    }
    __syncwarp();
  } else if (warp == kBwdGroups * 4 + 2) {
    constexpr uint32_t fmt = kBf16 ? 1u : 0u;
    constexpr uint32_t idesc_q = instr_desc_f16(fmt, 128, kD, 0, 1);   // dQ += dS K  (K is MN-major)
    const uint64_t dv0 = smem_desc_sw128(v_slot(0), 16, 1024);
    const uint64_t dk0t = smem_desc_sw128(k_slot(0), kHalfTile, 1024);
    int it = 0, u = 0;
    for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
      if (warp_uniform(skipped(w))) continue;
      const int total = warp_uniform(unit_items(w));
      for (int i = 0; i < total; ++i, ++it) {
        const int s = it % kDqStages;
        if (i == 0) mbar_wait(smem_u32(&sm->acc_empty), (u & 1) ^ 1, &g_lmk_status, kErrDqMma);
        mbar_wait(smem_u32(&sm->ds_ready[s]), (it / kDqStages) & 1, &g_lmk_status, kErrDqMma);
        tc_fence_after();
        const uint64_t dds = desc_advance(dv0, (uint32_t)s * 32768u), dkt = desc_advance(dk0t, (uint32_t)s * 32768u);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kBlk / 16; ++kk)
            mma_f16_ss(tmem_dq, desc_advance(dds, kk * 32), desc_advance(dkt, kk * 2048), idesc_q,
                       (i > 0 || kk > 0) ? 1u : 0u);
          mma_commit(smem_u32(&sm->empty[s]));
        }
      }
      if (elect_one()) mma_commit(smem_u32(&sm->acc_full[(it - 1) & 1]));     // drained by the warpgroup that took the last item
      ++u;
    }
    __syncwarp();
  } else {
    const int g = warp >> 2;                       // warpgroup: items with (running item count) % 2 == g
    const int row = tid & 127;
    const int half = row >> 6;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    int it0 = 0, u = 0, drains = 0;
    // dQ of a unit is drained by the warpgroup that took its last item, but only after that warpgroup has done the
    // prologue of the NEXT unit: the last dQ product queues behind the next unit's first S / dP products, so an
    // immediate drain would just wait for it.  (The next unit's first dQ product needs its first dS, far later.)
    int64_t drain_row = -1;
    bool drain_valid = false;                      // rows past the end of the sequence are computed and dropped
    auto drain = [&]() {
      mbar_wait(smem_u32(&sm->acc_full[g]), drains & 1, &g_lmk_status, kErrDqEpilogue);
      ++drains;
      tc_fence_after();
      if (kIrr) __syncwarp();
      uint4* orow = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(dq_ptr) + drain_row * D);
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_dq + c * 32 + lane_base, r);
        tmem_ld_wait();
        if (c == kD / 32 - 1) {
          tc_fence_before();
          mbar_arrive(smem_u32(&sm->acc_empty));     // the next unit may start accumulating
        }
#pragma unroll
        for (int v4 = 0; v4 < 4; ++v4) {
          uint4 pk;
          pk.x = pack2<kBf16>(__uint_as_float(r[8 * v4 + 0]), __uint_as_float(r[8 * v4 + 1]));
          pk.y = pack2<kBf16>(__uint_as_float(r[8 * v4 + 2]), __uint_as_float(r[8 * v4 + 3]));
          pk.z = pack2<kBf16>(__uint_as_float(r[8 * v4 + 4]), __uint_as_float(r[8 * v4 + 5]));
          pk.w = pack2<kBf16>(__uint_as_float(r[8 * v4 + 6]), __uint_as_float(r[8 * v4 + 7]));
          if (kWhole || (drain_valid && c * 32 + v4 * 8 < D)) orow[c * 4 + v4] = pk;
        }
      }
      drain_row = -1;
    };
    // The row statistics of the next unit are fetched while the current one runs, so their latency is never exposed.  The forward
    // kernel in front writes them and may be running when this kernel starts.
    float nM = 0.f, nL = 1.f;
    auto fetch_rows = [&](int w) {
      if (w >= n_units) return;
      const int r = unit_tile(w) * kQTile + row;
      const int64_t at = (int64_t)(w % BH) * Lq + (kWhole ? r : min(r, Lq - 1));
      nM = ld_behind_wait((kIrr && irr.R != nullptr ? irr.R : M_ptr) + at);
      nL = kIrr && irr.R != nullptr ? 1.f : ld_behind_wait(L_ptr + at);
    };
    fetch_rows(unit_of(0));
    for (int r = 0, w = unit_of(0); w < n_units; w = unit_of(++r)) {
      const int t = unit_tile(w), bh = w % BH, b = bh / H;
      int total = kIrr ? 0 : unit_items(w);
      const int64_t grow = (int64_t)bh * Lq + t * kQTile + row;
      const bool row_valid = kWhole || t * kQTile + row < Lq;
      const float M2L = kIrr && irr.R != nullptr ? nM : fmaf(nM, kLog2e, __log2f(nL));
      fetch_rows(unit_of(r + 1));
      // tile table: everything that depends on the unit alone first, then what hangs on it (kIrr: loads from global memory)
      const int pos = min(Lk - Lq + t * kQTile + row, Lk - 1);
      const bool skip = skipped(w);
      if constexpr (kIrr) total = warp_uniform(unit_items(w));
      const int n_last = total - 1;
      const int own = kIrr ? group_of(b, pos) : prefix_blocks + 2 * t + half;
      if (skip) continue;                           // after the prefetch, which belongs to the next unit
      const int end_own = kIrr ? end_of(b, own) : 0;
      // kIrr: first visible column of this warpgroup's items, read one item ahead (hidden columns of tile n)
      auto first_col = [&](int n) { return n < 0 ? 0 : warp_uniform(64 - (end_of(b, n) - (n > 0 ? end_of(b, n - 1) : -1))); };
      int c0 = kIrr ? first_col(n_last - ((it0 + g) & 1)) : 0;
      const int vis = min(kIrr ? 63 - (end_own - pos) : row & 63, kBlk - 2);
      // delta = rowsum(O * dO), straight from the swizzled tiles (one row per thread, 16-byte chunks); warpgroup 0
      // also publishes it for the dK/dV kernel, which runs after this one
      mbar_wait(smem_u32(&sm->qdo_full), u & 1, &g_lmk_status, kErrDqSoftmax);
      float delta = 0.f;
      uint32_t opw[kD / 64][32];      // this thread's row of the operand its warpgroup moves to TMEM (0: Q, 1: dO)
#pragma unroll
      for (int sub = 0; sub < kD / 64; ++sub)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t off = (uint32_t)sub * kTileBytes + (uint32_t)row * 128u + (uint32_t)((c ^ (row & 7)) << 4);
          uint32_t ov[4], gv[4];
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(ov[0]), "=r"(ov[1]), "=r"(ov[2]), "=r"(ov[3]) : "r"(o_tile + off));
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(gv[0]), "=r"(gv[1]), "=r"(gv[2]), "=r"(gv[3]) : "r"(do_tile + off));
          if (g == 1) {
#pragma unroll
            for (int e = 0; e < 4; ++e) opw[sub][4 * c + e] = gv[e];
          } else {
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(opw[sub][4 * c]), "=r"(opw[sub][4 * c + 1]), "=r"(opw[sub][4 * c + 2]),
                           "=r"(opw[sub][4 * c + 3]) : "r"(q_tile + off));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float2 fo, fg;
            if (kBf16) {
              fo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ov[e]));
              fg = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gv[e]));
            } else {
              fo = __half22float2(*reinterpret_cast<const __half2*>(&ov[e]));
              fg = __half22float2(*reinterpret_cast<const __half2*>(&gv[e]));
            }
            delta = fmaf(fo.x, fg.x, delta);
            delta = fmaf(fo.y, fg.y, delta);
          }
        }
      // The shared-memory tiles may take the next unit's rows.  TMA writes them through another proxy than these loads went
      // through, and an arrival alone does not hold it back until they are done: of 15 000 calls at B4 H16 L1024 D64 twenty had
      // rows of dQ from tiles half overwritten, always of a unit with no more items than stages, behind which the producer is
      // already waiting.
      fence_proxy_async_smem();
      mbar_arrive(smem_u32(&sm->delta_read));
      // row -> TMEM lane, 32-bit word j (two features) -> column j: the layout of a K-major A operand
      mbar_wait(smem_u32(&sm->ops_free), (u & 1) ^ 1, &g_lmk_status, kErrDqSoftmax);
      tc_fence_after();
      if (kIrr) __syncwarp();
      {
        const uint32_t dst = (g == 0 ? tmem_q : tmem_do) + lane_base;
        tmem_st_32x32b_x32(dst, opw[0]);
        if constexpr (kD == 128) tmem_st_32x32b_x32(dst + 32, opw[1]);
        tmem_st_wait();
      }
      tc_fence_before();
      mbar_arrive(smem_u32(&sm->ops_ready));
      if (g == 0 && row_valid) delta_ptr[grow] = delta;
      if (drain_row >= 0) drain();
      for (int i = (it0 + g) & 1; i < total; i += kBwdGroups) {
        const int it = it0 + i;
        const int s = it % kDqStages, sb = it % kSdpBufs;
        const int n = n_last - i;
        mbar_wait(smem_u32(&sm->s_full[sb]), (it / kSdpBufs) & 1, &g_lmk_status, kErrDqSoftmax);
        tc_fence_after();
        const int kind = n > own ? 0 : (n == own ? 1 : 2);
        const int c_now = c0;
        if (kIrr) c0 = first_col(n - kBwdGroups);
        uint64_t sp[32];
        const RowFactors f = bwd_weights<kIrr>(sp, c_now, tmem_s + sb * 64 + lane_base, kind, vis, scale_log2, M2L, [&]() {
          tc_fence_before();
          mbar_arrive(smem_u32(&sm->s_free[sb]));
        });
        mbar_wait(smem_u32(&sm->dp_full[sb]), (it / kSdpBufs) & 1, &g_lmk_status, kErrDqSoftmax);
        tc_fence_after();
        uint32_t wd[32];
        bwd_dscores<kBf16, kIrr>(wd, sp, f, tmem_dp + sb * 64 + lane_base, smem_u32(&sm->dp_free[sb]), kind, scale, delta);
        store_row_sw128(v_slot(s), row, wd);      // dS replaces the V tile of this stage, which dP has finished reading
        fence_proxy_async_smem();
        mbar_arrive(smem_u32(&sm->ds_ready[s]));
      }
      it0 += total;
      if (g == ((it0 - 1) & 1)) {
        drain_row = grow;
        drain_valid = row_valid;
      }
      ++u;
    }
    if (drain_row >= 0) drain();
    tc_fence_before();
  }
  __syncthreads();
  if (warp == kBwdGroups * 4 + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Driver-API calls need the device's primary context current on the calling thread; autograd worker threads
// arrive here before any runtime call has bound it.  cudaSetDevice binds it without synchronising the device.
inline void bind_context() {
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) (void)cudaSetDevice(dev);
}

EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tensor maps are cached: a training loop calls with the same few (pointer, shape, strides) again and again, and
// encoding five or six maps per call is a noticeable part of the host time of a 50 us kernel.  The key holds
// everything the encoding depends on, so a hit is always valid (a map describes addresses, not contents); the table
// is small, shared by all threads and replaced round-robin.
struct MapKey {
  const void* ptr;
  int kind, dtype, B, H, L, box, D;
  int64_t st[3];
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && kind == o.kind && dtype == o.dtype && B == o.B && H == o.H && L == o.L && box == o.box &&
           D == o.D && st[0] == o.st[0] && st[1] == o.st[1] && st[2] == o.st[2];
  }
};
constexpr int kMapCacheSize = 64;
struct MapCache {
  std::mutex mu;
  MapKey keys[kMapCacheSize];
  CUtensorMap maps[kMapCacheSize];
  int used = 0, next = 0;
};
MapCache& map_cache() {
  static MapCache c;
  return c;
}

template <typename EncodeFn>
int cached_map(CUtensorMap* m, const MapKey& key, EncodeFn encode) {
  MapCache& c = map_cache();
  {
    std::lock_guard<std::mutex> lock(c.mu);
    for (int i = 0; i < c.used; ++i)
      if (c.keys[i] == key) {
        *m = c.maps[i];
        return LMK_OK;
      }
  }
  const int rc = encode(m);
  if (rc != LMK_OK) return rc;
  std::lock_guard<std::mutex> lock(c.mu);
  const int slot = c.used < kMapCacheSize ? c.used++ : (c.next++ % kMapCacheSize);
  c.keys[slot] = key;
  c.maps[slot] = *m;
  return LMK_OK;
}

// [B, H, L, D] tensor with element strides {b, h, row}; box = 64 features x `box_rows` rows, 128-byte swizzle; what lies
// outside the tensor (rows past L, features past D) reads as zeros
int make_map_4d(CUtensorMap* m, const void* ptr, int dtype, int B, int H, int L, int D, const int64_t st[3], int box_rows) {
  const MapKey key{ptr, 4, dtype, B, H, L, box_rows, D, {st[0], st[1], st[2]}};
  return cached_map(m, key, [&](CUtensorMap* out) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return fail(LMK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)L, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)st[2] * 2, (cuuint64_t)st[1] * 2, (cuuint64_t)st[0] * 2};
    cuuint32_t box[4] = {64, (cuuint32_t)box_rows, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(out, dtype == LMK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                     const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(LMK_ERR_CUDA, "cuTensorMapEncodeTiled (4-D) failed with %d", (int)r);
    return (int)LMK_OK;
  });
}

// landmark keys: k viewed as [B, H, L/64, 64, D]; box = 64 features x 1 row-in-block x 64 blocks
int make_map_landmarks(CUtensorMap* m, const void* ptr, int dtype, int B, int H, int L, int D, const int64_t st[3],
                       int lm_box) {
  const MapKey key{ptr, 5, dtype, B, H, L, lm_box, D, {st[0], st[1], st[2]}};
  return cached_map(m, key, [&](CUtensorMap* out) {
    EncodeTiledFn enc = get_encode();
    if (!enc) return fail(LMK_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    // whole blocks only (the rows of a partial last block have no landmark among them); a sequence shorter than one block
    // has no landmark row at all, and its map no row 63
    cuuint64_t dims[5] = {(cuuint64_t)D, (cuuint64_t)(L < kBlk ? L : kBlk), (cuuint64_t)(L < kBlk ? 1 : L / kBlk), (cuuint64_t)H,
                          (cuuint64_t)B};
    cuuint64_t strides[4] = {(cuuint64_t)st[2] * 2, (cuuint64_t)st[2] * 2 * kBlk, (cuuint64_t)st[1] * 2,
                             (cuuint64_t)st[0] * 2};
    cuuint32_t box[5] = {64, 1, (cuuint32_t)lm_box, 1, 1};
    cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    CUresult r = enc(out, dtype == LMK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5,
                     const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(LMK_ERR_CUDA, "cuTensorMapEncodeTiled (landmarks) failed with %d", (int)r);
    return (int)LMK_OK;
  });
}

// Per-device launch facts, looked up once: the SM count and the opt-in to large dynamic shared memory for every kernel
// of this file (the attribute is a property of the function on a device, not of a launch).
constexpr int kMaxDevices = 64;
struct DeviceFacts {
  bool ready = false;
  int n_sm = 0;
};
template <int kTiles> constexpr size_t fwd_smem(bool irr) {
  return 1024 + (kTiles + kFwdStages<kTiles>) * 32768 + sizeof(Fwd2Smem<kFwdStages<kTiles>>) + (irr ? sizeof(IrrSmem) : 0);
}
static_assert(fwd_smem<2>(true) <= 232448 && fwd_smem<1>(true) <= 232448 / 2 - 1024, "shared memory of one SM");
template <int kD> constexpr size_t kSmemDkv =
    1024 + (2 + 2 * kDkvStages<kD>) * (kD / 64) * kTileBytes + 2 * kTileBytes + sizeof(DkvSmem<kDkvStages<kD>>);
static_assert(kSmemDkv<128> <= 232448 && kSmemDkv<64> <= 232448, "shared memory of one SM");
constexpr size_t kSmemDq = 1024 + 65536 + kDqStages * 32768 + 32768 + sizeof(DqSmem);

int device_facts(const DeviceFacts** out) {
  static std::mutex mu;
  static DeviceFacts facts[kMaxDevices];
  int dev = 0;
  LMK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(LMK_ERR_UNSUPPORTED, "device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  DeviceFacts& f = facts[dev];
  if (!f.ready) {
    LMK_CUDA(cudaDeviceGetAttribute(&f.n_sm, cudaDevAttrMultiProcessorCount, dev));
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
#define LMK_ATTRS(BF, DIM)                                                                                   \
    LMK_CUDA(cudaFuncSetAttribute(sm100_fwd2_kernel<BF, DIM, false, 1>, attr, (int)fwd_smem<1>(false)));     \
    LMK_CUDA(cudaFuncSetAttribute(sm100_fwd2_kernel<BF, DIM, true, 1>, attr, (int)fwd_smem<1>(true)));       \
    LMK_CUDA(cudaFuncSetAttribute(sm100_fwd2_kernel<BF, DIM, false, 2>, attr, (int)fwd_smem<2>(false)));     \
    LMK_CUDA(cudaFuncSetAttribute(sm100_fwd2_kernel<BF, DIM, true, 2>, attr, (int)fwd_smem<2>(true)));       \
    LMK_CUDA(cudaFuncSetAttribute(sm100_bwd_dq_kernel<BF, DIM, true, false>, attr, (int)kSmemDq));           \
    LMK_CUDA(cudaFuncSetAttribute(sm100_bwd_dq_kernel<BF, DIM, false, false>, attr, (int)kSmemDq));          \
    LMK_CUDA(cudaFuncSetAttribute(sm100_bwd_dq_kernel<BF, DIM, false, true>, attr, (int)kSmemDq));           \
    LMK_CUDA(cudaFuncSetAttribute(sm100_bwd_dkv_kernel<BF, DIM, true, false>, attr, (int)kSmemDkv<DIM>));    \
    LMK_CUDA(cudaFuncSetAttribute(sm100_bwd_dkv_kernel<BF, DIM, false, false>, attr, (int)kSmemDkv<DIM>));   \
    LMK_CUDA(cudaFuncSetAttribute(sm100_bwd_dkv_kernel<BF, DIM, false, true>, attr, (int)kSmemDkv<DIM>));
    LMK_ATTRS(true, 128) LMK_ATTRS(true, 64) LMK_ATTRS(false, 128) LMK_ATTRS(false, 64)
#undef LMK_ATTRS
    f.ready = true;
  }
  *out = &f;
  return LMK_OK;
}

// Upper bound on the CTAs of the persistent backward kernels; 0 = one per SM.  Only the tests lower it (to make every
// CTA walk through several work units at small sizes).
std::atomic<int> g_max_ctas{0};

// A tensor the TMA unit can address: 16-byte aligned base, positive strides that are multiples of 16 bytes
// (an expanded view has stride 0), rows at least one head apart.
bool tma_ok(const void* p, const int64_t st[3], int D = 128) {
  return ((uintptr_t)p % 16 == 0) && st[0] > 0 && st[1] > 0 && st[0] % 8 == 0 && st[1] % 8 == 0 && st[2] % 8 == 0 &&
         st[2] >= D;
}

}  // namespace

// whole tiles of full head dim: what an explicit request for this path asks for
bool attn_sm100_supported(int B, int H, int Lq, int Lk, int D, int block, int dtype) {
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D == 128 && block == kBlk && Lq >= kQTile && Lq % kQTile == 0 &&
         Lk % kBlk == 0 && Lk >= Lq && B >= 1 && H >= 1;
}

// everything the kernels take: any length (rows past the end read as zeros and are dropped), head dims below 128 (features
// past the end read as zeros; at most 64 of them run with half the products)
bool attn_sm100_takes(int B, int H, int Lq, int Lk, int D, int block, int dtype) {
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D >= 8 && D <= 128 && D % 8 == 0 && block == kBlk && Lq >= 1 &&
         Lk >= Lq && (Lk - Lq) % kBlk == 0 && B >= 1 && H >= 1;
}

bool attn_sm100_operands_ok(const AttnParams& p, bool backward) {
  if (!tma_ok(p.q, p.qs, p.D) || !tma_ok(p.k, p.ks, p.D) || !tma_ok(p.v, p.vs, p.D)) return false;
  if (backward && (!tma_ok(p.dO, p.dos, p.D) || (uintptr_t)p.o % 16 != 0)) return false;
  return true;
}

void attn_sm100_set_max_ctas(int n) { g_max_ctas.store(n > 0 ? n : 0); }

int tensor_map_4d(CUtensorMap* m, const void* ptr, int dtype, int B, int H, int L, const int64_t st[3], int box_rows) {
  bind_context();
  return make_map_4d(m, ptr, dtype, B, H, L, 128, st, box_rows);
}
bool tensor_map_operand_ok(const void* p, const int64_t st[3]) { return tma_ok(p, st); }

// Two query tiles a CTA share one K/V stream; one tile a CTA puts two CTAs on an SM, whose starts and ends overlap and which the
// hardware deals out in smaller pieces.  Measured (us, one / two):
//   D128, 32 heads of L = 512 11.5 / 13.5, 768 15.3 / 17.1, 896 19.2 / 17.3, 1024 22.2 / 20.7, 2048 43.0 / 39.9, 8192 545 / 469;
//   256 heads of 512 45.9 / 49.7.  Grids below 1.5 tiles an SM: 8 heads of 1024 18.0 / 18.8, 3072 44.1 / 45.1; at 1.73 (8 heads of
//   4096, 16 of 2048) both take the same.
//   Heads of 64 features have half the products for the stream to feed: 64 heads of 1024 22.2 / 25.7, of 2048 66 / 73, 32 heads of
//   4096 112 / 118, 8192 423 / 409; below two tiles an SM 8 heads of 4224 54 / 67, 4 of 8192 98 / 120.  Above 32 tiles one stays
//   ahead up to about five an SM (8 heads of 6144 80 / 94, 16 of 6144 127 / 133), where the line does not lie yet.
//   Groups as key tiles, D128: 51 keys, 128 heads of 512 29.6 / 31.7, 32 heads of 1024 28.2 / 31.4, of 1664 51 / 55, 1920 65 / 67;
//   32-key blocks, 32 heads of 1280 51.1 / 54.1, 1700 70 / 68 (an even number of tiles), 1920 81 / 86, 2000 90 / 86, 16 heads of
//   2000 (below two tiles an SM) 74 / 80.  D64: 32-key blocks, 64 heads of 1920 131 / 148, 2000 148 / 153.
// A single tile of a long history wants the deeper pipeline of the second form.
static int fwd_tiles_per_cta(int n_tiles, int BH, int n_sm, bool irr, int D) {
  if (n_tiles == 1) return 2;
  const int most = irr ? (D <= 64 ? 16 : 15) : (D <= 64 ? 32 : 6);
  const int64_t few = irr || D <= 64 ? 2 * n_sm : n_sm + n_sm / 2;
  return n_tiles <= most || (int64_t)n_tiles * BH <= few ? 1 : 2;
}

static int launch_fwd(const AttnParams& p, int dtype, const IrrArgs* irr, cudaStream_t st) {
  if (!attn_sm100_operands_ok(p, false))
    return fail(LMK_ERR_UNSUPPORTED, "tcgen05 path needs 16-byte aligned q/k/v with strides that are multiples of 8");
  bind_context();
  CUtensorMap tq, tk, tv, tl;
  int rc;
  if ((rc = make_map_4d(&tq, p.q, dtype, p.B, p.H, p.Lq, p.D, p.qs, kQTile)) != LMK_OK) return rc;
  if ((rc = make_map_4d(&tk, p.k, dtype, p.B, p.H, p.Lk, p.D, p.ks, kBlk)) != LMK_OK) return rc;
  if ((rc = make_map_4d(&tv, p.v, dtype, p.B, p.H, p.Lk, p.D, p.vs, kBlk)) != LMK_OK) return rc;
  const int whole_blocks = p.Lk / kBlk;
  const int lm_box = whole_blocks < 1 ? 1 : (whole_blocks < 64 ? whole_blocks : 64);
  const bool other = irr != nullptr && (irr->flags != nullptr || irr->block != 0);      // not the block-64 pattern
  if (other) tl = tk;               // not read
  else if ((rc = make_map_landmarks(&tl, p.k, dtype, p.B, p.H, p.Lk, p.D, p.ks, lm_box)) != LMK_OK) return rc;
  const float scale_log2 = p.scale * kLog2e;
  const DeviceFacts* facts = nullptr;
  if ((rc = device_facts(&facts)) != LMK_OK) return rc;
  const int n_tiles = (p.Lq + kQTile - 1) / kQTile;
  const int per_cta = fwd_tiles_per_cta(n_tiles, p.B * p.H, facts->n_sm, other, p.D);
  const dim3 grid(p.B * p.H, (n_tiles + per_cta - 1) / per_cta);
  // With the programmatic-stream-serialization attribute the set-up (barriers, TMEM, tensor maps) may run while the kernel in
  // front drains: it is a quarter of a short prompt's time (L = 77: 8.2 -> 5.9 us a call).
  cudaLaunchAttribute pdl[1];
  pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.stream = st;
  cfg.attrs = pdl;
  cfg.numAttrs = 1;
#define LMK_FWD_LAUNCH(BF, DIM, IRR, TILES)                                                                              \
  do {                                                                                                                   \
    cfg.blockDim = dim3(kFwdThreads<TILES>);                                                                             \
    cfg.dynamicSmemBytes = fwd_smem<TILES>(IRR);                                                                         \
    LMK_CUDA(cudaLaunchKernelEx(&cfg, sm100_fwd2_kernel<BF, DIM, IRR, TILES>, tq, tk, tv, tl, (void*)p.o, p.L, p.M, p.H, \
                                p.Lq, p.Lk, p.D, lm_box, scale_log2, (const void*)p.k, p.ks[0], p.ks[1], p.ks[2], args)); \
  } while (0)
#define LMK_FWD_TILES(BF, DIM, IRR)                                                           \
  do {                                                                                        \
    if (per_cta == 1) LMK_FWD_LAUNCH(BF, DIM, IRR, 1);                                        \
    else LMK_FWD_LAUNCH(BF, DIM, IRR, 2);                                                     \
  } while (0)
#define LMK_FWD_DTYPE(BF)                                                                     \
  do {                                                                                        \
    if (other) {                                                                     \
      if (p.D <= 64) LMK_FWD_TILES(BF, 64, true); else LMK_FWD_TILES(BF, 128, true);          \
    } else {                                                                                  \
      if (p.D <= 64) LMK_FWD_TILES(BF, 64, false); else LMK_FWD_TILES(BF, 128, false);        \
    }                                                                                         \
  } while (0)
  const IrrArgs args = irr != nullptr ? *irr : IrrArgs{};
  if (dtype == LMK_BF16) LMK_FWD_DTYPE(true);
  else LMK_FWD_DTYPE(false);
#undef LMK_FWD_DTYPE
#undef LMK_FWD_TILES
#undef LMK_FWD_LAUNCH
  LMK_CUDA(cudaGetLastError());
  return LMK_OK;
}

int attn_sm100_fwd(const AttnParams& p, int dtype, cudaStream_t st) { return launch_fwd(p, dtype, nullptr, st); }

// blocks below 64 in a regular pattern
bool attn_sm100_small_blocks(int B, int H, int Lq, int Lk, int D, int block, int dtype) {
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D >= 8 && D <= 128 && D % 8 == 0 && block >= 2 && block < kBlk && Lq >= 1 &&
         Lk >= Lq && (Lk - 1) / block < kIrrMaxTiles && B >= 1 && H >= 1;
}
int attn_sm100_small_blocks_fwd(const AttnParams& p, int dtype, cudaStream_t st) {
  IrrArgs a;
  a.block = p.block;
  return launch_fwd(p, dtype, &a, st);
}
// forward only, R instead of p.L and p.M (blocks of 64 or below)
int attn_sm100_fwd_lse(const AttnParams& p, float* R, int dtype, cudaStream_t st) {
  IrrArgs a;
  a.block = p.block == kBlk ? 0 : p.block;
  a.R = R;
  return launch_fwd(p, dtype, &a, st);
}
// landmarks anywhere: p.o and R; rows of the batch left to the two-pass kernels are marked in R
bool attn_sm100_flags(int Lk, int G) { return Lk <= kIrrMaxKeys && Lk <= kBlk * (G + 1); }
int attn_sm100_flags_fwd(const AttnParams& p, const uint8_t* flags, int64_t stride, int G, float* R, int dtype, cudaStream_t st) {
  IrrArgs a;
  a.flags = flags;
  a.stride = stride;
  a.G = G;
  a.R = R;
  return launch_fwd(p, dtype, &a, st);
}

static int launch_bwd(const AttnParams& p, int dtype, const IrrArgs* irr, cudaStream_t st) {
  if (!attn_sm100_operands_ok(p, true))
    return fail(LMK_ERR_UNSUPPORTED, "tcgen05 path needs 16-byte aligned tensors with strides that are multiples of 8");
  bind_context();
  CUtensorMap tq, tk, tv, tdo;
  int rc;
  const int64_t dense[3] = {(int64_t)p.H * p.Lq * p.D, (int64_t)p.Lq * p.D, (int64_t)p.D};
  if ((rc = make_map_4d(&tq, p.q, dtype, p.B, p.H, p.Lq, p.D, p.qs, kQTile)) != LMK_OK) return rc;
  if ((rc = make_map_4d(&tk, p.k, dtype, p.B, p.H, p.Lk, p.D, p.ks, kBlk)) != LMK_OK) return rc;
  if ((rc = make_map_4d(&tv, p.v, dtype, p.B, p.H, p.Lk, p.D, p.vs, kBlk)) != LMK_OK) return rc;
  if ((rc = make_map_4d(&tdo, p.dO, dtype, p.B, p.H, p.Lq, p.D, p.dos, kQTile)) != LMK_OK) return rc;
  float* delta = reinterpret_cast<float*>(p.workspace);
  const float scale_log2 = p.scale * kLog2e;
  const size_t smem_dkv = p.D <= 64 ? kSmemDkv<64> : kSmemDkv<128>, smem_dq = kSmemDq;
  CUtensorMap to;
  if ((rc = make_map_4d(&to, p.o, dtype, p.B, p.H, p.Lq, p.D, dense, kQTile)) != LMK_OK) return rc;
  const DeviceFacts* facts = nullptr;
  if ((rc = device_facts(&facts)) != LMK_OK) return rc;
  int n_sm = facts->n_sm;
  const int cap = g_max_ctas.load();
  if (cap >= 1 && cap < n_sm) n_sm = cap;
  // key tiles of a batch row: whole blocks, or at most that many groups
  const int max_tiles = irr == nullptr ? (p.Lk + kBlk - 1) / kBlk
                        : irr->flags != nullptr ? (irr->G < kIrrMaxTiles - 1 ? irr->G : kIrrMaxTiles - 1) + 1
                                                : (p.Lk - 1) / irr->block + 1;
  const int dkv_units = ((max_tiles + 1) / 2) * p.B * p.H;
  const int dq_units = ((p.Lq + kQTile - 1) / kQTile) * p.B * p.H;
  dim3 grid_dkv(dkv_units < n_sm ? dkv_units : n_sm), grid_dq(dq_units < n_sm ? dq_units : n_sm);
  // Both launches can carry the programmatic-stream-serialization attribute.  The dQ kernel waits for the kernel before it
  // right after its set-up (only the set-up overlaps).  The dK/dV kernel reads q, k, v, dO, L, M and the tile table, which
  // were complete before any CTA of the dQ kernel was behind its wait and could let this one start, and `delta`, which the
  // dQ kernel writes: its loads and S / dP products start on every SM the dQ kernel has left, and only its softmax threads
  // wait (griddepcontrol.wait) before they read delta.
  // (Blocks of 64 at B1 H32 L2048 206 -> 203 us, B4 H16 L1024 D64 120 -> 118.5; the layer with groups of 51 at B16 H8 T512
  // 166.7 -> 161.2.)
  cudaLaunchAttribute pdl[1];
  pdl[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg_dq = {}, cfg_dkv = {};
  cfg_dq.gridDim = grid_dq;  cfg_dq.blockDim = dim3(kDqThreads);  cfg_dq.dynamicSmemBytes = smem_dq;  cfg_dq.stream = st;
  cfg_dq.attrs = pdl;  cfg_dq.numAttrs = 1;
  cfg_dkv.gridDim = grid_dkv;  cfg_dkv.blockDim = dim3(kBwdThreads);  cfg_dkv.dynamicSmemBytes = smem_dkv;
  cfg_dkv.stream = st;  cfg_dkv.attrs = pdl;  cfg_dkv.numAttrs = 1;
  const float* Lc = p.L;
  const float* Mc = p.M;
  const float* deltac = delta;
  const int BH = p.B * p.H;
#define LMK_BWD_LAUNCH(BF, DIM, WHOLE, IRR)                                                                                \
  do {                                                                                                                     \
    LMK_CUDA(cudaLaunchKernelEx(&cfg_dq, sm100_bwd_dq_kernel<BF, DIM, WHOLE, IRR>, tq, tk, tv, tdo, to, Lc, Mc, delta,     \
                                p.dq, p.H, BH, p.Lq, p.Lk, p.D, p.scale, scale_log2, args));                               \
    LMK_CUDA(cudaLaunchKernelEx(&cfg_dkv, sm100_bwd_dkv_kernel<BF, DIM, WHOLE, IRR>, tq, tk, tv, tdo, Lc, Mc, deltac,      \
                                p.dk, p.dv, p.H, BH, p.Lq, p.Lk, p.D, p.scale, scale_log2, max_tiles, args));              \
  } while (0)
#define LMK_BWD_DIM(BF, DIM)                                                   \
  do {                                                                         \
    if (irr != nullptr) LMK_BWD_LAUNCH(BF, DIM, false, true);                  \
    else if (whole && p.D == DIM) LMK_BWD_LAUNCH(BF, DIM, true, false);        \
    else LMK_BWD_LAUNCH(BF, DIM, false, false);                                \
  } while (0)
#define LMK_BWD_DTYPE(BF)                                                      \
  do {                                                                         \
    if (p.D <= 64) LMK_BWD_DIM(BF, 64);                                        \
    else LMK_BWD_DIM(BF, 128);                                                 \
  } while (0)
  const IrrArgs args = irr != nullptr ? *irr : IrrArgs{};
  // instances without bounds where every tile is whole (the checks and run-time strides cost 8 us of 147 at L = 2048)
  const bool whole = p.Lq % kQTile == 0 && p.Lk % kBlk == 0;
  if (dtype == LMK_BF16) LMK_BWD_DTYPE(true);
  else LMK_BWD_DTYPE(false);
#undef LMK_BWD_DTYPE
#undef LMK_BWD_DIM
#undef LMK_BWD_LAUNCH
  LMK_CUDA(cudaGetLastError());
  return LMK_OK;
}

int attn_sm100_bwd(const AttnParams& p, int dtype, cudaStream_t st) { return launch_bwd(p, dtype, nullptr, st); }
int attn_sm100_small_blocks_bwd(const AttnParams& p, int dtype, cudaStream_t st) {
  IrrArgs a;
  a.block = p.block;
  return launch_bwd(p, dtype, &a, st);
}
size_t attn_sm100_plan_bytes(int B) { return sizeof(int) * (size_t)B * kIrrPlanInts; }
// p.workspace: delta; plan: attn_sm100_plan_bytes(B), written here.  Word 1 of a batch row's record (attn_sm100_plan_stride ints
// apart) tells the two-pass kernels whether the row is theirs.
int attn_sm100_flags_bwd(const AttnParams& p, const uint8_t* flags, int64_t stride, int G, const float* R, int* plan, int dtype,
                         cudaStream_t st) {
  LMK_CUDA(launch_overlapped(irr_plan_kernel, dim3(p.B), dim3(256), 0, st, flags, stride, p.Lk, G, plan));
  IrrArgs a;
  a.flags = flags;
  a.stride = stride;
  a.G = G;
  a.R = const_cast<float*>(R);
  a.plan = plan;
  return launch_bwd(p, dtype, &a, st);
}
int attn_sm100_plan_stride() { return kIrrPlanInts; }

size_t attn_sm100_bwd_workspace(int B, int H, int Lq, int, int) { return sizeof(float) * (size_t)B * H * Lq; }

// Device address of the status word on the current device, for kernels compiled in other translation units.
int* device_status_word() {
  int* ptr = nullptr;
  if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_lmk_status) != cudaSuccess) return nullptr;
  return ptr;
}

int device_status(int* out, int clear) {
  int v = 0;
  LMK_CUDA(cudaDeviceSynchronize());
  LMK_CUDA(cudaMemcpyFromSymbol(&v, g_lmk_status, sizeof(int)));
  if (clear && v != 0) {
    int z = 0;
    LMK_CUDA(cudaMemcpyToSymbol(g_lmk_status, &z, sizeof(int)));
  }
  if (out) *out = v;
  return LMK_OK;
}

}  // namespace lmk
