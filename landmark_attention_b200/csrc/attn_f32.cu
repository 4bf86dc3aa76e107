// Fused landmark attention for fp32 tensors with blocks of 64 keys: fp32 products and sums on the CUDA cores.
//
// fp32 has no full-precision tensor-core path, so the bound is the FMA rate (74 TFLOP/s on 148 SMs); every product is a
// register-tiled one (4 x 4 results a thread and step of four features: 8 16-byte shared-memory loads for 64 FMAs, as packed
// pairs), rows in shared memory padded by four floats so that no load has bank conflicts, softmax in registers across the 16 lanes
// that share a row.  Tiles of 32 query rows: config 1 (B2 H8 L512 D64) gives 256 CTAs, the longest 8 key blocks.
//   forward   CTA per 32 rows; keys and values of the next block arrive (cp.async) under the other product of this one.
//   dQ        the same with S and dP; writes delta.
//   dK, dV    a cluster of two CTAs per key block: each takes every second tile of rows, partial sums are added through
//             distributed shared memory in a fixed order (bit-reproducible, no atomics).
// Measured at B2 H8 L512 D64 (before: one warp per 4 rows, scalar key loads): forward 214 -> 32, dQ 281 -> 43.5, dK/dV 362 -> 56 us;
// one group of threads a CTA took 46, 57 and 71.
// Math and statistics as in attn_general.cu, which keeps the other block sizes and unaligned operands.
#include <cooperative_groups.h>
#include "common.cuh"
#include "attn_params.h"
#include "sm100_ptx.cuh"

namespace lmk {
namespace {

namespace cg = cooperative_groups;
using ptx::fma2;
using ptx::pk2;
using ptx::upk2;

constexpr int kBK = 64;      // keys of a block
constexpr int kRT = 32;      // query rows of a tile
constexpr int kPS = 68;      // row stride of the probability tiles
constexpr int kSplit = 2;    // groups of threads that take the key blocks (dK / dV: the row tiles) of a CTA in turn

__device__ __forceinline__ void cp16(float* dst, const float* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Place in the order of falling work of the c-th of `total` CTAs on `slots` SMs, two of which fit an SM.  Up to twice the slots
// all are resident from the start, so the second of an SM has to be light where its first is heavy: the rest comes in the order
// of rising work.  (B2 H8 L512: at most 9 blocks an SM instead of 12; forward 36 -> 32, dQ 50 -> 43.5 us.)  Longer grids are dealt out as SMs
// become free, heaviest first.
__device__ __forceinline__ int work_rank(int c, int total, int slots) {
  return c >= slots && total <= 2 * slots ? total - 1 - (c - slots) : c;
}

// Groups of kThreads threads of a CTA run at their own pace: barrier number 1 + group.
template <int kThreads>
__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kThreads) : "memory");
}

// rows row0 .. row0+kRows-1 of a [.., D] tensor into a padded tile by kThreads threads (this one is `tid`); rows past `limit`
// and features past D become zeros
template <int kD, int kRows, int kThreads>
__device__ __forceinline__ void load_tile(float* tile, const float* base, int64_t row_stride, int row0, int limit, int D, int tid) {
  for (int e = tid; e < kRows * (kD / 4); e += kThreads) {
    const int r = e / (kD / 4), c = (e - r * (kD / 4)) * 4;
    const bool ok = row0 + r < limit && c < D;
    cp16(tile + r * (kD + 4) + c, ok ? base + (int64_t)(row0 + r) * row_stride + c : base, ok);
  }
}
struct alignas(16) F4 { uint64_t a, b; };      // four floats as two packed pairs
__device__ __forceinline__ F4 ld4(const float* p) { return *reinterpret_cast<const F4*>(p); }

// R x 4 dot products over kD features: rows ty + step_r * i of A against rows tx + 16 * j of B
template <int kD, int R>
__device__ __forceinline__ void dots(const float* A, int step_r, const float* B, int ty, int tx, float (&s)[R][4]) {
  uint64_t acc[R][4];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  const float* a0 = A + ty * (kD + 4);
  const float* b0 = B + tx * (kD + 4);
#pragma unroll 4
  for (int d = 0; d < kD; d += 4) {
    F4 av[R], bv[4];
#pragma unroll
    for (int i = 0; i < R; ++i) av[i] = ld4(a0 + step_r * i * (kD + 4) + d);
#pragma unroll
    for (int j = 0; j < 4; ++j) bv[j] = ld4(b0 + 16 * j * (kD + 4) + d);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fma2(av[i].a, bv[j].a, acc[i][j]);
        acc[i][j] = fma2(av[i].b, bv[j].b, acc[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float lo, hi;
      upk2(acc[i][j], lo, hi);
      s[i][j] = lo + hi;
    }
}

// acc[i][.] += sum_j W[row_i][j] * X[j][4 tx + ..]: rows ty + 8 i of a [32, 64] weight tile times a [64, kD] tile
template <int kD>
__device__ __forceinline__ void weighted_rows(const float* W, const float* X, int ty, int tx, uint64_t (&acc)[4][kD / 32]) {
#pragma unroll 2
  for (int j = 0; j < kBK; j += 4) {
    float4 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(W + (ty + 8 * i) * kPS + j);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      F4 x[kD / 64];
#pragma unroll
      for (int c = 0; c < kD / 64; ++c) x[c] = ld4(X + (j + u) * (kD + 4) + 64 * c + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float f = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
        const uint64_t ff = pk2(f, f);
#pragma unroll
        for (int c = 0; c < kD / 64; ++c) {
          acc[i][2 * c] = fma2(ff, x[c].a, acc[i][2 * c]);
          acc[i][2 * c + 1] = fma2(ff, x[c].b, acc[i][2 * c + 1]);
        }
      }
    }
  }
}
// reductions over the 16 lanes that share a row
__device__ __forceinline__ float max16(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float sum16(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// last visible key of block n for a row whose own block is `own`: all but the landmark, up to the row, none
__device__ __forceinline__ int last_key(int n, int own, int pos) {
  return n < own ? kBK - 2 : (n == own ? min(pos & 63, kBK - 2) : -1);
}

template <int kD> constexpr size_t fwd_smem_f32 = sizeof(float) * (kRT * (kD + 4) + kSplit * (2 * kBK * (kD + 4) + kRT * kPS));

template <int kD>
__global__ void __launch_bounds__(128 * kSplit, kD == 64 ? 2 : 1) f32_fwd_kernel(AttnParams p, int n_sm) {
  extern __shared__ __align__(16) float sm[];
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  float* Qs = sm;
  const int group = threadIdx.x >> 7, tid = threadIdx.x & 127, tx = tid & 15, ty = tid >> 4;
  float* Ks = Qs + kRT * (kD + 4) + group * (2 * kBK * (kD + 4) + kRT * kPS);
  float* Vs = Ks + kBK * (kD + 4);
  float* Ps = Vs + kBK * (kD + 4);
  const int BH = p.B * p.H, work = work_rank(blockIdx.x, gridDim.x, n_sm), bh = work % BH, b = bh / p.H, h = bh - b * p.H;
  const int q0 = ((int)gridDim.x / BH - 1 - work / BH) * kRT, prefix = p.Lk - p.Lq;
  const float* q = static_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const float* k = static_cast<const float*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const float* v = static_cast<const float*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const int n_last = (prefix + min(q0 + kRT, p.Lq) - 1) / kBK;
  load_tile<kD, kRT, 128 * kSplit>(Qs, q, p.qs[2], q0, p.Lq, p.D, threadIdx.x);
  load_tile<kD, kBK, 128>(Ks, k, p.ks[2], group * kBK, p.Lk, p.D, tid);
  cp_commit();
  load_tile<kD, kBK, 128>(Vs, v, p.vs[2], group * kBK, p.Lk, p.D, tid);
  cp_commit();
  int pos[4];
  float m[4], l[4];
  uint64_t acc[4][kD / 32];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    pos[i] = prefix + q0 + ty + 8 * i;
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < kD / 32; ++c) acc[i][c] = 0ull;
  }
  cp_wait<1>();
  __syncthreads();                             // every group's part of the rows
  for (int n = group; n <= n_last; n += kSplit) {
    cp_wait<1>();
    group_sync<128>(group);
    float s[4][4];
    dots<kD, 4>(Qs, 8, Ks, ty, tx, s);
    group_sync<128>(group);
    if (n + kSplit <= n_last) load_tile<kD, kBK, 128>(Ks, k, p.ks[2], (n + kSplit) * kBK, p.Lk, p.D, tid);
    cp_commit();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int own = pos[i] >> 6, last = last_key(n, own, pos[i]);
      const bool grouped = n < own;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] *= p.scale;
        if (tx + 16 * j <= last) mx = fmaxf(mx, s[i][j]);
      }
      mx = max16(mx);
      const float lm = __shfl_sync(0xffffffffu, s[i][3], (threadIdx.x & 16) | 15);
      const float m_new = fmaxf(m[i], grouped ? lm : mx);
      const float shift = grouped ? mx : m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = tx + 16 * j <= last ? expf(s[i][j] - shift) : 0.f;
        sum += s[i][j];
      }
      sum = sum16(sum);
      const float sc = last < 0 ? 1.f : expf(m[i] - m_new);
      const float el = grouped ? expf(lm - m_new) : sum;
      l[i] = l[i] * sc + (last < 0 ? 0.f : el);
      if (last >= 0) m[i] = m_new;
      const float w = grouped ? el / sum : 1.f;
      const uint64_t sc2 = pk2(sc, sc);
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) acc[i][c] = ptx::mul2(acc[i][c], sc2);
#pragma unroll
      for (int j = 0; j < 4; ++j) Ps[(ty + 8 * i) * kPS + tx + 16 * j] = s[i][j] * w;
    }
    cp_wait<1>();
    group_sync<128>(group);
    weighted_rows<kD>(Ps, Vs, ty, tx, acc);
    group_sync<128>(group);
    if (n + kSplit <= n_last) load_tile<kD, kBK, 128>(Vs, v, p.vs[2], (n + kSplit) * kBK, p.Lk, p.D, tid);
    cp_commit();
  }
  // the first group adds the others' sums in their order; each leaves its own in its key tile
  cp_wait<0>();
  if (group > 0) {
    group_sync<128>(group);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) reinterpret_cast<uint64_t*>(Ks)[(i * (kD / 32) + c) * 128 + tid] = acc[i][c];
      Vs[i * 128 + tid] = m[i];
      Vs[(4 + i) * 128 + tid] = l[i];
    }
  }
  __syncthreads();
  if (group > 0) return;
#pragma unroll
  for (int g = 1; g < kSplit; ++g) {
    const float* Kg = Ks + g * (2 * kBK * (kD + 4) + kRT * kPS);
    const float* Vg = Kg + kBK * (kD + 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float mg = Vg[i * 128 + tid], top = fmaxf(m[i], mg);
      const float fa = m[i] == -INFINITY ? 0.f : expf(m[i] - top), fb = mg == -INFINITY ? 0.f : expf(mg - top);
      const uint64_t fa2 = pk2(fa, fa), fb2 = pk2(fb, fb);
#pragma unroll
      for (int c = 0; c < kD / 32; ++c)
        acc[i][c] = fma2(reinterpret_cast<const uint64_t*>(Kg)[(i * (kD / 32) + c) * 128 + tid], fb2, ptx::mul2(acc[i][c], fa2));
      l[i] = l[i] * fa + Vg[(4 + i) * 128 + tid] * fb;
      m[i] = top;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + ty + 8 * i;
    if (row >= p.Lq) continue;
    float* o = static_cast<float*>(p.o) + ((int64_t)bh * p.Lq + row) * p.D;
    const float inv = 1.f / l[i];
#pragma unroll
    for (int c = 0; c < kD / 64; ++c) {
      float4 r;
      upk2(acc[i][2 * c], r.x, r.y);
      upk2(acc[i][2 * c + 1], r.z, r.w);
      const int d = 64 * c + 4 * tx;
      if (d < p.D) *reinterpret_cast<float4*>(o + d) = make_float4(r.x * inv, r.y * inv, r.z * inv, r.w * inv);
    }
    if (tx == 0) {
      p.L[(int64_t)bh * p.Lq + row] = l[i];
      p.M[(int64_t)bh * p.Lq + row] = m[i];
    }
  }
}

template <int kD> constexpr size_t dq_smem_f32 = sizeof(float) * (2 * kRT * (kD + 4) + kSplit * (2 * kBK * (kD + 4) + kRT * kPS));

template <int kD>
__global__ void __launch_bounds__(128 * kSplit, kD == 64 ? 2 : 1) f32_bwd_dq_kernel(AttnParams p, int n_sm) {
  extern __shared__ __align__(16) float sm[];
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  float* Qs = sm;
  float* Gs = Qs + kRT * (kD + 4);            // dO
  const int group = threadIdx.x >> 7, tid = threadIdx.x & 127, tx = tid & 15, ty = tid >> 4;
  float* Ks = Gs + kRT * (kD + 4) + group * (2 * kBK * (kD + 4) + kRT * kPS);
  float* Vs = Ks + kBK * (kD + 4);
  float* Ps = Vs + kBK * (kD + 4);            // dS
  const int BH = p.B * p.H, work = work_rank(blockIdx.x, gridDim.x, n_sm), bh = work % BH, b = bh / p.H, h = bh - b * p.H;
  const int q0 = ((int)gridDim.x / BH - 1 - work / BH) * kRT, prefix = p.Lk - p.Lq;
  const float* q = static_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const float* k = static_cast<const float*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const float* v = static_cast<const float*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const float* g = static_cast<const float*>(p.dO) + b * p.dos[0] + h * p.dos[1];
  const int n_last = (prefix + min(q0 + kRT, p.Lq) - 1) / kBK;
  load_tile<kD, kRT, 128 * kSplit>(Qs, q, p.qs[2], q0, p.Lq, p.D, threadIdx.x);
  load_tile<kD, kRT, 128 * kSplit>(Gs, g, p.dos[2], q0, p.Lq, p.D, threadIdx.x);
  load_tile<kD, kBK, 128>(Ks, k, p.ks[2], group * kBK, p.Lk, p.D, tid);
  load_tile<kD, kBK, 128>(Vs, v, p.vs[2], group * kBK, p.Lk, p.D, tid);
  cp_commit();
  int pos[4];
  float M[4], Linv[4], delta[4];
  uint64_t acc[4][kD / 32];
  cp_wait<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty + 8 * i, row = q0 + r;
    const bool ok = row < p.Lq;
    const int64_t gr = (int64_t)bh * p.Lq + row;
    pos[i] = prefix + row;
    M[i] = ok ? p.M[gr] : 0.f;
    Linv[i] = ok ? 1.f / p.L[gr] : 0.f;
    float d = 0.f;
    if (ok) {
      const float* o = static_cast<const float*>(p.o) + gr * p.D;
#pragma unroll
      for (int c = 0; c < kD / 16; ++c) {
        const int f = tx + 16 * c;
        if (f < p.D) d = fmaf(o[f], Gs[r * (kD + 4) + f], d);
      }
    }
    delta[i] = sum16(d);
    if (ok && tx == 0 && group == 0) p.delta[gr] = delta[i];
#pragma unroll
    for (int c = 0; c < kD / 32; ++c) acc[i][c] = 0ull;
  }
  for (int n = group; n <= n_last; n += kSplit) {
    if (n != group) {
      group_sync<128>(group);
      load_tile<kD, kBK, 128>(Ks, k, p.ks[2], n * kBK, p.Lk, p.D, tid);
      load_tile<kD, kBK, 128>(Vs, v, p.vs[2], n * kBK, p.Lk, p.D, tid);
      cp_commit();
      cp_wait<0>();
      group_sync<128>(group);
    }
    float s[4][4], dp[4][4];
    dots<kD, 4>(Qs, 8, Ks, ty, tx, s);
    dots<kD, 4>(Gs, 8, Vs, ty, tx, dp);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int own = pos[i] >> 6, last = last_key(n, own, pos[i]);
      const bool grouped = n < own;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] *= p.scale;
        if (tx + 16 * j <= last) mx = fmaxf(mx, s[i][j]);
      }
      mx = max16(mx);
      const float lm = __shfl_sync(0xffffffffu, s[i][3], (threadIdx.x & 16) | 15);
      const float shift = grouped ? mx : M[i];
      float den = 0.f, nD = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = tx + 16 * j <= last ? expf(s[i][j] - shift) : 0.f;
        den += s[i][j];
        nD = fmaf(s[i][j], dp[i][j], nD);
      }
      den = sum16(den);
      nD = sum16(nD);
      const float gw = grouped ? expf(lm - M[i]) * Linv[i] : 0.f;      // the landmark's probability
      const float sub = grouped ? nD / den : delta[i];
      const float w = (grouped ? gw / den : Linv[i]) * p.scale;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float ds = s[i][j] * w * (dp[i][j] - sub);
        if (grouped && tx == 15 && j == 3) ds = gw * (sub - delta[i]) * p.scale;
        Ps[(ty + 8 * i) * kPS + tx + 16 * j] = ds;
      }
    }
    __syncwarp();                              // a row's weights are written and read by the same half-warp
    weighted_rows<kD>(Ps, Ks, ty, tx, acc);
  }
  if (group > 0) {                             // the first group adds the others' sums in their order
    group_sync<128>(group);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) reinterpret_cast<uint64_t*>(Ks)[(i * (kD / 32) + c) * 128 + tid] = acc[i][c];
  }
  __syncthreads();
  if (group > 0) return;
#pragma unroll
  for (int g = 1; g < kSplit; ++g)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < kD / 32; ++c)
        acc[i][c] = ptx::add2(acc[i][c], reinterpret_cast<const uint64_t*>(Ks + g * (2 * kBK * (kD + 4) + kRT * kPS))
                                             [(i * (kD / 32) + c) * 128 + tid]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = q0 + ty + 8 * i;
    if (row >= p.Lq) continue;
    float* o = static_cast<float*>(p.dq) + ((int64_t)bh * p.Lq + row) * p.D;
#pragma unroll
    for (int c = 0; c < kD / 64; ++c) {
      float4 r;
      upk2(acc[i][2 * c], r.x, r.y);
      upk2(acc[i][2 * c + 1], r.z, r.w);
      const int d = 64 * c + 4 * tx;
      if (d < p.D) *reinterpret_cast<float4*>(o + d) = r;
    }
  }
}

// keys, values | per group: rows of q and dO, P and dS tiles of 32 rows x 64 keys; partial sums reuse the front
template <int kD> constexpr size_t dkv_smem_f32 =
    sizeof(float) * (2 * kBK * (kD + 4) + kSplit * (2 * kRT * (kD + 4) + 2 * kRT * kPS));

template <int kD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256 * kSplit) f32_bwd_dkv_kernel(AttnParams p) {
  extern __shared__ __align__(16) float sm[];
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  float* Ks = sm;
  float* Vs = Ks + kBK * (kD + 4);
  const int group = threadIdx.x >> 8, tid = threadIdx.x & 255, tx = tid & 15, ty = tid >> 4;              // ty 0 .. 15
  float* Qs = Vs + kBK * (kD + 4) + group * (2 * kRT * (kD + 4) + 2 * kRT * kPS);
  float* Gs = Qs + kRT * (kD + 4);
  float* Ps = Gs + kRT * (kD + 4);
  float* Ds = Ps + kRT * kPS;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int BH = p.B * p.H, work = blockIdx.x >> 1;                        // one CTA an SM (registers): heaviest first
  const int n = work / BH, bh = work % BH, b = bh / p.H, h = bh - b * p.H;      // early blocks are seen by the most rows
  const int prefix = p.Lk - p.Lq, key0 = n * kBK;
  const float* q = static_cast<const float*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const float* k = static_cast<const float*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const float* v = static_cast<const float*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const float* g = static_cast<const float*>(p.dO) + b * p.dos[0] + h * p.dos[1];
  load_tile<kD, kBK, 256 * kSplit>(Ks, k, p.ks[2], key0, p.Lk, p.D, threadIdx.x);
  load_tile<kD, kBK, 256 * kSplit>(Vs, v, p.vs[2], key0, p.Lk, p.D, threadIdx.x);
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  // thread: keys 4 ty .. 4 ty + 3, features 4 tx + 64 c
  uint64_t dv[4][kD / 32], dk[4][kD / 32];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < kD / 32; ++c) dv[i][c] = dk[i][c] = 0ull;
  const int t_first = max(0, key0 - prefix) / kRT, n_tiles = (p.Lq + kRT - 1) / kRT;
  for (int t = t_first + rank + 2 * group; t < n_tiles; t += 2 * kSplit) {
    const int q0 = t * kRT;
    group_sync<256>(group);
    load_tile<kD, kRT, 256>(Qs, q, p.qs[2], q0, p.Lq, p.D, tid);
    load_tile<kD, kRT, 256>(Gs, g, p.dos[2], q0, p.Lq, p.D, tid);
    cp_commit();
    float M[2], Linv[2], delta[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = q0 + ty + 16 * i;
      const int64_t gr = (int64_t)bh * p.Lq + row;
      const bool ok = row < p.Lq;
      M[i] = ok ? p.M[gr] : 0.f;
      Linv[i] = ok ? 1.f / p.L[gr] : 0.f;
      delta[i] = ok ? p.delta[gr] : 0.f;
    }
    cp_wait<0>();
    group_sync<256>(group);
    float s[2][4], dp[2][4];
    dots<kD, 2>(Qs, 16, Ks, ty, tx, s);
    dots<kD, 2>(Gs, 16, Vs, ty, tx, dp);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int pos = prefix + q0 + ty + 16 * i, own = pos >> 6, last = last_key(n, own, pos);
      const bool grouped = n < own;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] *= p.scale;
        if (tx + 16 * j <= last) mx = fmaxf(mx, s[i][j]);
      }
      mx = max16(mx);
      const float lm = __shfl_sync(0xffffffffu, s[i][3], (threadIdx.x & 16) | 15);
      const float shift = grouped ? mx : M[i];
      float den = 0.f, nD = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        s[i][j] = tx + 16 * j <= last ? expf(s[i][j] - shift) : 0.f;
        den += s[i][j];
        nD = fmaf(s[i][j], dp[i][j], nD);
      }
      den = sum16(den);
      nD = sum16(nD);
      const float gw = grouped ? expf(lm - M[i]) * Linv[i] : 0.f;
      const float sub = grouped ? nD / den : delta[i];
      const float w = grouped ? gw / den : Linv[i];
      const int r = (ty + 16 * i) * kPS;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float pj = s[i][j] * w;
        float ds = pj * (dp[i][j] - sub) * p.scale;
        if (grouped && tx == 15 && j == 3) ds = gw * (sub - delta[i]) * p.scale;
        Ps[r + tx + 16 * j] = pj;
        Ds[r + tx + 16 * j] = ds;
      }
    }
    group_sync<256>(group);
#pragma unroll 2
    for (int r = 0; r < kRT; ++r) {
      const float4 pw = *reinterpret_cast<const float4*>(Ps + r * kPS + 4 * ty), dw = *reinterpret_cast<const float4*>(Ds + r * kPS + 4 * ty);
      const float pf[4] = {pw.x, pw.y, pw.z, pw.w}, df[4] = {dw.x, dw.y, dw.z, dw.w};
#pragma unroll
      for (int c = 0; c < kD / 64; ++c) {
        const F4 gv = ld4(Gs + r * (kD + 4) + 64 * c + 4 * tx), qv = ld4(Qs + r * (kD + 4) + 64 * c + 4 * tx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t pp = pk2(pf[i], pf[i]), dd = pk2(df[i], df[i]);
          dv[i][2 * c] = fma2(pp, gv.a, dv[i][2 * c]);
          dv[i][2 * c + 1] = fma2(pp, gv.b, dv[i][2 * c + 1]);
          dk[i][2 * c] = fma2(dd, qv.a, dk[i][2 * c]);
          dk[i][2 * c + 1] = fma2(dd, qv.b, dk[i][2 * c + 1]);
        }
      }
    }
  }
  // the first group adds the others' sums in their order
#pragma unroll
  for (int g1 = 1; g1 < kSplit; ++g1) {
    __syncthreads();
    uint64_t* part = reinterpret_cast<uint64_t*>(sm);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) {
        const int at = (i * (kD / 32) + c) * 512 + tid;
        if (group == g1) {
          part[at] = dv[i][c];
          part[at + 256] = dk[i][c];
        }
      }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < kD / 32; ++c) {
        const int at = (i * (kD / 32) + c) * 512 + tid;
        if (group == 0) {
          dv[i][c] = ptx::add2(dv[i][c], part[at]);
          dk[i][c] = ptx::add2(dk[i][c], part[at + 256]);
        }
      }
  }
  // the first CTA finishes dV, the second dK: each leaves the other's part in its own shared memory
  __syncthreads();
  float* mine = sm;                              // [64][kD]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < kD / 64; ++c) {
      if (group) break;
      F4 x;
      x.a = rank == 0 ? dk[i][2 * c] : dv[i][2 * c];
      x.b = rank == 0 ? dk[i][2 * c + 1] : dv[i][2 * c + 1];
      *reinterpret_cast<F4*>(mine + (4 * ty + i) * kD + 64 * c + 4 * tx) = x;
    }
  cluster.sync();
  const float* theirs = cluster.map_shared_rank(sm, rank ^ 1);
  float* out = static_cast<float*>(rank == 0 ? p.dv : p.dk) + ((int64_t)bh * p.Lk + key0) * p.D;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < kD / 64; ++c) {
      if (group) break;
      const int key = 4 * ty + i, d = 64 * c + 4 * tx;
      const float4 y = *reinterpret_cast<const float4*>(theirs + key * kD + d);
      float4 x;
      upk2(rank == 0 ? dv[i][2 * c] : dk[i][2 * c], x.x, x.y);
      upk2(rank == 0 ? dv[i][2 * c + 1] : dk[i][2 * c + 1], x.z, x.w);
      if (key0 + key < p.Lk && d < p.D)          // even tiles' sum + odd tiles' sum in both CTAs
        *reinterpret_cast<float4*>(out + (int64_t)key * p.D + d) = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
    }
  cluster.sync();                                // the other CTA may still be reading
}

bool vec_ok(const void* ptr, const int64_t st[3]) {
  return ((uintptr_t)ptr & 15) == 0 && st[0] % 4 == 0 && st[1] % 4 == 0 && st[2] % 4 == 0;
}
bool f32_operands_ok(const AttnParams& p) {
  return p.block == kBK && p.D <= 128 && p.D % 8 == 0 && vec_ok(p.q, p.qs) && vec_ok(p.k, p.ks) && vec_ok(p.v, p.vs);
}

template <int kD>
int fwd_launch(const AttnParams& p, cudaStream_t st) {
  int n_sm, rc = sm_count(&n_sm);
  if (rc != LMK_OK) return rc;
  LMK_CUDA(cudaFuncSetAttribute(f32_fwd_kernel<kD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem_f32<kD>));
  const int grid = p.B * p.H * ((p.Lq + kRT - 1) / kRT);
  LMK_CUDA(launch_overlapped(f32_fwd_kernel<kD>, dim3(grid), dim3(128 * kSplit), fwd_smem_f32<kD>, st, p, n_sm));
  return LMK_OK;
}
template <int kD>
int bwd_launch(const AttnParams& p, cudaStream_t st) {
  int n_sm, rc = sm_count(&n_sm);
  if (rc != LMK_OK) return rc;
  LMK_CUDA(cudaFuncSetAttribute(f32_bwd_dq_kernel<kD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dq_smem_f32<kD>));
  LMK_CUDA(cudaFuncSetAttribute(f32_bwd_dkv_kernel<kD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dkv_smem_f32<kD>));
  const int grid = p.B * p.H * ((p.Lq + kRT - 1) / kRT);
  LMK_CUDA(launch_overlapped(f32_bwd_dq_kernel<kD>, dim3(grid), dim3(128 * kSplit), dq_smem_f32<kD>, st, p, n_sm));
  LMK_CUDA(launch_overlapped(f32_bwd_dkv_kernel<kD>, dim3(2 * p.B * p.H * ((p.Lk + kBK - 1) / kBK)), dim3(256 * kSplit), dkv_smem_f32<kD>, st, p));
  return LMK_OK;
}

}  // namespace

// 1: launched, 0: not a problem for these kernels, < 0: error
int attn_f32_fwd(const AttnParams& p, cudaStream_t st) {
  if (!f32_operands_ok(p) || ((uintptr_t)p.o & 15)) return 0;
  const int rc = p.D <= 64 ? fwd_launch<64>(p, st) : fwd_launch<128>(p, st);
  return rc == LMK_OK ? 1 : rc;
}
int attn_f32_bwd(const AttnParams& p, cudaStream_t st) {
  if (!f32_operands_ok(p) || !vec_ok(p.dO, p.dos) || (((uintptr_t)p.dq | (uintptr_t)p.dk | (uintptr_t)p.dv) & 15)) return 0;
  const int rc = p.D <= 64 ? bwd_launch<64>(p, st) : bwd_launch<128>(p, st);
  return rc == LMK_OK ? 1 : rc;
}

}  // namespace lmk
