// Token generation behind a landmark block cache, one launch per layer (16-bit types, head dim 128):
// rotary of the new tokens' queries and keys, landmark scores, the top-k selection, attention over the selected blocks, the
// unfinished tail block and the new tokens themselves, and the append of the new keys / values to the cache.
// Reference: the cache branch of LlamaAttention.forward for short inputs (llama/llama_mem.py:318-430, 447-474).
//
// What bounds it: nothing but latency.  One token against 1024 blocks of 32 reads 11 MB (1.7 us at the HBM peak) and
// needs 11 MFLOP, so the design is about how much of that is in flight at once and how few dependent steps there are:
//   * a cluster of CL CTAs works on one (token, head): CL * 16 warps score the landmarks (8 lanes a row, 16 rows in
//     flight a warp, requested together with the query and the tables), every warp keeps its own k best and the CL * 16 * k
//     candidates go to the CTAs that need them through distributed shared memory;
//   * a candidate is one word, the 16-bit score made sortable above the inverted block number, so a maximum over a warp
//     is one reduction instruction and ties go to the lower block;
//   * selected blocks, tail and new tokens are cut into items of 16 key rows, one warp each (values requested before the
//     logits are computed); an item leaves (max, sum, unnormalised value sum) and the landmark's logit in the first CTA's
//     shared memory, which merges the <= 64 items.  Up to 16 items are all done by the first CTA's warps: the others
//     finish after the selection and there is one cluster barrier less.
// B1 H32, 32768 cached tokens (blocks of 32, tail 17, top 4): 60 launches, 190 us -> one of 15.4 us (pairs of floats and
// indices reduced by shuffles, eight warps a CTA, items over the cluster) -> 10.6 us.
#include <cooperative_groups.h>
#include <type_traits>
#include "common.cuh"
#include "mma16.cuh"
#include "sm100_ptx.cuh"

namespace lmk {
namespace {

namespace cg = cooperative_groups;

constexpr int kDecD = 128, kDecHalf = 64;
constexpr int kDecWarps = 16;
constexpr int kDecMaxItems = 64;
constexpr int kDecMaxK = 32;
constexpr float kL2e = 1.4426950408889634f;

struct DecParams {
  const void *q, *k_new, *v_new;
  int64_t qs[3], ks[3], vs[3];            // element strides {batch, head, row}
  void *k_cache, *v_cache;
  int64_t kcs[3], vcs[3];
  int len;                                // tokens in the cache
  int append;                             // write k_new / v_new behind them
  int block, top_k, n_blocks;
  const void *cos_t, *sin_t;
  int n_pos;
  void* out;                              // [B, H, T, 128] dense
  int H, T;
  float scale;
};

struct V4 { uint32_t w[4]; };
__device__ __forceinline__ V4 ldv(const void* p) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  return {{v.x, v.y, v.z, v.w}};
}

// rotate_half on the vector pair (lo, hi) = features [d0, d0+8) and [d0+64, d0+72): x * cos + rotate_half(x) * sin with the
// three roundings of the tensor formulation
template <typename T>
__device__ __forceinline__ void rotate(V4& lo, V4& hi, const V4& cl, const V4& ch, const V4& sl, const V4& sh) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const uint32_t l = lo.w[u], h = hi.w[u];
    lo.w[u] = Pair16<T>::add(Pair16<T>::mul(l, cl.w[u]), Pair16<T>::mul(h ^ 0x80008000u, sl.w[u]));
    hi.w[u] = Pair16<T>::add(Pair16<T>::mul(h, ch.w[u]), Pair16<T>::mul(l, sh.w[u]));
  }
}
template <typename T>
__device__ __forceinline__ float dot_pair(const float (&q)[16], const V4& lo, const V4& hi) {
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float2 x = Pair16<T>::f32(lo.w[u]), y = Pair16<T>::f32(hi.w[u]);
    a = fmaf(q[2 * u], x.x, a);
    b = fmaf(q[2 * u + 1], x.y, b);
    a = fmaf(q[8 + 2 * u], y.x, a);
    b = fmaf(q[8 + 2 * u + 1], y.y, b);
  }
  return a + b;
}
// Score (already rounded to the 16-bit type) and block as one word: larger score, then lower block; 0 is below all of them.
template <typename T>
__device__ __forceinline__ uint32_t cand_key(float score, int n) {
  const T t = from_f32<T>(score);
  uint32_t bits = *reinterpret_cast<const uint16_t*>(&t);
  if (bits == 0x8000u) bits = 0u;                                        // -0 counts as +0
  return ((bits ^ (bits & 0x8000u ? 0xffffu : 0x8000u)) << 16) | (0xffffu - (uint32_t)n);
}
__device__ __forceinline__ int cand_block(uint32_t key) { return 0xffff - (int)(key & 0xffffu); }

// dynamic shared memory, in words: items (m, s, landmark logit, coefficient, values) | picks | candidates | this CTA's keys
__host__ __device__ constexpr int dec_slice(int n, int cl) {             // landmarks of a CTA: four a step and warp
  return ((n + cl - 1) / cl + 4 * kDecWarps - 1) / (4 * kDecWarps) * (4 * kDecWarps);
}
__host__ __device__ constexpr size_t dec_smem(int n, int k, int cl) {
  return sizeof(float) * (kDecMaxItems * (4 + kDecD) + kDecMaxK + (size_t)cl * kDecWarps * k + dec_slice(n, cl));
}

template <typename T, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(kDecWarps * 32) decode_attend_kernel(DecParams p) {
  extern __shared__ __align__(16) float dec_smem_buf[];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  cluster.barrier_arrive();                       // completed by barrier_wait() before the first remote write
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const int t = blockIdx.x / CL, bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K = p.top_k, N = p.n_blocks, blk = p.block;
  float* it_m = dec_smem_buf;
  float* it_s = it_m + kDecMaxItems;
  float* it_lm = it_s + kDecMaxItems;
  float* it_c = it_lm + kDecMaxItems;
  float* it_o = it_c + kDecMaxItems;                               // [item][128]
  int* sel = reinterpret_cast<int*>(it_o + kDecMaxItems * kDecD);
  uint32_t* cand = reinterpret_cast<uint32_t*>(sel + kDecMaxK);    // [CL * 16 * K]
  uint32_t* keys = cand + CL * kDecWarps * K;

  const T* cos_t = static_cast<const T*>(p.cos_t);
  const T* sin_t = static_cast<const T*>(p.sin_t);
  const int full = N * blk, inc = p.len - full;
  auto clamp_pos = [&](int x) { return (int64_t)max(0, min(x, p.n_pos - 1)) * kDecD; };
  const int pos_base = full - (K + 1) * blk;

  const int nch = (blk + 15) / 16, n_sel = K * nch;
  const int n_loc_rows = inc + t + 1 - ((p.len + t) % blk == blk - 1 ? 1 : 0);     // a landmark does not see its own key
  const int n_items = n_sel + (n_loc_rows + 15) / 16;
  const bool solo = n_items <= kDecWarps;                          // all items in the first CTA

  // ---- the query, rotated at its position; a warp of the last CTA also stores the new key and value
  if (p.append && rank == CL - 1 && warp == 1) {
    const int c = (lane & 15) * 8;
    const bool key = lane < 16;
    const T* src = key ? static_cast<const T*>(p.k_new) + b * p.ks[0] + h * p.ks[1] + t * p.ks[2]
                       : static_cast<const T*>(p.v_new) + b * p.vs[0] + h * p.vs[1] + t * p.vs[2];
    T* dst = key ? static_cast<T*>(p.k_cache) + b * p.kcs[0] + h * p.kcs[1] + (int64_t)(p.len + t) * p.kcs[2]
                 : static_cast<T*>(p.v_cache) + b * p.vcs[0] + h * p.vcs[1] + (int64_t)(p.len + t) * p.vcs[2];
    *reinterpret_cast<uint4*>(dst + c) = *reinterpret_cast<const uint4*>(src + c);
  }
  const T* kc = static_cast<const T*>(p.k_cache) + b * p.kcs[0] + h * p.kcs[1];
  const T* vc = static_cast<const T*>(p.v_cache) + b * p.vcs[0] + h * p.vcs[1];
  const int sub = lane & 7, grp = lane >> 3, d0 = sub * 8;

  // ---- landmark scores of this CTA's slice: 8 lanes a row; every block but the newest K shares slot 0 and its tables
  const int per = dec_slice(N, CL), n0 = rank * per, n1 = min(N, n0 + per);
  const int steps = per / (4 * kDecWarps);
  constexpr int kFly = 4;                                         // steps whose rows are requested together
  V4 lo[kFly], hi[kFly];
  auto request = [&](int st0) {
#pragma unroll
    for (int u = 0; u < kFly; ++u) {
      const int n = n0 + 4 * kDecWarps * (st0 + u) + 4 * warp + grp;
      if (st0 + u < steps && n < n1) {
        const T* row = kc + ((int64_t)n * blk + blk - 1) * p.kcs[2] + d0;
        lo[u] = ldv(row);
        hi[u] = ldv(row + kDecHalf);
      } else {
        lo[u] = hi[u] = {{0u, 0u, 0u, 0u}};
      }
    }
  };
  request(0);
  const int64_t po0 = clamp_pos(pos_base + blk - 1) + d0;
  const V4 cl0 = ldv(cos_t + po0), ch0 = ldv(cos_t + po0 + kDecHalf), sl0 = ldv(sin_t + po0), sh0 = ldv(sin_t + po0 + kDecHalf);
  float q[16];
  {
    const T* qp = static_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1] + t * p.qs[2] + d0;
    const int64_t po = clamp_pos(p.len + t) + d0;
    V4 ql = ldv(qp), qh = ldv(qp + kDecHalf);
    rotate<T>(ql, qh, ldv(cos_t + po), ldv(cos_t + po + kDecHalf), ldv(sin_t + po), ldv(sin_t + po + kDecHalf));
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float2 x = Pair16<T>::f32(ql.w[u]), y = Pair16<T>::f32(qh.w[u]);
      q[2 * u] = x.x;
      q[2 * u + 1] = x.y;
      q[8 + 2 * u] = y.x;
      q[8 + 2 * u + 1] = y.y;
    }
  }
  uint32_t* my_keys = keys + warp * 4 * steps;
  for (int st0 = 0; st0 < steps; st0 += kFly) {
    if (st0) request(st0);
#pragma unroll
    for (int u = 0; u < kFly; ++u) {
      if (st0 + u >= steps) break;
      const int n = n0 + 4 * kDecWarps * (st0 + u) + 4 * warp + grp;
      if (n < N - K || n >= n1) {
        rotate<T>(lo[u], hi[u], cl0, ch0, sl0, sh0);
      } else {
        const int64_t po = clamp_pos(pos_base + (n - (N - K) + 1) * blk + blk - 1) + d0;
        rotate<T>(lo[u], hi[u], ldv(cos_t + po), ldv(cos_t + po + kDecHalf), ldv(sin_t + po), ldv(sin_t + po + kDecHalf));
      }
      float s = dot_pair<T>(q, lo[u], hi[u]);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      // the reference's matmul output and the scaling are each rounded to the input type; NaN ranks lowest
      s = to_f32(from_f32<T>(s)) * p.scale;
      if (sub == 0) my_keys[4 * (st0 + u) + grp] = n < n1 ? cand_key<T>(s == s ? s : -INFINITY, n) : 0u;
    }
  }
  __syncwarp();

  // ---- every warp's K best of its own rows, to every CTA of the cluster that works on items
  uint32_t won = 0;                                               // lane `it` keeps the it-th
  if (4 * steps <= 32) {
    uint32_t mine = lane < 4 * steps ? my_keys[lane] : 0u;
    for (int it = 0; it < K; ++it) {
      const uint32_t best = __reduce_max_sync(0xffffffffu, mine);
      if (mine == best) mine = 0u;
      if (lane == it) won = best;
    }
  } else {
    for (int it = 0; it < K; ++it) {
      uint32_t mine = 0u;
      for (int j = lane; j < 4 * steps; j += 32) mine = max(mine, my_keys[j]);
      const uint32_t best = __reduce_max_sync(0xffffffffu, mine);
      if (mine == best && best) {
        const int r = cand_block(best) - n0;
        my_keys[4 * (r / (4 * kDecWarps)) + (r & 3)] = 0u;
      }
      if (lane == it) won = best;
      __syncwarp();
    }
  }
  cluster.barrier_wait();
  if (lane < K) {
#pragma unroll
    for (int c = 0; c < CL; ++c)
      if (c == 0 || !solo) cluster.map_shared_rank(cand, c)[(rank * kDecWarps + warp) * K + lane] = won;
  }
  cluster.sync();
  if (solo && rank != 0) return;                                  // nothing reads this CTA's memory any more

  // ---- the final K, in ascending order of age: by every warp for itself from registers, by the first one if there are many
  const int n_cand = CL * kDecWarps * K;
  const bool few = n_cand <= 256;
  if (few || warp == 0) {
    int mine = 0x7fffffff;
    if (few) {
      uint32_t v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = lane + 32 * u < n_cand ? cand[lane + 32 * u] : 0u;
      for (int it = 0; it < K; ++it) {
        const uint32_t top = max(max(max(v[0], v[1]), max(v[2], v[3])), max(max(v[4], v[5]), max(v[6], v[7])));
        const uint32_t best = __reduce_max_sync(0xffffffffu, top);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (v[u] == best) v[u] = 0u;
        if (lane == it) mine = cand_block(best);
      }
    } else {
      for (int it = 0; it < K; ++it) {
        uint32_t top = 0u;
        for (int j = lane; j < n_cand; j += 32) top = max(top, cand[j]);
        const uint32_t best = __reduce_max_sync(0xffffffffu, top);
        if (top == best)
          for (int j = lane; j < n_cand; j += 32)
            if (cand[j] == best) cand[j] = 0u;
        if (lane == it) mine = cand_block(best);
        __syncwarp();
      }
    }
    int order = 0;
    for (int u = 0; u < K; ++u) order += __shfl_sync(0xffffffffu, mine, u) < mine ? 1 : 0;
    if (lane < K) sel[order] = mine;                              // all warps write the same
  }
  if (few) __syncwarp();
  else __syncthreads();

  // ---- items of 16 key rows: chunk c of selected block i, then chunks of the tail and the new tokens
  const float scale_log2 = p.scale * kL2e;
  float* m_out = cluster.map_shared_rank(it_m, 0);
  float* s_out = cluster.map_shared_rank(it_s, 0);
  float* lm_out = cluster.map_shared_rank(it_lm, 0);
  float* o_out = cluster.map_shared_rank(it_o, 0);
  for (int item = rank * kDecWarps + warp; item < n_items; item += CL * kDecWarps) {                // solo: rank 0, one each
    const bool selected = item < n_sel;
    const int i = selected ? item / nch : 0, c = selected ? item - i * nch : item - n_sel;
    const int nrows = min(16, (selected ? blk : n_loc_rows) - 16 * c);             // >= 1
    const T *kb, *vb;
    int pos0;
    if (selected) {
      const int s = sel[i];
      kb = kc + ((int64_t)s * blk + 16 * c) * p.kcs[2];
      vb = vc + ((int64_t)s * blk + 16 * c) * p.vcs[2];
      pos0 = pos_base + (i + (s >= N - K ? 1 : 0)) * blk + 16 * c;
    } else {
      kb = kc + (int64_t)(full + 16 * c) * p.kcs[2];
      vb = vc + (int64_t)(full + 16 * c) * p.vcs[2];
      pos0 = full + 16 * c;
    }
    auto row_of = [&](const T* cached, int64_t cs, const void* fresh, const int64_t (&fs)[3], int r) -> const T* {
      r = min(r, nrows - 1);
      if (selected || 16 * c + r < inc) return cached + (int64_t)r * cs;
      return static_cast<const T*>(fresh) + b * fs[0] + h * fs[1] + (int64_t)(16 * c + r - inc) * fs[2];
    };
    V4 vv[8];                                      // values: 16 lanes a row, requested before the logits need them
#pragma unroll
    for (int s = 0; s < 8; ++s) vv[s] = ldv(row_of(vb, p.vcs[2], p.v_new, p.vs, 2 * s + (lane >> 4)) + (lane & 15) * 8);
    float lg[4];
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      const int r = 4 * st + grp;
      const T* row = row_of(kb, p.kcs[2], p.k_new, p.ks, r) + d0;
      const int64_t po = clamp_pos(pos0 + min(r, nrows - 1)) + d0;
      V4 lo = ldv(row), hi = ldv(row + kDecHalf);
      rotate<T>(lo, hi, ldv(cos_t + po), ldv(cos_t + po + kDecHalf), ldv(sin_t + po), ldv(sin_t + po + kDecHalf));
      lg[st] = dot_pair<T>(q, lo, hi);
    }
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      lg[st] += __shfl_xor_sync(0xffffffffu, lg[st], 1);
      lg[st] += __shfl_xor_sync(0xffffffffu, lg[st], 2);
      lg[st] += __shfl_xor_sync(0xffffffffu, lg[st], 4);
      lg[st] *= scale_log2;
    }
    const int lm_row = selected ? blk - 1 - 16 * c : 99;          // the block's landmark, if this chunk holds it
    float mx = -INFINITY;
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      const int r = 4 * st + grp;
      if (r == lm_row && sub == 0) lm_out[item] = lg[st];
      if (r >= nrows || r == lm_row) lg[st] = -INFINITY;
      mx = fmaxf(mx, lg[st]);
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    float sum = 0.f;
#pragma unroll
    for (int st = 0; st < 4; ++st) {
      lg[st] = mx == -INFINITY ? 0.f : exp2f(lg[st] - mx);
      sum += lg[st];
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 8);
    sum += __shfl_xor_sync(0xffffffffu, sum, 16);
    float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 8; ++s) {                 // row 2 s + (lane >> 4): probability in register s >> 1 of group (row & 3)
      const float pr = __shfl_sync(0xffffffffu, lg[s >> 1], 8 * (2 * (s & 1) + (lane >> 4)));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 x = Pair16<T>::f32(vv[s].w[u]);
        o[2 * u] = fmaf(pr, x.x, o[2 * u]);
        o[2 * u + 1] = fmaf(pr, x.y, o[2 * u + 1]);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) o[u] += __shfl_xor_sync(0xffffffffu, o[u], 16);
    if (lane < 16) {
      float4* dst = reinterpret_cast<float4*>(o_out + item * kDecD + lane * 8);
      dst[0] = make_float4(o[0], o[1], o[2], o[3]);
      dst[1] = make_float4(o[4], o[5], o[6], o[7]);
    }
    if (lane == 0) {
      m_out[item] = mx;
      s_out[item] = sum;
    }
  }
  if (solo) {
    __syncthreads();
  } else {
    cluster.sync();
    if (rank != 0) return;
  }

  // ---- merge: softmax inside each block over its chunks, then the outer softmax over landmarks and local keys
  if (warp == 0) {
    float M = -INFINITY, S = 0.f, x = -INFINITY;
    if (lane < K) {
      for (int c = 0; c < nch; ++c) M = fmaxf(M, it_m[lane * nch + c]);
      for (int c = 0; c < nch; ++c) S += M == -INFINITY ? 0.f : it_s[lane * nch + c] * exp2f(it_m[lane * nch + c] - M);
      x = it_lm[lane * nch + nch - 1];
    }
    const bool loc = lane < n_items - n_sel;
    const float lm = loc ? it_m[n_sel + lane] : -INFINITY, ls = loc ? it_s[n_sel + lane] : 0.f;
    const float top = warp_max(fmaxf(x, lm));
    const float wx = top == -INFINITY || x == -INFINITY ? 0.f : exp2f(x - top);
    const float wl = top == -INFINITY || lm == -INFINITY ? 0.f : exp2f(lm - top);
    const float Z = warp_sum(wx + wl * ls);
    const float rz = Z > 0.f ? 1.f / Z : 0.f;
    if (lane < K)
      for (int c = 0; c < nch; ++c)
        it_c[lane * nch + c] = S > 0.f ? wx * rz * exp2f(it_m[lane * nch + c] - M) / S : 0.f;
    if (loc) it_c[n_sel + lane] = wl * rz;
  }
  __syncthreads();
  if (tid < kDecD) {
    float a = 0.f, b2 = 0.f;
    int e = 0;
    for (; e + 1 < n_items; e += 2) {
      a = fmaf(it_c[e], it_o[e * kDecD + tid], a);
      b2 = fmaf(it_c[e + 1], it_o[(e + 1) * kDecD + tid], b2);
    }
    if (e < n_items) a = fmaf(it_c[e], it_o[e * kDecD + tid], a);
    static_cast<T*>(p.out)[((int64_t)bh * p.T + t) * kDecD + tid] = from_f32<T>(a + b2);
  }
}

template <typename T, int CL>
int dec_launch(const DecParams& p, int BH, cudaStream_t st) {
  const size_t smem = dec_smem(p.n_blocks, p.top_k, CL);
  if (smem > 48 * 1024)
    LMK_CUDA(cudaFuncSetAttribute(decode_attend_kernel<T, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  LMK_CUDA(launch_overlapped(decode_attend_kernel<T, CL>, dim3(CL * p.T, BH), dim3(kDecWarps * 32), smem, st, p));
  return LMK_OK;
}

// The merge holds one item per 16 key rows, and the local items must fit one lane each.
bool dec_supported(int D, int block, int top_k, int n_blocks, int len, int T, int dtype) {
  const int nch = (block + 15) / 16;
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D == kDecD && block >= 2 && top_k >= 1 && top_k <= kDecMaxK &&
         n_blocks >= 1 && n_blocks <= 49152 && top_k <= n_blocks && T >= 1 && T <= 4096 && len >= n_blocks * block &&
         len - n_blocks * block + T <= block && nch <= 32 && (top_k + 1) * nch <= kDecMaxItems;
}

}  // namespace
}  // namespace lmk

using namespace lmk;

extern "C" int lmk_decode_supported(int D, int block, int top_k, int len, int T, int dtype) {
  return block >= 2 && dec_supported(D, block, top_k, len / block, len, T, dtype) ? 1 : 0;
}

extern "C" int lmk_decode_attend(const void* q, const void* k_new, const void* v_new, const int64_t q_strides[3],
                                 const int64_t k_strides[3], const int64_t v_strides[3], void* k_cache, void* v_cache,
                                 const int64_t k_cache_strides[3], const int64_t v_cache_strides[3], int len, int append,
                                 int block, int top_k, const void* cos_table, const void* sin_table, int n_pos, void* out,
                                 int B, int H, int T, int D, float sm_scale, int dtype, void* stream) {
  LMK_CHECK_ARG(q && k_new && v_new && k_cache && v_cache && cos_table && sin_table && out, "decode_attend: null pointer");
  LMK_CHECK_ARG(q_strides && k_strides && v_strides && k_cache_strides && v_cache_strides, "decode_attend: strides missing");
  LMK_CHECK_ARG(B >= 1 && H >= 1 && n_pos >= 1 && block >= 2 && (int64_t)B * H <= 65535, "decode_attend: bad sizes");
  if (!dec_supported(D, block, top_k, len / block, len, T, dtype))
    return fail(LMK_ERR_UNSUPPORTED, "decode_attend needs a 16-bit type, D=128, at least one whole block, the new tokens inside "
                "the unfinished block and (top_k + 1) * ceil(block / 16) <= %d (got dtype=%d D=%d block=%d top_k=%d len=%d T=%d)",
                kDecMaxItems, dtype, D, block, top_k, len, T);
  const uintptr_t align = (uintptr_t)q | (uintptr_t)k_new | (uintptr_t)v_new | (uintptr_t)k_cache | (uintptr_t)v_cache |
                          (uintptr_t)cos_table | (uintptr_t)sin_table;
  LMK_CHECK_ARG((align & 15) == 0, "decode_attend: pointers must be 16-byte aligned");
  DecParams p{};
  for (int i = 0; i < 3; ++i) {
    LMK_CHECK_ARG(q_strides[i] % 8 == 0 && k_strides[i] % 8 == 0 && v_strides[i] % 8 == 0 && k_cache_strides[i] % 8 == 0 &&
                  v_cache_strides[i] % 8 == 0, "decode_attend: strides must be multiples of 8 elements");
    p.qs[i] = q_strides[i]; p.ks[i] = k_strides[i]; p.vs[i] = v_strides[i];
    p.kcs[i] = k_cache_strides[i]; p.vcs[i] = v_cache_strides[i];
  }
  p.q = q; p.k_new = k_new; p.v_new = v_new; p.k_cache = k_cache; p.v_cache = v_cache;
  p.len = len; p.append = append; p.block = block; p.top_k = top_k; p.n_blocks = len / block;
  p.cos_t = cos_table; p.sin_t = sin_table; p.n_pos = n_pos; p.out = out; p.H = H; p.T = T; p.scale = sm_scale;
  const int BH = B * H;
  // 8 CTAs a (token, head) while that still leaves SMs free, 4 otherwise: more CTAs only shorten the scoring phase.  Measured (us, 8 / 4
  // CTAs, blocks of 32): 1024 blocks, 8 heads 9.69 / 9.81, 16 heads (the line) 12.5 / 10.0, 18 12.6 / 10.0, 32 15.8 / 10.1; 100 blocks,
  // 8 heads 9.2 / 8.5, 16 11.7 / 8.7.  Eight pay for a handful of heads and many blocks only, and by 1 %; between 10 and 18 heads
  // they cost up to 2.5 us.
  int n_sm = 0;
  const int rc = sm_count(&n_sm);
  if (rc != LMK_OK) return rc;
  const bool wide = BH * T * 8 <= n_sm;
  if (dtype == LMK_BF16)
    return wide ? dec_launch<__nv_bfloat16, 8>(p, BH, (cudaStream_t)stream) : dec_launch<__nv_bfloat16, 4>(p, BH, (cudaStream_t)stream);
  return wide ? dec_launch<__half, 8>(p, BH, (cudaStream_t)stream) : dec_launch<__half, 4>(p, BH, (cudaStream_t)stream);
}
