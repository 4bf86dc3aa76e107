// lm_benchmark's block cache at evaluation time (16-bit types, head dim 128): block selection, the retrieved prefix, and the
// prefix part of att @ v.
// Reference: MemLMCacheStorage.retrieve_for_query (lm_benchmark/models/caches/mem_cache.py:41-109) and the cache branch of
// CausalSelfAttention.forward (lm_benchmark/models/landmark.py:236-243).
//
//   block_select   scores of 64 tokens against all (<= 128) landmark keys as mma.sync tiles, softmax over the blocks and the
//                  top-k of every token in registers: one launch, nothing but the indices written.
//   prefix_gather  the interface returns every token's selected values as a tensor, so writing it is the floor (1.7 GB at B16
//                  H8 T255 top 4 of blocks of 51).  One CTA per (block, head) instead of one per (token, pick): the block's
//                  keys and values are read once into shared memory, the tokens that picked it are found by a scan of the
//                  indices, each gets the values by one bulk store (13 KB, asynchronous) and its logits from mma.sync tiles of
//                  16 tokens that hold the block at the same rank (the rank sets the rotation).  No rotated copies of the keys
//                  are written and nothing is concatenated afterwards: the unfinished tail is one more "block".
//   prefix_pv      probabilities times the retrieved values, added to the chunk's own part: HBM-bound, one read of the values.
#include "common.cuh"
#include "mma16.cuh"

namespace lmk {
namespace {

constexpr int kBD = 128, kBH = 64;
constexpr int kPad = 160;                 // 16-bit elements of a shared row: the 16-byte loads of an mma fragment hit all banks once
constexpr int kSelMaxN = 128;
constexpr int kGatherMaxBlk = 128;

// one 16-byte vector of the low half (features d0..d0+7) and its partner of the high half, rotated at table row `pos`
template <typename T>
__device__ __forceinline__ void rotate_pair(uint4& lo, uint4& hi, const T* cos_t, const T* sin_t, int64_t po, int rotary) {
  if (rotary == LMK_ROTARY_NONE) return;
  const uint4 cl = *reinterpret_cast<const uint4*>(cos_t + po), ch = *reinterpret_cast<const uint4*>(cos_t + po + kBH);
  const uint4 sl = *reinterpret_cast<const uint4*>(sin_t + po), sh = *reinterpret_cast<const uint4*>(sin_t + po + kBH);
  uint32_t *l = reinterpret_cast<uint32_t*>(&lo), *h = reinterpret_cast<uint32_t*>(&hi);
  const uint32_t *c0 = reinterpret_cast<const uint32_t*>(&cl), *c1 = reinterpret_cast<const uint32_t*>(&ch);
  const uint32_t *s0 = reinterpret_cast<const uint32_t*>(&sl), *s1 = reinterpret_cast<const uint32_t*>(&sh);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    uint32_t pl, ph;
    if (rotary == LMK_ROTARY_HALF) {
      pl = h[u] ^ 0x80008000u;
      ph = l[u];
    } else {
      pl = __byte_perm(l[u], l[u], 0x1032) ^ 0x00008000u;
      ph = __byte_perm(h[u], h[u], 0x1032) ^ 0x00008000u;
    }
    const uint32_t a = Pair16<T>::add(Pair16<T>::mul(l[u], c0[u]), Pair16<T>::mul(pl, s0[u]));
    h[u] = Pair16<T>::add(Pair16<T>::mul(h[u], c1[u]), Pair16<T>::mul(ph, s1[u]));
    l[u] = a;
  }
}
__device__ __forceinline__ int age_of(int phys, int ring_start, int n) {
  const int l = phys - ring_start;
  return l < 0 ? l + n : l;
}

// ------------------------------------------------------------------------------------------------ selection
// NB groups of 8 landmarks.  128 threads = 64 tokens; q is dense [B*H, T, 128].
template <typename T, int NB>
__global__ void __launch_bounds__(128) block_select_kernel(const T* __restrict__ q, const T* __restrict__ lm, lmk_cache_desc d,
                                                           const T* __restrict__ cos_t, const T* __restrict__ sin_t, int n_pos,
                                                           int rotary, float* __restrict__ probs, int32_t* __restrict__ idx,
                                                           int H, int Tq, float scale) {
  extern __shared__ __align__(16) uint8_t sel_buf[];
  T* ks = reinterpret_cast<T*>(sel_buf);                           // [NB * 8][kPad], rotated landmark keys
  const int bh = blockIdx.y, b = bh / H, h = bh - b * H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int N = d.n_blocks, K = d.top_k;
  for (int e = tid; e < NB * 8 * 8; e += 128) {
    const int n = e >> 3, d0 = (e & 7) * 8;
    uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
    if (n < N) {
      const T* row = lm + b * d.stride_b + h * d.stride_h + (int64_t)n * d.stride_block + (int64_t)(d.block - 1) * d.stride_row;
      lo = *reinterpret_cast<const uint4*>(row + d0);
      hi = *reinterpret_cast<const uint4*>(row + d0 + kBH);
      const int age = age_of(n, d.ring_start, N), slot = age >= N - K ? age - (N - K) + 1 : 0;
      const int pos = max(0, min(d.pos_base + slot * d.block + d.block - 1, n_pos - 1));
      rotate_pair<T>(lo, hi, cos_t, sin_t, (int64_t)pos * kBD + d0, rotary);
    }
    *reinterpret_cast<uint4*>(ks + n * kPad + d0) = lo;
    *reinterpret_cast<uint4*>(ks + n * kPad + d0 + kBH) = hi;
  }
  const int t0 = blockIdx.x * 64 + warp * 16;
  uint4 a[4], a8[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const T* r0 = q + ((int64_t)bh * Tq + min(t0 + g, Tq - 1)) * kBD + 32 * c + 8 * t4;
    const T* r8 = q + ((int64_t)bh * Tq + min(t0 + g + 8, Tq - 1)) * kBD + 32 * c + 8 * t4;
    a[c] = *reinterpret_cast<const uint4*>(r0);
    a8[c] = *reinterpret_cast<const uint4*>(r8);
  }
  __syncthreads();
  if (t0 >= Tq) return;
  float acc[NB][4];
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
      mma_chunk<T>(acc[nb], a[c], a8[c], *reinterpret_cast<const uint4*>(ks + (nb * 8 + g) * kPad + 32 * c + 8 * t4));
  }
#pragma unroll
  for (int half = 0; half < 2; ++half) {                           // rows t0 + g and t0 + g + 8: 2 NB columns a lane
    const int t = t0 + g + 8 * half;
    float mx = -INFINITY;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = nb * 8 + 2 * t4 + e;
        float& v = acc[nb][2 * half + e];
        // the reference's matmul output and the scaling are each rounded to the input type
        v = n < N ? rnd<T>(rnd<T>(v) * scale) : -INFINITY;
        mx = fmaxf(mx, v);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    float sum = 0.f;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float& v = acc[nb][2 * half + e];
        v = nb * 8 + 2 * t4 + e < N ? expf(v - mx) : 0.f;
        sum += v;
      }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = nb * 8 + 2 * t4 + e;
        float& v = acc[nb][2 * half + e];
        v = rnd<T>(v / sum);
        if (probs != nullptr && n < N && t < Tq) probs[((int64_t)bh * Tq + t) * N + n] = v;
        v = v == v ? v : -INFINITY;                                // NaN ranks lowest
      }
    if (idx == nullptr) continue;
    uint32_t taken = 0;                                            // bit 2 nb + e
    int picks[8], ages[8];
    for (int it = 0; it < K; ++it) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int n = nb * 8 + 2 * t4 + e;
          const float v = acc[nb][2 * half + e];
          if (n < N && !((taken >> (2 * nb + e)) & 1u) && (bi == 0x7fffffff || v > best)) {    // ascending n: ties keep the lower
            best = v;
            bi = n;
          }
        }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) {
          best = ov;
          bi = oi;
        }
      }
      if (((bi & 7) >> 1) == t4) taken |= 1u << (2 * (bi >> 3) + (bi & 1));
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (u == it) {
          picks[u] = bi;
          ages[u] = age_of(bi, d.ring_start, N);
        }
    }
    if (t < Tq) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (u >= K || (u & 3) != t4) continue;
        int rank = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) rank += (w < K && ages[w] < ages[u]) ? 1 : 0;
        idx[((int64_t)bh * Tq + t) * K + rank] = picks[u];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ gather
struct PrefixParams {
  const void *q;                          // dense [B*H, T, 128]
  const void *k_cache, *v_cache;
  lmk_cache_desc kd, vd;
  const int32_t* idx;                     // pick i of token t of head h of batch row b: idx[b is[0] + h is[1] + t is[2] + i]
  int64_t is[3];
  const void *cos_t, *sin_t;
  int n_pos, rotary;
  const void *tail_k, *tail_v;            // rows of the unfinished block
  int64_t ts[3];                          // their element strides {batch, head, row}
  int tail_len, tail_pos;
  void *att, *v_out;                      // [B*H, T, P], [B*H, T, P, 128],  P = top_k * block + tail_len
  int H, T;
  float scale;
};

constexpr int kGatherThreads = 256;
// keys as read | keys rotated for one rank | values (dense, the source of the bulk stores) | token list | rank counters
__host__ __device__ constexpr size_t gather_smem(int rows, int T) {
  const int r8 = (rows + 7) & ~7;
  return (size_t)r8 * kPad * 2 * 2 + (size_t)rows * kBD * 2 + (size_t)T * 4 + 2 * 36 * 4;
}

template <typename T>
__global__ void __launch_bounds__(kGatherThreads) prefix_gather_kernel(PrefixParams p) {
  extern __shared__ __align__(128) uint8_t gat_buf[];
  const int n = blockIdx.x, bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int N = p.kd.n_blocks, K = p.kd.top_k, blk = p.kd.block;
  const bool tail = n == N;
  const int rows = tail ? p.tail_len : blk, r8 = (rows + 7) & ~7;
  const int P = K * blk + p.tail_len;
  T* vsm = reinterpret_cast<T*>(gat_buf);                               // [rows][128]
  T* kraw = vsm + rows * kBD;                                           // [r8][kPad]
  T* krot = kraw + r8 * kPad;
  int* list = reinterpret_cast<int*>(krot + r8 * kPad);                 // tokens, grouped by rank
  int* count = list + p.T;                                              // [33]
  int* start = count + 36;
  const int n_ranks = tail ? 1 : K;

  // ---- which tokens picked this block, and at which rank
  if (tid < 33) count[tid] = 0;
  __syncthreads();
  const int32_t* idx = p.idx + b * p.is[0] + h * p.is[1];
  const int picks = p.T * K;
  if (tail) {
    for (int t = tid; t < p.T; t += kGatherThreads) list[t] = t;
    if (tid == 0) count[0] = p.T;
  } else {
    for (int e = tid; e < picks; e += kGatherThreads) {
      const int t = e / K, i = e - t * K;
      if (idx[t * p.is[2] + i] == n) atomicAdd(&count[i], 1);
    }
  }
  __syncthreads();
  if (tid == 0) {
    int run = 0;
    for (int i = 0; i < n_ranks; ++i) {
      start[i] = run;
      run += count[i];
    }
    start[n_ranks] = run;
  }
  __syncthreads();
  const int total = start[n_ranks];
  if (total == 0) return;                                               // uniform
  if (!tail) {
    if (tid < 33) count[tid] = 0;
    __syncthreads();
    for (int e = tid; e < picks; e += kGatherThreads) {                 // order inside a rank does not matter
      const int t = e / K, i = e - t * K;
      if (idx[t * p.is[2] + i] == n) list[start[i] + atomicAdd(&count[i], 1)] = t;
    }
  }

  // ---- the block's keys and values, once
  const T* ksrc = tail ? static_cast<const T*>(p.tail_k) + b * p.ts[0] + h * p.ts[1]
                       : static_cast<const T*>(p.k_cache) + b * p.kd.stride_b + h * p.kd.stride_h + (int64_t)n * p.kd.stride_block;
  const T* vsrc = tail ? static_cast<const T*>(p.tail_v) + b * p.ts[0] + h * p.ts[1]
                       : static_cast<const T*>(p.v_cache) + b * p.vd.stride_b + h * p.vd.stride_h + (int64_t)n * p.vd.stride_block;
  const int64_t krs = tail ? p.ts[2] : p.kd.stride_row, vrs = tail ? p.ts[2] : p.vd.stride_row;
  for (int e = tid; e < r8 * 16; e += kGatherThreads) {
    const int r = e >> 4, c = (e & 15) * 8;
    uint4 kv = make_uint4(0, 0, 0, 0);
    if (r < rows) {
      kv = *reinterpret_cast<const uint4*>(ksrc + r * krs + c);
      *reinterpret_cast<uint4*>(vsm + r * kBD + c) = *reinterpret_cast<const uint4*>(vsrc + r * vrs + c);
    }
    *reinterpret_cast<uint4*>(kraw + r * kPad + c) = kv;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();

  // ---- values: one bulk store per token, issued by the lanes of one warp while the others work on the logits
  if (warp == kGatherThreads / 32 - 1) {
    const uint32_t src = (uint32_t)__cvta_generic_to_shared(vsm);
    const uint32_t bytes = (uint32_t)rows * kBD * 2;
    int rank = 0;
    for (int e = lane; e < total; e += 32) {
      while (e >= start[rank + 1]) ++rank;
      T* dst = static_cast<T*>(p.v_out) + (((int64_t)bh * p.T + list[e]) * P + (tail ? K : rank) * blk) * kBD;
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }

  // ---- logits: for every rank in use the keys are rotated once, then tiles of 16 tokens x 8 keys
  const T *cos_t = static_cast<const T*>(p.cos_t), *sin_t = static_cast<const T*>(p.sin_t);
  const T* q = static_cast<const T*>(p.q) + (int64_t)bh * p.T * kBD;
  const bool recent = !tail && age_of(n, p.kd.ring_start, N) >= N - K;
  for (int rank = 0; rank < n_ranks; ++rank) {
    const int e0 = start[rank], e1 = start[rank + 1];
    if (e0 == e1) continue;                                             // uniform
    const int pos0 = tail ? p.tail_pos : p.kd.pos_base + (rank + (recent ? 1 : 0)) * blk;
    for (int e = tid; e < r8 * 8; e += kGatherThreads) {
      const int r = e >> 3, d0 = (e & 7) * 8;
      uint4 lo = *reinterpret_cast<const uint4*>(kraw + r * kPad + d0), hi = *reinterpret_cast<const uint4*>(kraw + r * kPad + d0 + kBH);
      const int pos = max(0, min(pos0 + min(r, rows - 1), p.n_pos - 1));
      rotate_pair<T>(lo, hi, cos_t, sin_t, (int64_t)pos * kBD + d0, p.rotary);
      *reinterpret_cast<uint4*>(krot + r * kPad + d0) = lo;
      *reinterpret_cast<uint4*>(krot + r * kPad + d0 + kBH) = hi;
    }
    __syncthreads();
    const int nbs = r8 / 8, tiles = (e1 - e0 + 15) / 16;
    for (int m = 0; m < tiles; ++m) {
      const int ea = e0 + 16 * m + g, eb = ea + 8;
      const int ta = list[min(ea, e1 - 1)], tb = list[min(eb, e1 - 1)];
      uint4 a[4], a8[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        a[c] = *reinterpret_cast<const uint4*>(q + (int64_t)ta * kBD + 32 * c + 8 * t4);
        a8[c] = *reinterpret_cast<const uint4*>(q + (int64_t)tb * kBD + 32 * c + 8 * t4);
      }
      for (int nb = warp; nb < nbs; nb += kGatherThreads / 32) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c)
          mma_chunk<T>(acc, a[c], a8[c], *reinterpret_cast<const uint4*>(krot + (nb * 8 + g) * kPad + 32 * c + 8 * t4));
        const int key = nb * 8 + 2 * t4, col = (tail ? K : rank) * blk + key;
        T* oa = static_cast<T*>(p.att) + ((int64_t)bh * p.T + ta) * P + col;
        T* ob = static_cast<T*>(p.att) + ((int64_t)bh * p.T + tb) * P + col;
#pragma unroll
        for (int e = 0; e < 2; ++e) {          // the matmul and the scaling are each rounded to the 16-bit type
          if (key + e >= rows) continue;
          if (ea < e1) oa[e] = from_f32<T>(rnd<T>(acc[e]) * p.scale);
          if (eb < e1) ob[e] = from_f32<T>(rnd<T>(acc[2 + e]) * p.scale);
        }
      }
    }
    __syncthreads();                                                    // krot is rewritten for the next rank
  }
  if (warp == kGatherThreads / 32 - 1) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ------------------------------------------------------------------------------------------------ prefix part of att @ v
// y[b,h,t,:] += sum_j T(probs[b,h,t,j]) V[b,h,t,j,:], probabilities rounded to T as the reference casts them, fp32 sums.  One CTA
// per (t, batch*head): 16 lanes a row, 16 rows a step, four steps in flight.
template <typename T>
__global__ void __launch_bounds__(256) prefix_pv_kernel(const float* __restrict__ probs, int64_t ld, const T* __restrict__ v,
                                                        int64_t vb, int64_t vh, int64_t vt, T* __restrict__ y, int H, int Tq, int P) {
  extern __shared__ __align__(16) float pv_buf[];                       // probabilities, then partial sums [8][128]
  const int t = blockIdx.x, bh = blockIdx.y, b = bh / H, h = bh - b * H, tid = threadIdx.x;
  const float* pr = probs + ((int64_t)bh * Tq + t) * ld;
  for (int j = tid; j < P; j += 256) pv_buf[j] = rnd<T>(pr[j]);
  __syncthreads();
  const int c = (tid & 15) * 8, r0 = tid >> 4;
  const T* src = v + b * vb + h * vh + t * vt + c;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int r = r0; r < P; r += 16) {
    const uint4 w = __ldcs(reinterpret_cast<const uint4*>(src + (int64_t)r * kBD));
    const T* e = reinterpret_cast<const T*>(&w);
    const float x = pv_buf[r];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u] = fmaf(x, to_f32(e[u]), acc[u]);
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], 16);
  __syncthreads();
  if ((tid & 31) < 16)
#pragma unroll
    for (int u = 0; u < 8; ++u) pv_buf[(tid >> 5) * kBD + c + u] = acc[u];
  __syncthreads();
  if (tid < kBD) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += pv_buf[w * kBD + tid];
    T* o = y + ((int64_t)bh * Tq + t) * kBD + tid;
    *o = from_f32<T>(to_f32(*o) + rnd<T>(s));
  }
}

bool vec_aligned(const lmk_cache_desc* d) {
  return d->stride_b % 8 == 0 && d->stride_h % 8 == 0 && d->stride_block % 8 == 0 && d->stride_row % 8 == 0;
}

}  // namespace
}  // namespace lmk

using namespace lmk;

extern "C" int lmk_block_select_supported(int D, int n_blocks, int top_k, int dtype) {
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D == kBD && n_blocks >= 1 && n_blocks <= kSelMaxN && top_k >= 0 && top_k <= 8 &&
         top_k <= n_blocks ? 1 : 0;
}

extern "C" int lmk_block_select(const void* q, const void* landmark_keys, const lmk_cache_desc* desc, const void* cos_table,
                                const void* sin_table, int n_pos, int rotary, float* probs, int32_t* idx, int B, int H, int T,
                                int D, float sm_scale, int dtype, void* stream) {
  LMK_CHECK_ARG(q && landmark_keys && desc && (probs || idx), "block_select: null pointer");
  if (!lmk_block_select_supported(D, desc->n_blocks, desc->top_k, dtype) || !vec_aligned(desc))
    return fail(LMK_ERR_UNSUPPORTED, "block_select: 16-bit type, D=128, at most %d blocks, top_k <= 8", kSelMaxN);
  LMK_CHECK_ARG(rotary >= LMK_ROTARY_NONE && rotary <= LMK_ROTARY_INTERLEAVED &&
                (rotary == LMK_ROTARY_NONE || (cos_table && sin_table && n_pos >= 1)),
                "block_select: rotary tables missing");
  LMK_CHECK_ARG(B >= 1 && H >= 1 && T >= 1 && (int64_t)B * H <= 65535, "block_select: bad sizes");
  LMK_CHECK_ARG(idx == nullptr || desc->top_k >= 1, "block_select: indices asked for with top_k = 0");
  LMK_CHECK_ARG((((uintptr_t)q | (uintptr_t)landmark_keys | (uintptr_t)cos_table | (uintptr_t)sin_table) & 15) == 0,
                "block_select: pointers must be 16-byte aligned");
  const dim3 grid((T + 63) / 64, B * H);
  const int nb = (desc->n_blocks + 7) / 8;
#define LMK_SEL(TT, NB)                                                                                                   \
  block_select_kernel<TT, NB><<<grid, 128, (size_t)NB * 8 * kPad * 2, (cudaStream_t)stream>>>(                            \
      (const TT*)q, (const TT*)landmark_keys, *desc, (const TT*)cos_table, (const TT*)sin_table, n_pos, rotary, probs, idx, \
      H, T, sm_scale)
#define LMK_SEL_N(TT)                                                                             \
  do {                                                                                            \
    if (nb <= 4) LMK_SEL(TT, 4); else if (nb <= 8) LMK_SEL(TT, 8); else LMK_SEL(TT, 16);          \
  } while (0)
  if (dtype == LMK_BF16) LMK_SEL_N(__nv_bfloat16);
  else LMK_SEL_N(__half);
#undef LMK_SEL_N
#undef LMK_SEL
  LMK_CUDA(cudaGetLastError());
  return LMK_OK;
}

extern "C" int lmk_prefix_gather_supported(int D, int block, int top_k, int T, int tail_len, int dtype) {
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D == kBD && block >= 1 && block <= kGatherMaxBlk && tail_len >= 0 &&
         tail_len <= kGatherMaxBlk && top_k >= 1 && top_k <= 32 && T >= 1 && T <= 8192 ? 1 : 0;
}

extern "C" int lmk_prefix_gather(const void* q, const void* k_cache, const void* v_cache, const lmk_cache_desc* kdesc,
                                 const lmk_cache_desc* vdesc, const int32_t* idx, const int64_t idx_strides[3],
                                 const void* cos_table, const void* sin_table, int n_pos, int rotary, const void* tail_k,
                                 const void* tail_v, const int64_t tail_strides[3], int tail_len, int tail_pos, void* att,
                                 void* v_out, int B, int H, int T, int D, float sm_scale, int dtype, void* stream) {
  LMK_CHECK_ARG(q && k_cache && v_cache && kdesc && vdesc && idx && idx_strides && att && v_out, "prefix_gather: null pointer");
  LMK_CHECK_ARG(tail_len == 0 || (tail_k && tail_v && tail_strides), "prefix_gather: tail rows missing");
  if (!lmk_prefix_gather_supported(D, kdesc->block, kdesc->top_k, T, tail_len, dtype) || !vec_aligned(kdesc) || !vec_aligned(vdesc))
    return fail(LMK_ERR_UNSUPPORTED, "prefix_gather: 16-bit type, D=128, block and tail <= %d, T <= 8192", kGatherMaxBlk);
  LMK_CHECK_ARG(kdesc->n_blocks >= 1 && kdesc->top_k <= kdesc->n_blocks && kdesc->block == vdesc->block, "prefix_gather: bad descriptor");
  LMK_CHECK_ARG(rotary >= LMK_ROTARY_NONE && rotary <= LMK_ROTARY_INTERLEAVED &&
                (rotary == LMK_ROTARY_NONE || (cos_table && sin_table && n_pos >= 1)),
                "prefix_gather: rotary tables missing");
  LMK_CHECK_ARG(B >= 1 && H >= 1 && (int64_t)B * H <= 65535, "prefix_gather: bad sizes");
  uintptr_t align = (uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)cos_table | (uintptr_t)sin_table | (uintptr_t)v_out;
  PrefixParams p{};
  if (tail_len > 0) {
    align |= (uintptr_t)tail_k | (uintptr_t)tail_v;
    for (int i = 0; i < 3; ++i) {
      LMK_CHECK_ARG(tail_strides[i] % 8 == 0, "prefix_gather: tail strides must be multiples of 8");
      p.ts[i] = tail_strides[i];
    }
  }
  LMK_CHECK_ARG((align & 15) == 0, "prefix_gather: pointers must be 16-byte aligned");
  p.q = q; p.k_cache = k_cache; p.v_cache = v_cache; p.kd = *kdesc; p.vd = *vdesc; p.idx = idx;
  for (int i = 0; i < 3; ++i) p.is[i] = idx_strides[i];
  p.cos_t = cos_table; p.sin_t = sin_table; p.n_pos = n_pos; p.rotary = rotary;
  p.tail_k = tail_k; p.tail_v = tail_v; p.tail_len = tail_len; p.tail_pos = tail_pos;
  p.att = att; p.v_out = v_out; p.H = H; p.T = T; p.scale = sm_scale;
  const size_t smem = gather_smem(kdesc->block > tail_len ? kdesc->block : tail_len, T);
  const dim3 grid(kdesc->n_blocks + (tail_len > 0 ? 1 : 0), B * H);
#define LMK_GAT(TT)                                                                                                        \
  do {                                                                                                                     \
    LMK_CUDA(cudaFuncSetAttribute(prefix_gather_kernel<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));      \
    prefix_gather_kernel<TT><<<grid, kGatherThreads, smem, (cudaStream_t)stream>>>(p);                                     \
  } while (0)
  if (dtype == LMK_BF16) LMK_GAT(__nv_bfloat16);
  else LMK_GAT(__half);
#undef LMK_GAT
  LMK_CUDA(cudaGetLastError());
  return LMK_OK;
}

extern "C" int lmk_prefix_pv(const float* probs, int64_t probs_ld, const void* v, const int64_t v_strides[3], void* y, int B, int H,
                             int T, int P, int D, int dtype, void* stream) {
  LMK_CHECK_ARG(probs && v && v_strides && y, "prefix_pv: null pointer");
  if ((dtype != LMK_BF16 && dtype != LMK_F16) || D != kBD || P > 8192)
    return fail(LMK_ERR_UNSUPPORTED, "prefix_pv: 16-bit type, D=128, at most 8192 prefix rows");
  LMK_CHECK_ARG(B >= 1 && H >= 1 && T >= 1 && P >= 1 && (int64_t)B * H <= 65535, "prefix_pv: bad sizes");
  LMK_CHECK_ARG(((uintptr_t)v & 15) == 0 && v_strides[0] % 8 == 0 && v_strides[1] % 8 == 0 && v_strides[2] % 8 == 0,
                "prefix_pv: values must be rows of 16-byte vectors");
  const size_t smem = sizeof(float) * (P > 8 * kBD ? P : 8 * kBD);
  const dim3 grid(T, B * H);
  if (dtype == LMK_BF16)
    prefix_pv_kernel<__nv_bfloat16><<<grid, 256, smem, (cudaStream_t)stream>>>(probs, probs_ld, (const __nv_bfloat16*)v,
        v_strides[0], v_strides[1], v_strides[2], (__nv_bfloat16*)y, H, T, P);
  else
    prefix_pv_kernel<__half><<<grid, 256, smem, (cudaStream_t)stream>>>(probs, probs_ld, (const __half*)v, v_strides[0],
        v_strides[1], v_strides[2], (__half*)y, H, T, P);
  LMK_CUDA(cudaGetLastError());
  return LMK_OK;
}
