// Stand-alone landmark grouped softmax (forward and backward) on materialised score rows.
//
// One warp owns one row [Lk].  Keys that are neither landmark, last-section nor hidden belong to the group whose
// id is the running count of landmarks (an inclusive prefix count, so ids never decrease along the row and each
// group is a contiguous run once bucket members are given the identity element).  The bucket = {landmarks,
// last-section keys, hidden keys} has its own softmax.  Group reductions are segmented warp scans keyed on the
// prefix count; the last lane of each segment is the only writer of that group's slot, and chunks are visited
// in order, so results are bit-reproducible (no floating-point atomics).
//
// Reference semantics: llama/llama_mem.py:168-243 (guards = 0) and lm_benchmark/models/landmark.py:37-119
// (guards = 1: an all -inf group yields 0 instead of NaN, :48,:54).
#include <algorithm>

#include "common.cuh"
#include "mma16.cuh"
#include "sm100_ptx.cuh"
#include "attn_params.h"

namespace lmk {
namespace {

constexpr int kGsWarps = 4;

struct GsParams {
  const void* x;
  int64_t xs[3];
  const uint8_t* is_mem; int64_t ms[4];
  const uint8_t* last; int64_t ls[4];
  const uint8_t* hidden; int64_t hs[4];
  float* probs;
  float* group_prob; int max_mem_cnt;
  const float* gprobs;
  void* gx; int gx_as_x;     // gx holds fp32, or x's type where gx_as_x is set
  int B, H, Lq, Lk, guards, max_groups;
  // causal mode of the rows kernel: the three masks are derived from one flag per (batch row, key) and the rule
  // "query i sees keys 0 .. i + Lk - Lq" (mask block of lm_benchmark/models/landmark.py:210-224); hidden scores count
  // as -inf whatever x holds there
  const uint8_t* row_flags; int64_t row_flags_stride; int causal;
  int* status;          // device status word: set to kErrSoftmaxGroups when a row holds max_groups or more landmarks
};

enum { kErrSoftmaxGroups = 501 };

struct Elem {
  float x;
  bool mem, last, hid, bucket, in;
  int c;   // inclusive landmark count
};

template <typename T>
struct RowReader {
  const T* x;
  const uint8_t *m, *l, *h;
  int64_t mcs, lcs, hcs;
  int Lk, lane;
  int base;   // landmarks seen before the current chunk
  __device__ __forceinline__ void restart() { base = 0; }
  __device__ __forceinline__ Elem load(int j0) {
    Elem e;
    int j = j0 + lane;
    e.in = j < Lk;
    e.x = e.in ? to_f32(x[j]) : -INFINITY;
    e.mem = e.in && m[j * mcs] != 0;
    e.last = e.in && l[j * lcs] != 0;
    e.hid = e.in && h != nullptr && h[j * hcs] != 0;
    unsigned bal = __ballot_sync(0xffffffffu, e.mem);
    e.c = base + __popc(bal & (0xffffffffu >> (31 - lane)));
    base += __popc(bal);
    e.bucket = e.mem || e.last || e.hid || !e.in;
    return e;
  }
};

// inclusive segmented scans over lanes; segments = runs of equal key
__device__ __forceinline__ float seg_scan_max(float v, int key, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    float u = __shfl_up_sync(0xffffffffu, v, o);
    int k = __shfl_up_sync(0xffffffffu, key, o);
    if (lane >= o && k == key) v = fmaxf(v, u);
  }
  return v;
}
__device__ __forceinline__ float seg_scan_sum(float v, int key, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    float u = __shfl_up_sync(0xffffffffu, v, o);
    int k = __shfl_up_sync(0xffffffffu, key, o);
    if (lane >= o && k == key) v += u;
  }
  return v;
}
__device__ __forceinline__ bool seg_tail(int key, int lane) {
  int nk = __shfl_down_sync(0xffffffffu, key, 1);
  return lane == 31 || nk != key;
}

template <typename T, bool kBackward>
__global__ void __launch_bounds__(kGsWarps * 32) grouped_softmax_kernel(GsParams p) {
  extern __shared__ float gs_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G = p.max_groups;
  float* gmax = gs_smem + (size_t)warp * G * 4;
  float* gsum = gmax + G;
  float* gw = gsum + G;     // exp(landmark score - bucket max) of the landmark closing each group
  float* gc = gw + G;       // backward: sum over the group of inner prob * grad
  const int64_t row = (int64_t)blockIdx.x * kGsWarps + warp;
  const int64_t rows = (int64_t)p.B * p.H * p.Lq;
  if (row >= rows) return;
  const int b = (int)(row / ((int64_t)p.H * p.Lq));
  const int h = (int)((row / p.Lq) % p.H);
  const int i = (int)(row % p.Lq);

  RowReader<T> rd;
  rd.x = reinterpret_cast<const T*>(p.x) + b * p.xs[0] + h * p.xs[1] + i * p.xs[2];
  rd.m = p.is_mem + b * p.ms[0] + h * p.ms[1] + i * p.ms[2];
  rd.l = p.last + b * p.ls[0] + h * p.ls[1] + i * p.ls[2];
  rd.h = p.hidden ? p.hidden + b * p.hs[0] + h * p.hs[1] + i * p.hs[2] : nullptr;
  rd.mcs = p.ms[3]; rd.lcs = p.ls[3]; rd.hcs = p.hs[3];
  rd.Lk = p.Lk; rd.lane = lane;
  const bool guards = p.guards != 0;

  for (int g = lane; g < G; g += 32) {
    gmax[g] = -INFINITY;
    gsum[g] = 0.f;
    gw[g] = 0.f;
    gc[g] = 0.f;
  }
  __syncwarp();

  // pass 1: maxima
  float bmax = -INFINITY;
  rd.restart();
  for (int j0 = 0; j0 < p.Lk; j0 += 32) {
    Elem e = rd.load(j0);
    bmax = fmaxf(bmax, (e.bucket && e.in) ? e.x : -INFINITY);
    float v = seg_scan_max(e.bucket ? -INFINITY : e.x, e.c, lane);
    if (seg_tail(e.c, lane) && e.c < G) gmax[e.c] = fmaxf(gmax[e.c], v);
    __syncwarp();
  }
  if (lane == 0 && rd.base >= G && p.status != nullptr) atomicCAS(p.status, 0, kErrSoftmaxGroups);
  bmax = warp_max(bmax);
  if (guards && isinf(bmax)) bmax = 0.f;

  // pass 2: sums; remember exp(landmark - bmax) per closed group
  float bsum = 0.f;
  rd.restart();
  for (int j0 = 0; j0 < p.Lk; j0 += 32) {
    Elem e = rd.load(j0);
    float ex = 0.f;
    if (e.in) {
      if (e.bucket) {
        ex = expf(e.x - bmax);
        bsum += ex;
        if (e.mem && e.c - 1 < G) gw[e.c - 1] = ex;
      } else if (e.c < G) {
        float mx = gmax[e.c];
        if (guards && isinf(mx)) mx = 0.f;
        ex = expf(e.x - mx);
      }
    }
    float v = seg_scan_sum(e.bucket ? 0.f : ex, e.c, lane);
    if (seg_tail(e.c, lane) && e.c < G) gsum[e.c] += v;
    __syncwarp();
  }
  bsum = warp_sum(bsum);
  const float binv = (guards && bsum < 0.5f) ? 0.f : 1.f / bsum;

  if (!kBackward) {
    float* out = p.probs + row * p.Lk;
    float last_total = 0.f;
    rd.restart();
    for (int j0 = 0; j0 < p.Lk; j0 += 32) {
      Elem e = rd.load(j0);
      float pr = 0.f;
      if (e.in) {
        if (e.bucket) {
          pr = e.last ? expf(e.x - bmax) * binv : 0.f;
          if (!guards && !e.last) pr = expf(e.x - bmax) * binv * 0.f;   // keeps NaN propagation of the llama flavour
          last_total += e.last ? pr : 0.f;
        } else if (e.c < G) {
          float mx = gmax[e.c];
          if (guards && isinf(mx)) mx = 0.f;
          float den = gsum[e.c];
          float inner = (guards && den < 0.5f) ? 0.f : expf(e.x - mx) / den;
          pr = inner * (gw[e.c] * binv);
        }
        out[j0 + lane] = pr;
      }
    }
    if (p.group_prob != nullptr) {
      last_total = warp_sum(last_total);
      float* gp = p.group_prob + row * p.max_mem_cnt;
      for (int g = lane; g < p.max_mem_cnt - 1; g += 32) gp[g] = g < G ? gw[g] * binv : 0.f;
      if (lane == 0) gp[p.max_mem_cnt - 1] = last_total;
    }
  } else {
    // pass 3: c_g = sum_j inner_j * grad_j per group, T = sum_j P_j * grad_j over the row
    const float* gr = p.gprobs + row * p.Lk;
    float total = 0.f;
    rd.restart();
    for (int j0 = 0; j0 < p.Lk; j0 += 32) {
      Elem e = rd.load(j0);
      float contrib = 0.f;
      if (e.in) {
        float gj = gr[j0 + lane];
        if (e.bucket) {
          if (e.last) total += expf(e.x - bmax) * binv * gj;
        } else if (e.c < G) {
          float mx = gmax[e.c];
          if (guards && isinf(mx)) mx = 0.f;
          float den = gsum[e.c];
          float inner = (guards && den < 0.5f) ? 0.f : expf(e.x - mx) / den;
          contrib = inner * gj;
          total += contrib * gw[e.c] * binv;
        }
      }
      float v = seg_scan_sum(contrib, e.c, lane);
      if (seg_tail(e.c, lane) && e.c < G) gc[e.c] += v;
      __syncwarp();
    }
    total = warp_sum(total);
    // pass 4: gradients
    rd.restart();
    for (int j0 = 0; j0 < p.Lk; j0 += 32) {
      Elem e = rd.load(j0);
      if (!e.in) continue;
      float gj = gr[j0 + lane];
      float dx = 0.f;
      if (e.bucket) {
        float bj = expf(e.x - bmax) * binv;
        float hj = (e.last ? gj : 0.f) + ((e.mem && e.c - 1 < G) ? gc[e.c - 1] : 0.f);
        dx = (e.hid && !e.last && !e.mem) ? 0.f : bj * (hj - total);
      } else if (e.c < G) {
        float mx = gmax[e.c];
        if (guards && isinf(mx)) mx = 0.f;
        float den = gsum[e.c];
        float inner = (guards && den < 0.5f) ? 0.f : expf(e.x - mx) / den;
        dx = inner * gw[e.c] * binv * (gj - gc[e.c]);
      }
      if (p.gx_as_x) reinterpret_cast<T*>(p.gx)[row * p.Lk + j0 + lane] = from_f32<T>(dx);
      else reinterpret_cast<float*>(p.gx)[row * p.Lk + j0 + lane] = dx;
    }
  }
}


// ---------------------------------------------------------------------------------------------------------------
// Rows of up to kFastMaxLk keys: the row is copied from global memory to shared memory once (cp.async, the whole row
// in flight at a time), eight contiguous keys per lane, and kept there (raw scores, then exponentials) together with
// the decoded mask bits and the landmark count in front of every lane's keys.  A lane walks its eight keys
// sequentially; only the partial result of the group that is open at the lane's last key (and, for lanes holding a
// landmark, the part in front of its first landmark) crosses lanes, through one segmented scan per 256 keys instead
// of one per 32.  Chunks of 256 keys that are hidden and -inf throughout (the upper triangle of a causal score
// matrix) are recognised in the first pass and skipped by the others.  All sums are taken in a fixed order, so
// results are bit-reproducible.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kFastMaxLk = 4096;
constexpr int kFastChunk = 256;
constexpr size_t kFastMaxSmem = 96 * 1024;
constexpr float kLog2e = 1.4426950408889634f;

// exp(a - b) as 2^((a - b) * log2 e): the difference is formed first, so that the argument's rounding error stays
// proportional to the (small) distance from the maximum.
__device__ __forceinline__ float exp_diff(float a, float b) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"((a - b) * kLog2e));
  return y;
}

// Raw flags of a lane's eight keys, one byte per key: lo = keys 0-3, hi = keys 4-7;
// bit 0 landmark, bit 1 last section, bit 2 hidden, bit 3 inside the row.  Keys beyond the row's end read 0x04.
struct RawFlags { uint32_t lo, hi; };

// Byte-wise forms of the row accesses for rows whose pieces are unaligned, strided or cut by the row's end; kept out
// of line so that the common path stays small in the instruction cache.
__device__ __noinline__ uint2 mask_bytes_slow(const uint8_t* p, int64_t cs, int j, int n_in) {
  uint2 w = make_uint2(0u, 0u);
  for (int v = 0; v < n_in; ++v)
    if (p[(int64_t)(j + v) * cs] & 1u) (v < 4 ? w.x : w.y) |= 1u << (8 * (v & 3));
  return w;
}
__device__ __noinline__ float4 load4f_slow(const float* g, int n) {
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  if (n > 0) r.x = g[0];
  if (n > 1) r.y = g[1];
  if (n > 2) r.z = g[2];
  if (n > 3) r.w = g[3];
  return r;
}
__device__ __noinline__ void store4f_slow(float* g, int n, float4 r) {
  if (n > 0) g[0] = r.x;
  if (n > 1) g[1] = r.y;
  if (n > 2) g[2] = r.z;
  if (n > 3) g[3] = r.w;
}

struct MaskRow {
  const uint8_t* p;
  int64_t cs;
  bool vec;
  __device__ __forceinline__ void init(const uint8_t* ptr, int64_t stride) {
    p = ptr; cs = stride;
    vec = ptr != nullptr && stride == 1 && (reinterpret_cast<uintptr_t>(ptr) & 7) == 0;
  }
  // eight mask bytes (bit 0 of each is the truth value) of keys j .. j + 7; n_in of them lie inside the row
  __device__ __forceinline__ uint2 load8(int j, int n_in) const {
    if (p == nullptr) return make_uint2(0u, 0u);
    if (vec && n_in == 8) {
      const uint2 w = *reinterpret_cast<const uint2*>(p + j);
      return make_uint2(w.x & 0x01010101u, w.y & 0x01010101u);
    }
    return mask_bytes_slow(p, cs, j, n_in);
  }
};

// Flags of a lane's eight keys after the first pass, one nibble per key: key v sits in byte v & 3, nibble v >> 2;
// bit 0 landmark, bit 1 last section, bit 2 bucket (landmark, last section, hidden or outside the row),
// bit 3 hidden without being landmark or last section.
__device__ __forceinline__ uint32_t nibble_flags(uint32_t t) {
  const uint32_t bucket = (t | (t >> 1) | (t >> 2) | ~(t >> 3)) & 0x01010101u;
  const uint32_t off = (t >> 2) & ~(t >> 1) & ~t & 0x01010101u;
  return (t & 0x03030303u) | (bucket << 2) | (off << 3);
}
#define LMK_KEY_FLAG(F, v, bit) ((((F) >> (8 * ((v) & 3) + 4 * ((v) >> 2) + (bit))) & 1u) != 0)

// Per (chunk, lane) record kept in shared memory.
//   flags: see nibble_flags
//   info:  c0 (13 bits) | landmarks in the lane << 13 (4 bits) | scan flags << 17 (6 bits) | dead << 23
struct Meta {
  uint32_t flags, info;
  __device__ __forceinline__ int c0() const { return (int)(info & 0x1fffu); }
  __device__ __forceinline__ int nlm() const { return (int)((info >> 13) & 15u); }
  __device__ __forceinline__ bool dead() const { return (info >> 23) & 1u; }
};

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Eight floats of one lane in the row buffer: two 16-byte accesses, conflict-free across the warp.
__device__ __forceinline__ void row_put(float* buf, int lane, const float (&x)[8]) {
  *reinterpret_cast<float4*>(buf + lane * 4) = make_float4(x[0], x[1], x[2], x[3]);
  *reinterpret_cast<float4*>(buf + 128 + lane * 4) = make_float4(x[4], x[5], x[6], x[7]);
}
__device__ __forceinline__ void row_get(const float* buf, int lane, float (&x)[8]) {
  float4 a = *reinterpret_cast<const float4*>(buf + lane * 4), b = *reinterpret_cast<const float4*>(buf + 128 + lane * 4);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void load8f(const float* g, bool vec, int n_in, float (&x)[8]) {
  float4 a, b;
  if (vec && n_in == 8) {
    a = *reinterpret_cast<const float4*>(g);
    b = *reinterpret_cast<const float4*>(g + 4);
  } else {
    a = load4f_slow(g, n_in);
    b = load4f_slow(g + 4, n_in - 4);
  }
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void store8f(float* g, bool vec, int n_in, const float (&x)[8]) {
  const float4 a = make_float4(x[0], x[1], x[2], x[3]), b = make_float4(x[4], x[5], x[6], x[7]);
  if (vec && n_in == 8) {
    *reinterpret_cast<float4*>(g) = a;
    *reinterpret_cast<float4*>(g + 4) = b;
  } else {
    store4f_slow(g, n_in, a);
    store4f_slow(g + 4, n_in - 4, b);
  }
}

// Copies the lane's keys of every chunk into the row buffer: asynchronously where the 16-byte pieces are aligned
// and wholly inside the row, with plain loads elsewhere (-inf beyond the row's end).  16-bit scores are parked in
// the upper half of the chunk's slot and widened by stage_get.
template <typename T>
__device__ __forceinline__ void stage_row(const T* x, int Lk, int n_chunks, int lane, float* xbuf) {
  const bool xvec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  // chunks in which this lane's eight keys lie wholly inside the row
  const int n_full = xvec ? max(Lk - lane * 8 - 8 + kFastChunk, 0) / kFastChunk : 0;
  {
    const T* src = x + lane * 8;
    uint32_t dst = (uint32_t)__cvta_generic_to_shared(xbuf + lane * 4);
    for (int k = 0; k < n_full; ++k) {
      if constexpr (sizeof(T) == 4) {
        cp_async16(dst, src);
        cp_async16(dst + 512, src + 4);
      } else {
        cp_async16(dst + 512, src);
      }
      src += kFastChunk;
      dst += kFastChunk * 4;
    }
  }
  for (int k = n_full; k < n_chunks; ++k) {
    const int j = k * kFastChunk + lane * 8;
    float* buf = xbuf + k * kFastChunk;
    float t[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) t[v] = j + v < Lk ? to_f32(x[j + v]) : -INFINITY;
    if constexpr (sizeof(T) == 4) {
      row_put(buf, lane, t);
    } else {                                  // park as 16-bit values, like the asynchronous copies
      T* e = reinterpret_cast<T*>(buf + 128 + lane * 4);
#pragma unroll
      for (int v = 0; v < 8; ++v) e[v] = from_f32<T>(t[v]);
    }
  }
}
template <typename T>
__device__ __forceinline__ void stage_get(float* buf, int lane, float (&x)[8]) {
  if constexpr (sizeof(T) == 4) {
    row_get(buf, lane, x);
  } else {
    uint4 w = *reinterpret_cast<const uint4*>(buf + 128 + lane * 4);
    const T* e = reinterpret_cast<const T*>(&w);
#pragma unroll
    for (int v = 0; v < 8; ++v) x[v] = to_f32(e[v]);
    row_put(buf, lane, x);                      // only this lane's own parked bytes are overwritten
  }
}

// Folds the per-lane partial results of one chunk into the per-group accumulators.  `head` covers the lane's keys in
// front of its first landmark (all of them if it has none) and belongs to group c0; `tail` covers the keys behind its
// last landmark and belongs to group c0 + nlm.  Groups that begin and end inside one lane were written by that lane.
// flags: bit s (s < 5) = step s of the segmented scan combines with the lane 2^s below, bit 5 = the lane ends a run
// of lanes whose last key lies in the same group.
template <bool kMax>
__device__ __forceinline__ void fold_chunk(float head, float tail, int nlm, int c0, uint32_t flags, float* acc, int G,
                                           int lane) {
  const int key = c0 + nlm;
  float v = nlm ? tail : head;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    float u = __shfl_up_sync(0xffffffffu, v, 1 << s);
    if ((flags >> s) & 1u) v = kMax ? fmaxf(v, u) : v + u;
  }
  const float hn = __shfl_down_sync(0xffffffffu, head, 1);
  if (flags & 32u) {
    if (lane < 31) v = kMax ? fmaxf(v, hn) : v + hn;
    if (key < G) acc[key] = kMax ? fmaxf(acc[key], v) : acc[key] + v;
  }
  if (lane == 0 && nlm > 0 && c0 < G) acc[c0] = kMax ? fmaxf(acc[c0], head) : acc[c0] + head;
  __syncwarp();
}

// (batch, head, query) of a row; B * H fits 32 bits
__device__ __forceinline__ void row_index(const GsParams& p, int64_t row, int& b, int& h, int& i) {
  uint32_t bh;
  if ((int64_t)p.B * p.H * p.Lq <= 0xffffffffLL) {
    bh = (uint32_t)row / (uint32_t)p.Lq;
    i = (int)((uint32_t)row - bh * (uint32_t)p.Lq);
  } else {
    bh = (uint32_t)(row / p.Lq);
    i = (int)(row - (int64_t)bh * p.Lq);
  }
  b = (int)(bh / (uint32_t)p.H);
  h = (int)(bh - (uint32_t)b * (uint32_t)p.H);
}

template <typename T, bool kBackward, bool kCausal>
__device__ __forceinline__ void grouped_softmax_chunked_row(const GsParams& p, int n_chunks, int64_t row, float* xbuf) {
  const int lane = threadIdx.x & 31;
  const int G = p.max_groups;
  Meta* meta = reinterpret_cast<Meta*>(xbuf + (size_t)n_chunks * kFastChunk) + lane;   // [chunk][lane]
  float* gmax = xbuf + (size_t)n_chunks * (kFastChunk + 64);
  float* gsum = gmax + G;
  float* gw = gsum + G;     // exp(landmark score - bucket max) of the landmark closing each group
  float* gc = gw + G;       // backward: sum over the group of inner prob * grad
  int b, h, i;
  row_index(p, row, b, h, i);
  const bool guards = p.guards != 0;

  const T* xrow = reinterpret_cast<const T*>(p.x) + b * p.xs[0] + h * p.xs[1] + i * p.xs[2];
  constexpr bool causal = kCausal;
  const int pi = i + p.Lk - p.Lq;                   // causal mode: the last key this query sees
  const int n_live = causal ? min(n_chunks, pi / kFastChunk + 1) : n_chunks;   // chunks with a visible key
  stage_row<T>(xrow, p.Lk, n_live, lane, xbuf);            // asynchronous copies, awaited below
  MaskRow mm, ml, mh;
  int p_last = -1;                                  // causal mode: the last landmark in front of key pi
  if (causal) {
    mm.init(p.row_flags + b * p.row_flags_stride, 1);
    ml.init(nullptr, 0);
    mh.init(nullptr, 0);
    for (int j0 = (max(pi - 1, 0) / kFastChunk) * kFastChunk; j0 >= 0 && p_last < 0; j0 -= kFastChunk) {
      const int j = j0 + lane * 8;
      const uint2 m = mm.load8(j, min(max(min(p.Lk, pi) - j, 0), 8));      // keys in front of pi only
      const uint64_t w = ((uint64_t)m.y << 32) | m.x;
      int best = w ? j + (63 - __clzll((long long)w)) / 8 : -1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
      p_last = best;
    }
  } else {
    mm.init(p.is_mem + b * p.ms[0] + h * p.ms[1] + i * p.ms[2], p.ms[3]);
    ml.init(p.last + b * p.ls[0] + h * p.ls[1] + i * p.ls[2], p.ls[3]);
    mh.init(p.hidden ? p.hidden + b * p.hs[0] + h * p.hs[1] + i * p.hs[2] : nullptr, p.hs[3]);
  }
  auto low_bytes = [](int n) -> uint64_t { return n >= 8 ? ~0ull : ((1ull << (8 * n)) - 1ull); };
  auto load_flags = [&](int k) -> RawFlags {
    const int j = k * kFastChunk + lane * 8;
    const int n_in = min(max(p.Lk - j, 0), 8);
    RawFlags f;
    if (causal) {
      constexpr uint64_t kOnes = 0x0101010101010101ull;
      const uint2 m = mm.load8(j, n_in);
      const uint64_t m64 = ((uint64_t)m.y << 32) | m.x;
      const uint64_t inside = kOnes & low_bytes(n_in);
      const uint64_t vis = inside & low_bytes(min(max(pi - j + 1, 0), 8));       // keys 0 .. pi
      const uint64_t front = kOnes & low_bytes(min(max(pi - j, 0), 8));           // keys in front of pi
      const uint64_t open = kOnes & ~low_bytes(min(max(p_last + 1 - j, 0), 8));   // keys behind the last landmark
      const uint64_t mem = m64 & vis & front;        // a landmark at pi itself is masked like a hidden key
      const uint64_t last = vis & ~m64 & open;
      const uint64_t hid = kOnes & ~(mem | last | (vis & ~m64));
      const uint64_t w = mem | (last << 1) | (hid << 2) | (inside << 3);
      f.lo = (uint32_t)w;
      f.hi = (uint32_t)(w >> 32);
      return f;
    }
    const uint2 m = mm.load8(j, n_in), l = ml.load8(j, n_in), hd = mh.load8(j, n_in);
    f.lo = m.x | (l.x << 1) | (hd.x << 2);
    f.hi = m.y | (l.y << 1) | (hd.y << 2);
    if (n_in == 8) {
      f.lo |= 0x08080808u;
      f.hi |= 0x08080808u;
    } else {                                    // keys beyond the row's end: hidden, outside
      const uint64_t inside = n_in ? (0x0808080808080808ull >> (8 * (8 - n_in))) : 0ull;
      const uint64_t w = (((uint64_t)f.hi << 32) | f.lo) | inside | (0x0404040404040404ull & ~(inside >> 1));
      f.lo = (uint32_t)w;
      f.hi = (uint32_t)(w >> 32);
    }
    return f;
  };

  const RawFlags raw0 = load_flags(0);              // under way while the row arrives
  for (int g = lane; g < G; g += 32) {
    gmax[g] = -INFINITY;
    gsum[g] = 0.f;
    gw[g] = 0.f;
    gc[g] = 0.f;
  }
  cp_async_wait_all();
  __syncwarp();

  // pass 1: decode the masks, count the landmarks, group and bucket maxima
  float bmax = -INFINITY;
  {
    int base = 0;
    RawFlags raw = raw0;
    for (int k = 0; k < n_chunks; ++k) {
      if (k >= n_live) {                            // causal mode: nothing visible from here on, nothing was read
        meta[k * 32] = Meta{0u, (uint32_t)base | (1u << 23)};
        continue;
      }
      RawFlags nraw = raw;
      if (k + 1 < n_live) nraw = load_flags(k + 1);
      float x[8];
      stage_get<T>(xbuf + k * kFastChunk, lane, x);
      if (causal && k == n_live - 1) {              // hidden scores count as -inf whatever the tensor holds
#pragma unroll
        for (int v = 0; v < 8; ++v)
          if (((v < 4 ? raw.lo : raw.hi) >> (8 * (v & 3) + 2)) & 1u) x[v] = -INFINITY;
        row_put(xbuf + k * kFastChunk, lane, x);
      }
      // all keys of the lane hidden, none a landmark or in the last section
      const bool shut = (raw.lo & raw.hi & 0x04040404u) == 0x04040404u && ((raw.lo | raw.hi) & 0x03030303u) == 0u;
      if (__all_sync(0xffffffffu, shut)) {
        bool inert = true;
#pragma unroll
        for (int v = 0; v < 8; ++v) inert = inert && x[v] == -INFINITY;
        if (__all_sync(0xffffffffu, inert)) {     // nothing finite either: the other passes skip the chunk
          meta[k * 32] = Meta{0u, (uint32_t)base | (1u << 23)};
          raw = nraw;
          continue;
        }
      }
      const uint32_t F = nibble_flags(raw.lo) | (nibble_flags(raw.hi) << 4);
      const int nlm = __popc(F & 0x11111111u);
      // landmarks in front of this lane's keys within the chunk
      const unsigned starts = __ballot_sync(0xffffffffu, nlm != 0);
      int c0;
      if (__ballot_sync(0xffffffffu, nlm > 1) == 0) {
        c0 = base + __popc(starts & ((1u << lane) - 1u));
        base += __popc(starts);
      } else {
        int inc = nlm;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          int t = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += t;
        }
        c0 = base + inc - nlm;
        base += __shfl_sync(0xffffffffu, inc, 31);
      }
      // a lane holding a landmark begins a run of lanes whose last key lies in the same group
      const unsigned below = starts & ((2u << lane) - 1u);
      const int dist = lane - (below ? 31 - __clz(below) : 0);
      uint32_t flags = (1u << (32 - __clz(dist))) - 1u;
      if (lane == 31 || ((starts >> 1) >> lane) & 1u) flags |= 32u;

      float run = -INFINITY, head = -INFINITY;
      int c = c0;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        if (LMK_KEY_FLAG(F, v, 0)) {
          if (c == c0) head = run;
          else if (c < G) gmax[c] = fmaxf(gmax[c], run);
          run = -INFINITY;
          ++c;
        }
        const bool bk = LMK_KEY_FLAG(F, v, 2);           // keys outside the row hold -inf
        run = fmaxf(run, bk ? -INFINITY : x[v]);
        bmax = fmaxf(bmax, bk ? x[v] : -INFINITY);
      }
      meta[k * 32] = Meta{F, (uint32_t)c0 | ((uint32_t)nlm << 13) | (flags << 17)};
      fold_chunk<true>(nlm ? head : run, run, nlm, c0, flags, gmax, G, lane);
      raw = nraw;
    }
    if (lane == 0 && base >= G && p.status != nullptr) atomicCAS(p.status, 0, kErrSoftmaxGroups);
  }
  bmax = warp_max(bmax);
  if (guards && isinf(bmax)) bmax = 0.f;

  // stabiliser of group c; +inf beyond the last slot makes every exponential of such a group 0
  auto group_max = [&](int c) -> float {
    if (c >= G) return INFINITY;
    const float mx = gmax[c];
    return (guards && isinf(mx)) ? 0.f : mx;
  };

  // pass 2: exponentials (kept in the row buffer), group and bucket sums, landmark weights
  float bsum = 0.f;
  for (int k = 0; k < n_chunks; ++k) {
    const Meta mt = meta[k * 32];
    if (mt.dead()) continue;
    float x[8];
    row_get(xbuf + k * kFastChunk, lane, x);
    const uint32_t F = mt.flags;
    const int c0 = mt.c0();
    int c = c0;
    float mx = group_max(c);
    float run = 0.f, head = 0.f;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const bool bk = LMK_KEY_FLAG(F, v, 2);
      const float ex = exp_diff(x[v], bk ? bmax : mx);     // keys beyond the row's end hold -inf
      x[v] = ex;
      bsum += bk ? ex : 0.f;
      run += bk ? 0.f : ex;
      if (LMK_KEY_FLAG(F, v, 0)) {
        if (c < G) gw[c] = ex;
        if (c == c0) head = run;
        else if (c < G) gsum[c] += run;
        run = 0.f;
        ++c;
        mx = group_max(c);
      }
    }
    row_put(xbuf + k * kFastChunk, lane, x);
    fold_chunk<false>(mt.nlm() ? head : run, run, mt.nlm(), c0, mt.info >> 17, gsum, G, lane);
  }
  bsum = warp_sum(bsum);
  const float binv = (guards && bsum < 0.5f) ? 0.f : 1.f / bsum;

  // scale of a non-bucket key of group c: its outer weight over its group's sum
  auto inv_den = [&](int c) -> float {
    if (c >= G) return 0.f;
    const float den = gsum[c];                      // 0 only for a group without keys: nothing is scaled by it
    return ((guards && den < 0.5f) || den == 0.f) ? 0.f : 1.f / den;
  };
  auto weight = [&](int c) -> float { return c < G ? gw[c] * binv : 0.f; };

  if (!kBackward) {
    float* out = p.probs + row * p.Lk;
    const bool ovec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const float off = guards ? 0.f : binv * 0.f;    // bucket keys outside the last section (NaN if binv is not finite)
    const bool want_gp = p.group_prob != nullptr;
    float last_total = 0.f;
    for (int k = 0; k < n_chunks; ++k) {
      const Meta mt = meta[k * 32];
      const int j = k * kFastChunk + lane * 8;
      const int n_in = min(max(p.Lk - j, 0), 8);
      float x[8];
      if (mt.dead()) {
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = 0.f * off;
        store8f(out + j, ovec, n_in, x);
        continue;
      }
      row_get(xbuf + k * kFastChunk, lane, x);
      const uint32_t F = mt.flags;
      int c = mt.c0();
      float sc = inv_den(c) * weight(c);
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const float s = LMK_KEY_FLAG(F, v, 1) ? binv : (LMK_KEY_FLAG(F, v, 2) ? off : sc);
        x[v] *= s;
        if (LMK_KEY_FLAG(F, v, 0)) {
          ++c;
          sc = inv_den(c) * weight(c);
        }
      }
      if (want_gp) {
#pragma unroll
        for (int v = 0; v < 8; ++v) last_total += LMK_KEY_FLAG(F, v, 1) ? x[v] : 0.f;
      }
      store8f(out + j, ovec, n_in, x);
    }
    if (want_gp) {
      last_total = warp_sum(last_total);
      float* gp = p.group_prob + row * p.max_mem_cnt;
      for (int g = lane; g < p.max_mem_cnt - 1; g += 32) gp[g] = g < G ? gw[g] * binv : 0.f;
      if (lane == 0) gp[p.max_mem_cnt - 1] = last_total;
    }
  } else {
    const float* gr = p.gprobs + row * p.Lk;
    const bool gvec = (reinterpret_cast<uintptr_t>(gr) & 15) == 0;
    auto store_grad = [&](int j, int n_in, const float (&x)[8]) {
      if (p.gx_as_x && sizeof(T) == 2) {
        T* o = reinterpret_cast<T*>(p.gx) + row * p.Lk + j;
#pragma unroll
        for (int v = 0; v < 8; ++v)
          if (v < n_in) o[v] = from_f32<T>(x[v]);
      } else {
        float* o = reinterpret_cast<float*>(p.gx) + row * p.Lk;
        store8f(o + j, (reinterpret_cast<uintptr_t>(o) & 15) == 0, n_in, x);
      }
    };
    // pass 3: c_g = sum_j inner_j * grad_j per group, total = sum_j P_j * grad_j over the row
    float total = 0.f;
    // the gradients of the next live chunk are requested before the current one is worked on
    auto load_grad = [&](int k, float (&g)[8]) {
      const int j = k * kFastChunk + lane * 8;
      load8f(gr + j, gvec, min(max(p.Lk - j, 0), 8), g);
    };
    Meta mnext = meta[0];
    float gn[8];
    if (!mnext.dead()) load_grad(0, gn);
    for (int k = 0; k < n_chunks; ++k) {
      const Meta mt = mnext;
      float x[8], g[8];
#pragma unroll
      for (int v = 0; v < 8; ++v) g[v] = gn[v];
      if (k + 1 < n_chunks) {
        mnext = meta[(k + 1) * 32];
        if (!mnext.dead()) load_grad(k + 1, gn);
      }
      if (mt.dead()) continue;
      row_get(xbuf + k * kFastChunk, lane, x);
      const uint32_t F = mt.flags;
      const int c0 = mt.c0();
      int c = c0;
      float id = inv_den(c), wt = weight(c);
      float run = 0.f, head = 0.f, lsum = 0.f;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const float xg = x[v] * g[v];
        lsum += LMK_KEY_FLAG(F, v, 1) ? xg : 0.f;
        run += LMK_KEY_FLAG(F, v, 2) ? 0.f : xg;
        if (LMK_KEY_FLAG(F, v, 0)) {
          run *= id;
          total += run * wt;
          if (c == c0) head = run;
          else if (c < G) gc[c] += run;
          run = 0.f;
          ++c;
          id = inv_den(c);
          wt = weight(c);
        }
      }
      run *= id;
      total += run * wt + lsum * binv;
      fold_chunk<false>(mt.nlm() ? head : run, run, mt.nlm(), c0, mt.info >> 17, gc, G, lane);
    }
    total = warp_sum(total);
    // pass 4: gradients
    mnext = meta[0];
    if (!mnext.dead()) load_grad(0, gn);
    for (int k = 0; k < n_chunks; ++k) {
      const Meta mt = mnext;
      const int j = k * kFastChunk + lane * 8;
      const int n_in = min(max(p.Lk - j, 0), 8);
      float x[8], g[8];
#pragma unroll
      for (int v = 0; v < 8; ++v) g[v] = gn[v];
      if (k + 1 < n_chunks) {
        mnext = meta[(k + 1) * 32];
        if (!mnext.dead()) load_grad(k + 1, gn);
      }
      if (mt.dead()) {
#pragma unroll
        for (int v = 0; v < 8; ++v) x[v] = 0.f;
        store_grad(j, n_in, x);
        continue;
      }
      row_get(xbuf + k * kFastChunk, lane, x);
      const uint32_t F = mt.flags;
      int c = mt.c0();
      float sc = inv_den(c) * weight(c), cg = c < G ? gc[c] : 0.f;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const bool bk = LMK_KEY_FLAG(F, v, 2), is_last = LMK_KEY_FLAG(F, v, 1);
        // bucket: P_j * ((g_j if last section) - total); group member: P_j * (g_j - c_g)
        const float s = bk ? (LMK_KEY_FLAG(F, v, 3) ? 0.f : binv) : sc;
        const float a = (bk && !is_last) ? 0.f : g[v];
        float dx = x[v] * s * (a - (bk ? total : cg));
        if (LMK_KEY_FLAG(F, v, 0)) {                 // a landmark also receives its group's c_g
          dx = x[v] * binv * ((is_last ? g[v] : 0.f) + cg - total);
          ++c;
          sc = inv_den(c) * weight(c);
          cg = c < G ? gc[c] : 0.f;
        }
        x[v] = dx;
      }
      store_grad(j, n_in, x);
    }
  }
}
#undef LMK_KEY_FLAG

template <typename T, bool kBackward, bool kCausal>
__global__ void __launch_bounds__(kGsWarps * 32) grouped_softmax_rows_kernel(GsParams p, int n_chunks) {
  extern __shared__ __align__(16) float gs_smem[];
  const int warp = threadIdx.x >> 5;
  const int64_t row = (int64_t)blockIdx.x * kGsWarps + warp;
  if (row >= (int64_t)p.B * p.H * p.Lq) return;
  grouped_softmax_chunked_row<T, kBackward, kCausal>(
      p, n_chunks, row, gs_smem + warp * ((size_t)n_chunks * (kFastChunk + 64) + 4 * (size_t)p.max_groups));
}

// ---------------------------------------------------------------------------------------------------------------
// Rows of up to about 2048 keys with at most two landmarks in 1/32 of the row: lane l owns the 4 n4 contiguous keys
// from l * 4 n4 on (n4 = ceil(keys / 128)), in shared memory through all passes.  A group is then the tail of one lane, whole
// lanes behind it and the head of the lane that holds its landmark: one segmented scan over the lanes per pass reduces
// every group of the row, and two shuffles hand each lane the results of the (at most two) groups its keys lie in; where lanes
// hold two landmarks, the keys between them are a third one.  Nothing per group is kept in memory and no pass looks
// anything up per key.  A row with three landmarks in a lane is done by the chunked form above.
//
// Bound by the instructions per row (two thirds of the issue slots at 40 % of the copy bandwidth), so what can be shared is:
// a warp takes the same query of several heads in turn, and masks that are broadcast over the heads are read, packed to a
// bit per key and split into groups once.  The gradients arrive under the two passes that rebuild the exponentials.  The
// passes are loops over four keys: with the keys in registers and the loops unrolled the kernel took as long (104 + 129 us),
// its code no longer fitted the instruction caches.  A guarded row is worked on only up to its
// last score above -inf, which halves a causal matrix.
//
// Keys are counted from the 4-element boundary at or in front of the row's place in the dense results (`lead` keys earlier),
// so rows of any length are copied, read and written four elements at a time except for the row's two ends.
// B16 H8 512 x 512 fp32, landmarks every 51 keys: forward 138 -> 98 us, backward 216 -> 130 us.  Two landmarks in a lane have code of
// their own (rows of 1064 keys, groups of 32, B2 H32, forward and backward: 994 -> 668 us; by the chunked form 1054).  The chunked form costs
// more from here than as a kernel of its own: rows in which a lane holds three landmarks and more take 1.1 to 1.4 times as long as when
// all rows were done that way (forward and backward, us: B2 H8 1024 x 1024 with groups of 8 170 -> 222, B1 H4 2048 x 2048 with groups
// of 16 221 -> 252, of 8 254 -> 301); whether a row is one of them is only known from its flags.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kLaneMaxPieces = 16;             // n4 of the longest row

// A row in shared memory as pieces of four keys, 16 bytes each (scores of 16 bits wait in the upper half of theirs).
struct LaneRow {
  float* buf;
  int lane;
  // place of the row's c-th piece: one place left out after eight spreads the strides of two to eight pieces, with which
  // the lanes read their own keys, over the banks
  static __device__ __forceinline__ int slot(int c) { return c + (c >> 3); }

  // starts copying the row's keys (counted with its lead) [lead, n) into n4 pieces a lane, `fill` elsewhere.
  // src: key 0, i.e. `lead` elements in front of the row
  template <typename E>
  __device__ __forceinline__ void stage(const E* src, int lead, int n, int n4, float fill) {
    const bool vec = (reinterpret_cast<uintptr_t>(src) & (4 * sizeof(E) - 1)) == 0;
#pragma unroll 1
    for (int c = lane; c < 32 * n4; c += 32) {
      float* d = buf + slot(c) * 4 + (sizeof(E) == 4 ? 0 : 2);
      if (vec && 4 * c >= lead && 4 * c + 4 <= n) {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(d);
        if constexpr (sizeof(E) == 4) cp_async16(a, src + 4 * c);
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(src + 4 * c) : "memory");
      } else {
        E* e = reinterpret_cast<E*>(d);
#pragma unroll 1
        for (int v = 0; v < 4; ++v) e[v] = (4 * c + v >= lead && 4 * c + v < n) ? src[4 * c + v] : from_f32<E>(fill);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  template <typename E>
  __device__ __forceinline__ void get(int slot_c, float* x) const {
    if constexpr (sizeof(E) == 4) {
      const float4 a = reinterpret_cast<const float4*>(buf)[slot_c];
      x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    } else {
      const uint2 w = reinterpret_cast<const uint2*>(buf)[2 * slot_c + 1];
      const E* e = reinterpret_cast<const E*>(&w);
#pragma unroll
      for (int v = 0; v < 4; ++v) x[v] = to_f32(e[v]);
    }
  }
  __device__ __forceinline__ void put(int slot_c, const float* x) {
    reinterpret_cast<float4*>(buf)[slot_c] = make_float4(x[0], x[1], x[2], x[3]);
  }
  // keys [lead, n) to `out` (key 0): n4 pieces a lane from shared memory, zeros behind them
  template <typename E>
  __device__ __forceinline__ void write(E* out, int lead, int n, int n4) const {
    const bool vec = (reinterpret_cast<uintptr_t>(out) & (4 * sizeof(E) - 1)) == 0;
#pragma unroll 1
    for (int c = lane; 4 * c < n; c += 32) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < 32 * n4) a = reinterpret_cast<const float4*>(buf)[slot(c)];
      if (vec && 4 * c >= lead && 4 * c + 4 <= n) {
        if constexpr (sizeof(E) == 4) {
          *reinterpret_cast<float4*>(out + 4 * c) = a;
        } else {
          const E t[4] = {from_f32<E>(a.x), from_f32<E>(a.y), from_f32<E>(a.z), from_f32<E>(a.w)};
          *reinterpret_cast<uint2*>(out + 4 * c) = *reinterpret_cast<const uint2*>(t);
        }
      } else {
        const float t[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int v = 0; v < 4; ++v)
          if (4 * c + v >= lead && 4 * c + v < n) out[4 * c + v] = from_f32<E>(t[v]);
      }
    }
  }
};

// one bit for each of a lane's keys
template <int K>
struct Bits {
  uint32_t w[(K + 31) / 32];
  // bits of the keys of piece q in the lowest four places (others behind them)
  __device__ __forceinline__ uint32_t piece(int q) const {
    return (K <= 32 || q < 8 ? w[0] : w[K <= 32 ? 0 : 1]) >> (4 * (q & 7));
  }
  // the lowest n of K bits
  static __device__ __forceinline__ Bits low(int n) {
    Bits r;
#pragma unroll
    for (int i = 0; i < (K + 31) / 32; ++i) {
      const int m = n - 32 * i;
      r.w[i] = m >= 32 ? ~0u : m <= 0 ? 0u : (1u << m) - 1u;
    }
    return r;
  }
  template <typename F>
  static __device__ __forceinline__ Bits zip(F f) {
    Bits r;
#pragma unroll
    for (int i = 0; i < (K + 31) / 32; ++i) r.w[i] = f(i);
    return r;
  }
  __device__ __forceinline__ int count() const {
    int n = 0;
#pragma unroll
    for (int i = 0; i < (K + 31) / 32; ++i) n += __popc(w[i]);
    return n;
  }
  __device__ __forceinline__ int first() const {           // K where none is set
    int r = K;
#pragma unroll
    for (int i = (K + 31) / 32 - 1; i >= 0; --i)
      if (w[i]) r = 32 * i + __ffs(w[i]) - 1;
    return r;
  }
  __device__ __forceinline__ int top() const {              // highest set bit, -1 where none is set
    int r = -1;
#pragma unroll
    for (int i = 0; i < (K + 31) / 32; ++i)
      if (w[i]) r = 32 * i + 31 - __clz(w[i]);
    return r;
  }
};

__device__ __noinline__ uint32_t mask_quad_slow(const uint8_t* p, int64_t cs, int j, int n) {
  uint32_t b = 0;
  for (int v = 0; v < 4; ++v)
    if (j + v >= 0 && j + v < n) b |= (p[(int64_t)(j + v) * cs] & 1u) << v;
  return b;
}

// bit v of the result = bit 0 of mask byte j0 + v (0 outside the n keys of the row); only words that hold a byte of the
// row are read
template <int K>
__device__ __forceinline__ Bits<K> load_bits(const uint8_t* p, int64_t cs, int j0, int n4, int n) {
  Bits<K> r = Bits<K>::low(0);
  if (cs == 1) {
    const int mis = (int)(reinterpret_cast<uintptr_t>(p) & 3), at = j0 + mis;
    const int first = at >> 2, sh = (at & 3) * 8, words = (mis + n + 3) >> 2;
    const uint32_t* base = reinterpret_cast<const uint32_t*>(p - mis) + first;
    uint32_t w0 = (unsigned)first < (unsigned)words ? base[0] : 0u;
#pragma unroll
    for (int q = 0; q < K / 4; ++q) {
      if (q >= n4) break;
      const uint32_t w1 = (unsigned)(first + q + 1) < (unsigned)words ? base[q + 1] : 0u;
      // bits 0, 8, 16, 24 -> 0 .. 3
      r.w[q >> 3] |= (((__funnelshift_r(w0, w1, sh) & 0x01010101u) * 0x01020408u) >> 24) << (4 * (q & 7));
      w0 = w1;
    }
  } else {
#pragma unroll 1
    for (int q = 0; q < n4; ++q) {
      const uint32_t quad = mask_quad_slow(p, cs, j0 + 4 * q, n) << (4 * (q & 7));
      if (K <= 32 || q < 8) r.w[0] |= quad;
      else r.w[K <= 32 ? 0 : 1] |= quad;
    }
  }
  const Bits<K> in = Bits<K>::low(n - j0), before = Bits<K>::low(-j0);
#pragma unroll
  for (int i = 0; i < (K + 31) / 32; ++i) r.w[i] &= in.w[i] & ~before.w[i];
  return r;
}

// Which lanes a lane's groups reach to.  Group a holds the lane's keys up to its landmark (all of them where it has
// none), group b the keys behind it; a group is closed by the lane of its landmark (none for the row's last group).
struct LaneGroups {
  int lane, dist, src_a, src_b;
  bool own, has_a, has_b;
  __device__ __forceinline__ LaneGroups(int lane_, unsigned owners) : lane(lane_) {
    own = (owners >> lane) & 1u;
    const unsigned below = owners & ((2u << lane) - 1u);                  // landmark lanes up to this one
    dist = lane - (below ? 31 - __clz(below) : 0);
    const unsigned from = owners & ~((1u << lane) - 1u), behind = owners & ~((2u << lane) - 1u);
    has_a = from != 0;
    has_b = behind != 0;
    src_a = has_a ? __ffs(from) - 1 : 31;
    src_b = has_b ? __ffs(behind) - 1 : 31;
  }
  // a: the lane's share of group a, b: of group b (counted where it owns a landmark).  Returns both groups' totals;
  // `closed`: the total of the group that this lane's landmark closes.
  template <bool kMax>
  __device__ __forceinline__ void reduce(float a, float b, float& ta, float& tb, float& closed) const {
    float v = own ? b : a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float u = __shfl_up_sync(0xffffffffu, v, o);
      if (o <= dist) v = kMax ? fmaxf(v, u) : v + u;
    }
    float prev = __shfl_up_sync(0xffffffffu, v, 1);
    if (lane == 0) prev = kMax ? -INFINITY : 0.f;
    closed = kMax ? fmaxf(prev, a) : prev + a;
    const float open = __shfl_sync(0xffffffffu, v, 31);
    ta = __shfl_sync(0xffffffffu, closed, src_a);
    tb = __shfl_sync(0xffffffffu, closed, src_b);
    if (!has_a) ta = open;
    if (!has_b) tb = open;
  }
};

// the masks of a causal row: f = landmark flags, pi = the last key the query sees, `before` = places in front of the row
template <int K>
__device__ __forceinline__ void causal_masks(const Bits<K>& f, const Bits<K>& before, int pi, int lead, int j0, Bits<K>& mem,
                                             Bits<K>& last, Bits<K>& act, Bits<K>& bk) {
  using Mask = Bits<K>;
  const Mask upto = Mask::low(lead + pi + 1 - j0), front = Mask::low(lead + pi - j0);
  const Mask vis = Mask::zip([&](int w) { return upto.w[w] & ~before.w[w]; });
  mem = Mask::zip([&](int w) { return f.w[w] & front.w[w]; });
  const unsigned with = __ballot_sync(0xffffffffu, mem.count() != 0);
  int p_last = __shfl_sync(0xffffffffu, j0 + mem.top(), with ? 31 - __clz(with) : 0);
  if (!with) p_last = -1;
  const Mask closed = Mask::low(p_last + 1 - j0);
  last = Mask::zip([&](int w) { return vis.w[w] & ~f.w[w] & ~closed.w[w]; });
  act = Mask::zip([&](int w) { return vis.w[w] & (~f.w[w] | mem.w[w]); });
  bk = Mask::zip([&](int w) { return mem.w[w] | last.w[w] | ~act.w[w]; });
}

// Passes 1 and 2 of a row: maxima of the groups and of the bucket, then exponentials (they replace the scores in shared
// memory), sums and landmark weights.  binv: 1 / the bucket's sum; for the lane's groups a and b: i = 1 / the group's sum, w = the
// landmark's share of the bucket; elm: exponential of the lane's own landmark.
// What lies between a lane's landmarks (gm): nothing (kInner = kNone: one landmark a lane at most), a group of its own that the second
// one (lm2_slot) closes (kOne), or groups that the caller has worked out (kDone: their places are left alone).
enum { kNone, kOne, kDone };
struct LaneWeights { float binv, ia, ib, wa, wb, elm, im, wm, elm2; };
template <typename T, int K, int kInner>
__device__ __forceinline__ LaneWeights lane_weights(LaneRow& xr, int c0, int n4, int lm_slot, const Bits<K>& ga, const Bits<K>& gb,
                                                    const Bits<K>& bk, const LaneGroups& lg, int ca, int G, bool guards,
                                                    const Bits<K>& gm = Bits<K>(), int lm2_slot = 0, int nlm = 1) {
  constexpr bool kTwo = kInner == kOne;
  const int cb = kInner != kNone ? ca + max(nlm, 1) : ca + 1;
  float vm = -INFINITY;
  // pass 1: group and bucket maxima
  float va = -INFINITY, vb = -INFINITY, bmax = -INFINITY;
#pragma unroll 1
  for (int q = 0; q < n4; ++q) {
    const uint32_t fa = ga.piece(q), fb = gb.piece(q), fk = bk.piece(q);
    float x[4];
    xr.get<T>(xr.slot(c0 + q), x);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      if ((fa >> v) & 1u) va = fmaxf(va, x[v]);
      if ((fb >> v) & 1u) vb = fmaxf(vb, x[v]);
      if ((fk >> v) & 1u) bmax = fmaxf(bmax, x[v]);
      if (kTwo && ((gm.piece(q) >> v) & 1u)) vm = fmaxf(vm, x[v]);
    }
  }
  // the landmarks' scores
  auto score = [&](int at) { return sizeof(T) == 4 ? xr.buf[at] : to_f32(reinterpret_cast<const T*>(xr.buf)[2 * at + 4 - (at & 3)]); };
  float elm = score(lm_slot), elm2 = kTwo ? score(lm2_slot) : 0.f;
  bmax = warp_max(bmax);
  if (guards && isinf(bmax)) bmax = 0.f;
  float ma, mb, closed;
  lg.reduce<true>(va, vb, ma, mb, closed);
  // stabilisers; +inf beyond the last slot makes every exponential of such a group 0
  ma = ca >= G ? INFINITY : (guards && isinf(ma)) ? 0.f : ma;
  mb = cb >= G ? INFINITY : (guards && isinf(mb)) ? 0.f : mb;

  const float mm = ca + 1 >= G ? INFINITY : (guards && isinf(vm)) ? 0.f : vm;

  // pass 2: exponentials, group and bucket sums
  float bsum = 0.f;
  va = vb = vm = 0.f;
#pragma unroll 1
  for (int q = 0; q < n4; ++q) {
    const uint32_t fa = ga.piece(q), fb = gb.piece(q), fk = bk.piece(q);
    const int at = xr.slot(c0 + q);
    float x[4];
    xr.get<T>(at, x);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const bool ib = (fb >> v) & 1u, ik = (fk >> v) & 1u;
      const bool im = kTwo && ((gm.piece(q) >> v) & 1u);
      if (kInner == kDone && ((gm.piece(q) >> v) & 1u)) continue;
      x[v] = exp_diff(x[v], ik ? bmax : ib ? mb : im ? mm : ma);       // keys outside the row hold -inf
      if (im) vm += x[v];
      if ((fa >> v) & 1u) va += x[v];
      if (ib) vb += x[v];
      if (ik) bsum += x[v];
    }
    xr.put(at, x);
  }
  elm = exp_diff(elm, bmax);
  elm2 = exp_diff(elm2, bmax);
  bsum = warp_sum(bsum);
  const float binv = (guards && bsum < 0.5f) ? 0.f : 1.f / bsum;
  float da, db;
  lg.reduce<false>(va, vb, da, db, closed);
  // scale of a non-bucket key: its landmark's weight over its group's sum (0 only for a group without keys)
  auto inv_den = [&](int c, float den) -> float {
    return (c >= G || (guards && den < 0.5f) || den == 0.f) ? 0.f : 1.f / den;
  };
  const float ia = inv_den(ca, da), ib = inv_den(cb, db);
  float wa = __shfl_sync(0xffffffffu, elm, lg.src_a), wb = __shfl_sync(0xffffffffu, elm, lg.src_b);
  wa = lg.has_a && ca < G ? wa * binv : 0.f;
  wb = lg.has_b && cb < G ? wb * binv : 0.f;
  const float im = inv_den(ca + 1, vm), wm = ca + 1 < G ? elm2 * binv : 0.f;
  return {binv, ia, ib, wa, wb, elm, im, wm, elm2};
}

template <typename T, bool kBackward, bool kCausal>
__device__ __noinline__ void grouped_softmax_crowded_row(const GsParams& p, int n_chunks, int64_t row, float* buf) {
  grouped_softmax_chunked_row<T, kBackward, kCausal>(p, n_chunks, row, buf);
}

template <typename T, bool kBackward, bool kCausal, int K>
__global__ void __launch_bounds__(kGsWarps * 32, K == 32 ? 8 : 6)
    grouped_softmax_lanes_kernel(const __grid_constant__ GsParams p, int n_chunks, int per_head_group, int per_warp) {
  extern __shared__ __align__(16) float gs_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const int head_groups = (p.H + per_head_group - 1) / per_head_group;
  const unsigned task = blockIdx.x * kGsWarps + warp;             // (batch row, group of heads, query)
  const int bg = (int)(task / (unsigned)p.Lq), i = (int)(task - (unsigned)bg * p.Lq);
  if (bg >= p.B * head_groups) return;
  const int b = bg / head_groups, h0 = (bg - b * head_groups) * per_head_group, h1 = min(h0 + per_head_group, p.H);
  const bool guards = p.guards != 0;
  const int G = p.max_groups, Lk = p.Lk;
  // scores, then exponentials (and the forward's results) in the first half of the warp's memory, gradients (and the
  // backward's results) in the second
  LaneRow xr{gs_smem + (size_t)warp * per_warp, lane};
  LaneRow gr{xr.buf + (kBackward ? per_warp >> 1 : 0), lane};
  const bool shared_masks = kCausal || ((p.ms[1] | p.ls[1] | p.hs[1]) == 0);
  const int pi = i + Lk - p.Lq;                         // causal: the last key this query sees
  int seen = Lk;                                        // keys whose scores are read
  if (kCausal) seen = pi + ((p.row_flags[b * p.row_flags_stride + pi] & 1u) ? 0 : 1);   // a landmark at pi itself is hidden

  auto row_of = [&](int h) { return ((int64_t)b * p.H + h) * p.Lq + i; };
  auto lead_of = [&](int h) { return (int)((row_of(h) * Lk) & 3); };

  using Mask = Bits<K>;
  // what follows from the masks, kept while they, the lead and the number of pieces stay the same
  Mask last, bk, act, ga, gb, gm;   // last section, bucket, all but merely hidden keys, members of the lane's groups
  unsigned owners = 0;              // lanes with a landmark
  int n4 = 0, lead = -1, c0 = 0, nlm = 0, lm_slot = 0, lm2_slot = 0;     // c0: the lane's first piece
  bool crowded = false, two = false, lm_last = false, lm2_last = false;      // lm_last: the landmark is in the last section too
  unsigned later = 0;               // heads whose row has three landmarks in one lane
  for (int h = h0; h < h1; ++h) {
    const int64_t row = row_of(h);
    const int lead_h = lead_of(h);
    int n = lead_h + seen;          // keys that the row is worked on for
    int n4_h = max((n + 127) >> 7, 1);
    // Where the row's extent does not depend on its scores the masks come first: a crowded row is then not even read here.
    auto stage_scores = [&]() {
      xr.stage<T>(reinterpret_cast<const T*>(p.x) + b * p.xs[0] + h * p.xs[1] + i * p.xs[2] - lead_h, lead_h, lead_h + seen,
                  max((lead_h + seen + 127) >> 7, 1), -INFINITY);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
    };
    const bool by_scores = !kCausal && guards;
    if (by_scores) stage_scores();
    if (!kCausal && guards) {
      // scores of -inf at the row's end weigh nothing, whatever their flags say, and neither does a landmark among them
      int top = 0;
#pragma unroll 1
      for (int c = lane; c < 32 * n4_h; c += 32) {
        float e[4];
        xr.get<T>(xr.slot(c), e);
        if (e[0] != -INFINITY || e[1] != -INFINITY || e[2] != -INFINITY || e[3] != -INFINITY) top = c + 1;
      }
      n = min(4 * __reduce_max_sync(0xffffffffu, top), n);
      n4_h = max((n + 127) >> 7, 1);
    }
    if (!shared_masks || n4_h != n4 || lead_h != lead) {
      n4 = n4_h;
      lead = lead_h;
      c0 = lane * n4;
      const int j0 = 4 * c0;
      Mask mem;
      const Mask in = Mask::low(lead + Lk - j0), before = Mask::low(lead - j0);
      if (kCausal) {
        causal_masks<K>(load_bits<K>(p.row_flags + b * p.row_flags_stride, 1, j0 - lead, n4, Lk), before, pi, lead, j0, mem, last,
                        act, bk);
      } else {
        mem = load_bits<K>(p.is_mem + b * p.ms[0] + h * p.ms[1] + i * p.ms[2], p.ms[3], j0 - lead, n4, Lk);
        last = load_bits<K>(p.last + b * p.ls[0] + h * p.ls[1] + i * p.ls[2], p.ls[3], j0 - lead, n4, Lk);
        Mask hid = Mask::low(0);
        if (p.hidden != nullptr)
          hid = load_bits<K>(p.hidden + b * p.hs[0] + h * p.hs[1] + i * p.hs[2], p.hs[3], j0 - lead, n4, Lk);
        bk = Mask::zip([&](int w) { return mem.w[w] | last.w[w] | hid.w[w] | ~in.w[w] | before.w[w]; });
        act = Mask::zip([&](int w) { return ~bk.w[w] | mem.w[w] | last.w[w]; });
      }
      nlm = mem.count();
      crowded = __any_sync(0xffffffffu, nlm > 2);
      two = __any_sync(0xffffffffu, nlm == 2);
      owners = __ballot_sync(0xffffffffu, nlm != 0);
      // the lane's landmarks t <= t2: group a in front of the first, group b behind the last, a group of its own between them
      const int t = mem.first(), t2 = nlm ? mem.top() : K;
      const Mask upto = Mask::low(t), upto2 = Mask::low(t2);
      ga = Mask::zip([&](int w) { return ~bk.w[w] & upto.w[w]; });
      gb = Mask::zip([&](int w) { return ~bk.w[w] & ~upto2.w[w]; });
      gm = Mask::zip([&](int w) { return ~bk.w[w] & ~upto.w[w] & upto2.w[w]; });
      lm_last = nlm != 0 && ((last.piece(t >> 2) >> (t & 3)) & 1u);
      lm2_last = nlm != 0 && ((last.piece(t2 >> 2) >> (t2 & 3)) & 1u);
      lm_slot = xr.slot(min(c0 + (t >> 2), 32 * n4 - 1)) * 4 + (t & 3);
      lm2_slot = xr.slot(min(c0 + (t2 >> 2), 32 * n4 - 1)) * 4 + (t2 & 3);
    }
    if (crowded) {
      later |= 1u << (h - h0);
      continue;
    }
    if (!by_scores) stage_scores();
    if (kBackward) gr.stage<float>(p.gprobs + row * Lk - lead, lead, n, n4, 0.f);
    auto finish = [&](auto two_in_a_lane) {
    constexpr bool kTwo = decltype(two_in_a_lane)::value;
    asm volatile("" : "+r"(owners));                     // recomputed for every head rather than kept in registers
    const LaneGroups lg(lane, owners);
    int ca = __popc(owners & ((1u << lane) - 1u)), n_groups = __popc(owners);
    if constexpr (kTwo) {                               // landmarks in front of the lane
      int inc = nlm;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
      }
      ca = inc - nlm;
      n_groups = __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0 && n_groups >= G && p.status != nullptr) atomicCAS(p.status, 0, kErrSoftmaxGroups);

    const LaneWeights lw = lane_weights<T, K, kTwo ? kOne : kNone>(xr, c0, n4, lm_slot, ga, gb, bk, lg, ca, G, guards, gm, lm2_slot, nlm);
    const float binv = lw.binv, ia = lw.ia, ib = lw.ib, wa = lw.wa, elm = lw.elm;
    float va, vb, closed;
    const float sa = ia * wa, sb = ib * lw.wb, sm = lw.im * lw.wm;

    if (!kBackward) {
      const float none = guards ? 0.f : binv * 0.f;     // bucket keys outside the last section (NaN if binv is not finite)
      float last_total = 0.f;
#pragma unroll 1
      for (int q = 0; q < n4; ++q) {
        const uint32_t fa = ga.piece(q), fb = gb.piece(q), fl = last.piece(q);
        const int at = xr.slot(c0 + q);
        float x[4];
        xr.get<float>(at, x);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const bool il = (fl >> v) & 1u;
          x[v] *= il ? binv : (fb >> v) & 1u ? sb : (kTwo && ((gm.piece(q) >> v) & 1u)) ? sm : (fa >> v) & 1u ? sa : none;
          if (il) last_total += x[v];
        }
        xr.put(at, x);
      }
      if (p.group_prob != nullptr) {
        last_total = warp_sum(last_total);
        float* gp = p.group_prob + row * p.max_mem_cnt;
        for (int g = n_groups + lane; g < p.max_mem_cnt - 1; g += 32) gp[g] = 0.f;
        if (lg.own && ca < p.max_mem_cnt - 1) gp[ca] = wa;
        if (kTwo && nlm == 2 && ca + 1 < p.max_mem_cnt - 1) gp[ca + 1] = lw.wm;
        if (lane == 0) gp[p.max_mem_cnt - 1] = last_total;
      }
      __syncwarp();
      xr.write<float>(p.probs + row * Lk - lead, lead, lead + Lk, n4);
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      // pass 3: c_g = sum_j inner_j * grad_j per group, total = sum_j P_j * grad_j over the row
      float lsum = 0.f, vm = 0.f;
      va = vb = 0.f;
#pragma unroll 1
      for (int q = 0; q < n4; ++q) {
        const uint32_t fa = ga.piece(q), fb = gb.piece(q), fl = last.piece(q);
        const int at = xr.slot(c0 + q);
        float x[4], g[4];
        xr.get<float>(at, x);
        gr.get<float>(at, g);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          if ((fa >> v) & 1u) va = fmaf(x[v], g[v], va);
          if ((fb >> v) & 1u) vb = fmaf(x[v], g[v], vb);
          if ((fl >> v) & 1u) lsum = fmaf(x[v], g[v], lsum);
          if (kTwo && ((gm.piece(q) >> v) & 1u)) vm = fmaf(x[v], g[v], vm);
        }
      }
      float c_a, c_b;
      lg.reduce<false>(va, vb, c_a, c_b, closed);
      c_a *= ia;
      c_b *= ib;
      const float c_m = kTwo ? vm * lw.im : 0.f;
      const float total = warp_sum((lg.own ? closed * ia * wa : 0.f) + (kTwo && nlm == 2 ? c_m * lw.wm : 0.f) + lsum * binv);
      // pass 4: last section P_j * (g_j - total), group member P_j * (g_j - c_g); a landmark P_j * (c_g - total), plus g_j
      // if it is in the last section too
      const float lm_g = lm_last ? gr.buf[lm_slot] : 0.f;
      const float lm2_g = kTwo && lm2_last ? gr.buf[lm2_slot] : 0.f;
#pragma unroll 1
      for (int q = 0; q < n4; ++q) {
        const uint32_t fb = gb.piece(q), fl = last.piece(q), fx = act.piece(q);
        const int at = xr.slot(c0 + q);
        float x[4], g[4];
        xr.get<float>(at, x);
        gr.get<float>(at, g);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const bool ib = (fb >> v) & 1u, il = (fl >> v) & 1u;
          const bool im = kTwo && ((gm.piece(q) >> v) & 1u);
          const float s = il ? binv : ib ? sb : im ? sm : sa, sub = il ? total : ib ? c_b : im ? c_m : c_a;
          x[v] = (fx >> v) & 1u ? x[v] * s * (g[v] - sub) : 0.f;
        }
        gr.put(at, x);                                  // the lane's own pieces, read just before
      }
      if (lg.own) gr.buf[lm_slot] = elm * binv * (lm_g + c_a - total);
      if (kTwo && nlm == 2) gr.buf[lm2_slot] = lw.elm2 * binv * (lm2_g + c_m - total);
      __syncwarp();
      if (p.gx_as_x) gr.write<T>(reinterpret_cast<T*>(p.gx) + row * Lk - lead, lead, lead + Lk, n4);
      else gr.write<float>(reinterpret_cast<float*>(p.gx) + row * Lk - lead, lead, lead + Lk, n4);
    }
    };
    if (two) finish(std::true_type{});
    else finish(std::false_type{});
    __syncwarp();                                       // the results have been read
  }
  for (; later; later &= later - 1) {
    grouped_softmax_crowded_row<T, kBackward, kCausal>(p, n_chunks, row_of(h0 + __ffs(later) - 1), xr.buf);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------------------------
// Attention rows behind a retrieved prefix, up to the prefix' values: local scores, grouped softmax over [prefix | chunk] and
// the local part of probabilities times values (the cache branch of CausalSelfAttention.forward,
// lm_benchmark/models/landmark.py:196-243).  One CTA per 16 queries of a head, its rows in shared memory from the scores to the
// probabilities; scores and local output as mma.sync tiles, rounded where the tensor formulation rounds (the product, the
// scaling, the probabilities, the output).  Written out: the prefix' probabilities (fp32) and the local output.
// Bound by latency: 5 MB of operands and 80 MB of prefix logits and probabilities at B16 H8 T255 P204; library products, scaling,
// concatenation, softmax and casts as kernels of their own took 167 us, this one takes 98 us (32 rows a CTA, half as many warps an SM: 130).
// ---------------------------------------------------------------------------------------------------------------
constexpr int kCrRows = 16, kCrTiles = kCrRows / 16, kCrThreads = 256, kCrVPitch = 136;
constexpr size_t kCrMaxSmem = 224 * 1024;

struct CrParams {
  const void *q, *k, *v;
  int64_t qs[3], ks[3], vs[3];
  const void* prefix;                   // [B, H, T, P] dense logits
  const uint8_t* flags; int64_t flags_stride;      // [B, P + T]
  float* probs;                         // [B, H, T, P]
  void* out;                            // [B, H, T, 128]
  int H, T, P, G;
  float scale;
  int* status;
};
__host__ __device__ constexpr int cr_pieces(int W) { return (W + 10 + 127) / 128; }      // lead, and scores are computed for eight keys at a time
__host__ __device__ constexpr int cr_prob_pitch(int T) { return ((T + 15) & ~15) + 8; }
// The rows of scores; once their probabilities are written the value tiles take their place, which leaves room for a fourth CTA on
// an SM (62.7 -> 45.3 KB at B16 H8 T255 P204: the kernel 111 -> 98.4 us).
__host__ __device__ constexpr size_t cr_rows_bytes(int W) {
  const size_t rows = sizeof(float) * kCrRows * 144 * (size_t)cr_pieces(W), values = 2 * 64 * kCrVPitch;
  return rows > values ? rows : values;
}
__host__ __device__ constexpr size_t cr_smem(int T, int P) { return cr_rows_bytes(P + T) + 2 * (size_t)kCrRows * cr_prob_pitch(T); }

// A row in which landmarks share a lane (cached rows).  The groups between a lane's landmarks lie in the lane: it works them out first,
// one after the other, as far as exponential over sum; the rest of the row goes the way of the other rows, and the last pass, back to
// front, gives the inner groups their landmarks' weights.  Probabilities replace the scores.
// Every key is looked at a fixed number of times, however many landmarks there are.  The call (us; with the scores and the softmax as
// tensor operations / a walk of the whole row for every group / this): B16 H8 T255 P204, a landmark every 8 keys 468 / 2150 / 388, every
// 2 552 / 6954 / 404; B4 H8 T512 P512, every 16 505 / 4797 / 563, every 2 581 / 29 170 / 591.
template <int K>
__device__ __noinline__ void crowded_smem_row(LaneRow xr, int c0, int n4, Bits<K> mem, Bits<K> last, Bits<K> bk, unsigned owners, int G) {
  const int nlm = mem.count();
  int ca = nlm;                                         // landmarks in front of the lane
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, ca, o);
    if (xr.lane >= o) ca += u;
  }
  ca -= nlm;
  const int t = mem.first(), t2 = nlm ? mem.top() : K;
  const Bits<K> upto = Bits<K>::low(t), upto2 = Bits<K>::low(t2);
  const Bits<K> ga = Bits<K>::zip([&](int w) { return ~bk.w[w] & upto.w[w]; });
  const Bits<K> gb = Bits<K>::zip([&](int w) { return ~bk.w[w] & ~upto2.w[w]; });
  const Bits<K> gm = Bits<K>::zip([&](int w) { return ~bk.w[w] & ~upto.w[w] & upto2.w[w]; });
  auto at = [&](int v) { return xr.slot(c0 + (v >> 2)) * 4 + (v & 3); };
  auto bit = [](const Bits<K>& m, int v) { return (m.piece(v >> 2) >> (v & 3)) & 1u; };
  if (nlm > 1) {
    for (int s = t, c = ca + 1; s < t2; ++c) {          // the group behind the landmark at s
      float mx = -INFINITY, den = 0.f;
      int e = s + 1;
      for (; !bit(mem, e); ++e)
        if (bit(gm, e)) mx = fmaxf(mx, xr.buf[at(e)]);
      if (isinf(mx)) mx = 0.f;
      for (int v = s + 1; v < e; ++v)
        if (bit(gm, v)) {
          const float x = exp_diff(xr.buf[at(v)], mx);
          xr.buf[at(v)] = x;
          den += x;
        }
      const float inv = c >= G || den < 0.5f ? 0.f : 1.f / den;
      for (int v = s + 1; v < e; ++v)
        if (bit(gm, v)) xr.buf[at(v)] *= inv;
      s = e;
    }
  }
  const LaneGroups lg(xr.lane, owners);
  const int lm_slot = xr.slot(min(c0 + (t >> 2), 32 * n4 - 1)) * 4 + (t & 3);
  const LaneWeights lw = lane_weights<float, K, kDone>(xr, c0, n4, lm_slot, ga, gb, bk, lg, ca, G, true, gm, 0, nlm);
  const float sa = lw.ia * lw.wa, sb = lw.ib * lw.wb;
  float w = 0.f;                                        // of the landmark passed last
  int c = ca + nlm;
#pragma unroll 1
  for (int q = n4 - 1; q >= 0; --q) {
    const uint32_t fa = ga.piece(q), fb = gb.piece(q), fm = gm.piece(q), fl = last.piece(q), lm = mem.piece(q);
    float x[4];
    xr.get<float>(xr.slot(c0 + q), x);
#pragma unroll
    for (int v = 3; v >= 0; --v) {
      if ((lm >> v) & 1u) w = --c < G ? x[v] * lw.binv : 0.f;
      x[v] *= (fl >> v) & 1u ? lw.binv : (fb >> v) & 1u ? sb : (fm >> v) & 1u ? w : (fa >> v) & 1u ? sa : 0.f;
    }
    xr.put(xr.slot(c0 + q), x);
  }
}

template <typename T, int K>
__global__ void __launch_bounds__(kCrThreads, K == 32 ? 4 : 2) cached_rows_kernel(const __grid_constant__ CrParams p) {
  extern __shared__ __align__(16) float gs_smem[];
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
  const int bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H;
  const int q0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * kCrRows;             // longest rows first
  const int W = p.P + p.T, n4max = cr_pieces(W), row_floats = 144 * n4max, pitch = cr_prob_pitch(p.T);
  const int lead = (4 - (p.P & 3)) & 3;                                       // the chunk's first key starts a piece
  T* pb = reinterpret_cast<T*>(gs_smem + cr_rows_bytes(W) / sizeof(float));   // [16][pitch] local probabilities
  T* vt = reinterpret_cast<T*>(gs_smem);                                      // [64][kCrVPitch] values, when the scores are done with
  const T* q = reinterpret_cast<const T*>(p.q) + b * p.qs[0] + h * p.qs[1];
  const T* k = reinterpret_cast<const T*>(p.k) + b * p.ks[0] + h * p.ks[1];
  const T* v = reinterpret_cast<const T*>(p.v) + b * p.vs[0] + h * p.vs[1];
  const int n_keys = min(q0 + kCrRows, p.T);                                  // keys that any of the rows sees

  // ---- local scores
  {
    uint4 a[kCrTiles][4], a8[kCrTiles][4];
#pragma unroll
    for (int m = 0; m < kCrTiles; ++m)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        a[m][c] = *reinterpret_cast<const uint4*>(q + (int64_t)min(q0 + 16 * m + g, p.T - 1) * p.qs[2] + 32 * c + 8 * t4);
        a8[m][c] = *reinterpret_cast<const uint4*>(q + (int64_t)min(q0 + 16 * m + 8 + g, p.T - 1) * p.qs[2] + 32 * c + 8 * t4);
      }
    for (int nb = warp; nb * 8 < n_keys; nb += kCrThreads / 32) {
      const T* kr = k + (int64_t)min(nb * 8 + g, p.T - 1) * p.ks[2] + 8 * t4;
      uint4 kv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) kv[c] = *reinterpret_cast<const uint4*>(kr + 32 * c);
#pragma unroll
      for (int m = 0; m < kCrTiles; ++m) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) mma_chunk<T>(acc, a[m][c], a8[m][c], kv[c]);
        const int e = lead + p.P + nb * 8 + 2 * t4;                           // even: both keys in one piece
        const int at = LaneRow::slot(e >> 2) * 4 + (e & 3);
        float* s = gs_smem + (16 * m + g) * row_floats + at;
        *reinterpret_cast<float2*>(s) = make_float2(rnd<T>(rnd<T>(acc[0]) * p.scale), rnd<T>(rnd<T>(acc[1]) * p.scale));
        *reinterpret_cast<float2*>(s + 8 * row_floats) =
            make_float2(rnd<T>(rnd<T>(acc[2]) * p.scale), rnd<T>(rnd<T>(acc[3]) * p.scale));
      }
    }
  }
  __syncthreads();

  // ---- softmax: a warp's rows one after the other
  for (int r = warp; r < kCrRows; r += kCrThreads / 32) {
    LaneRow xr{gs_smem + r * row_floats, lane};
    T* prow = pb + r * pitch;
    const int i = q0 + r;
    if (i >= p.T) {
      for (int j = lane; j < pitch; j += 32) prow[j] = from_f32<T>(0.f);
      continue;
    }
    const uint8_t* fl = p.flags + b * p.flags_stride;
    const int pi = p.P + i, n = lead + pi + ((fl[pi] & 1u) ? 0 : 1), n4 = max((n + 127) >> 7, 1);
    const T* pre = reinterpret_cast<const T*>(p.prefix) + ((int64_t)bh * p.T + i) * p.P;
    if (lane < lead) xr.buf[lane] = -INFINITY;
    for (int e = n + lane; e < 128 * n4; e += 32) xr.buf[LaneRow::slot(e >> 2) * 4 + (e & 3)] = -INFINITY;
    for (int c = lane; c < p.P; c += 32) {
      const int e = lead + c;
      if (e < n) xr.buf[LaneRow::slot(e >> 2) * 4 + (e & 3)] = to_f32(pre[c]);
    }
    __syncwarp();
    using Mask = Bits<K>;
    const int c0 = lane * n4, j0 = 4 * c0;
    Mask mem, last, act, bk;
    causal_masks<K>(load_bits<K>(fl, 1, j0 - lead, n4, W), Mask::low(lead - j0), pi, lead, j0, mem, last, act, bk);
    const int nlm = mem.count();
    const unsigned owners = __ballot_sync(0xffffffffu, nlm != 0);
    const int n_groups = __reduce_add_sync(0xffffffffu, nlm);
    if (lane == 0 && n_groups >= p.G && p.status != nullptr) atomicCAS(p.status, 0, kErrSoftmaxGroups);
    if (__any_sync(0xffffffffu, nlm > 1)) {
      crowded_smem_row<K>(xr, c0, n4, mem, last, bk, owners, p.G);
    } else {
      const LaneGroups lg(lane, owners);
      const int t = mem.first();
      const Mask upto = Mask::low(t);
      const Mask ga = Mask::zip([&](int w) { return ~bk.w[w] & upto.w[w]; });
      const Mask gb = Mask::zip([&](int w) { return ~bk.w[w] & ~upto.w[w]; });
      const int lm_slot = xr.slot(min(c0 + (t >> 2), 32 * n4 - 1)) * 4 + (t & 3);
      const LaneWeights lw =
          lane_weights<float, K, kNone>(xr, c0, n4, lm_slot, ga, gb, bk, lg, __popc(owners & ((1u << lane) - 1u)), p.G, true);
      const float sa = lw.ia * lw.wa, sb = lw.ib * lw.wb;
#pragma unroll 1
      for (int c = 0; c < n4; ++c) {
        const uint32_t fa = ga.piece(c), fb = gb.piece(c), fl2 = last.piece(c);
        const int at = xr.slot(c0 + c);
        float x[4];
        xr.get<float>(at, x);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          x[u] *= (fl2 >> u) & 1u ? lw.binv : (fb >> u) & 1u ? sb : (fa >> u) & 1u ? sa : 0.f;
        xr.put(at, x);
      }
    }
    __syncwarp();
    float* pr = p.probs + ((int64_t)bh * p.T + i) * p.P;
    for (int c = lane; c < p.P; c += 32) {
      const int e = lead + c;
      pr[c] = e < 128 * n4 ? xr.buf[LaneRow::slot(e >> 2) * 4 + (e & 3)] : 0.f;
    }
    for (int j = lane; j < pitch; j += 32) {
      const int e = lead + p.P + j;
      prow[j] = from_f32<T>(j < p.T && e < n ? xr.buf[LaneRow::slot(e >> 2) * 4 + (e & 3)] : 0.f);
    }
  }

  // ---- local output: warp w has features 16 w .. 16 w + 15 of all rows
  float acc[kCrTiles][2][4] = {};
  for (int j0 = 0; j0 < n_keys; j0 += 64) {
    __syncthreads();                                    // probabilities written, scores done with; the tile before has been read
    for (int e = tid; e < 64 * 16; e += kCrThreads) {
      const int r = e >> 4, c = (e & 15) * 8;
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (j0 + r < n_keys) x = *reinterpret_cast<const uint4*>(v + (int64_t)(j0 + r) * p.vs[2] + c);
      *reinterpret_cast<uint4*>(vt + r * kCrVPitch + c) = x;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 64; kk += 16) {
      if (j0 + kk >= n_keys) break;
      uint32_t bf[4], af[kCrTiles][4];
      // values of keys kk .. kk + 15, features 16 warp .. + 15: two 16 x 8 B fragments
      ldmatrix_x4_trans(bf, vt + (kk + (lane & 15)) * kCrVPitch + 16 * warp + 8 * (lane >> 4));
#pragma unroll
      for (int m = 0; m < kCrTiles; ++m) ldmatrix_x4(af[m], pb + (16 * m + (lane & 15)) * pitch + j0 + kk + 8 * (lane >> 4));
#pragma unroll
      for (int m = 0; m < kCrTiles; ++m) {
        mma16<T>(acc[m][0], af[m][0], af[m][1], af[m][2], af[m][3], bf[0], bf[1]);
        mma16<T>(acc[m][1], af[m][0], af[m][1], af[m][2], af[m][3], bf[2], bf[3]);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < kCrTiles; ++m)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int i = q0 + 16 * m + 8 * half + g;
      if (i >= p.T) continue;
      T* o = reinterpret_cast<T*>(p.out) + ((int64_t)bh * p.T + i) * 128 + 16 * warp + 2 * t4;
#pragma unroll
      for (int nn = 0; nn < 2; ++nn) {
        o[8 * nn] = from_f32<T>(acc[m][nn][2 * half]);
        o[8 * nn + 1] = from_f32<T>(acc[m][nn][2 * half + 1]);
      }
    }
}

static size_t fast_smem_bytes(int Lk, int max_groups) {
  const size_t n_chunks = (size_t)(Lk + kFastChunk - 1) / kFastChunk;
  return sizeof(float) * kGsWarps * (n_chunks * (kFastChunk + 64) + 4 * (size_t)max_groups);
}

template <bool kBackward>
int launch(const GsParams& p, int dtype, cudaStream_t st) {
  const int64_t rows = (int64_t)p.B * p.H * p.Lq;
  if (rows == 0 || p.Lk == 0) return LMK_OK;
  GsParams& pw = const_cast<GsParams&>(p);
  pw.status = device_status_word();
  unsigned grid = (unsigned)((rows + kGsWarps - 1) / kGsWarps);
  const bool fast = p.Lk <= kFastMaxLk && fast_smem_bytes(p.Lk, p.max_groups) <= kFastMaxSmem;
  if (p.causal && !fast)
    return fail(LMK_ERR_UNSUPPORTED, "grouped_softmax_causal: rows of %d keys with %d groups do not fit the row kernel "
                                     "(at most %d keys); build the masks and use lmk_grouped_softmax_fwd", p.Lk,
                p.max_groups, kFastMaxLk);
  const int n_chunks = (p.Lk + kFastChunk - 1) / kFastChunk;
  size_t smem = fast ? fast_smem_bytes(p.Lk, p.max_groups) : sizeof(float) * 4 * (size_t)p.max_groups * kGsWarps;
  // pieces a lane of the longest row, counted with its lead (rows of a multiple of four keys have none)
  const int n4 = (p.Lk + (p.Lk % 4 ? 3 : 0) + 127) / 128;
  const bool lanes = fast && n4 <= kLaneMaxPieces && rows < (1LL << 31);
  // Heads a warp takes in turn: as many as leave every SM three rounds of
  // warps (causal rows differ in length), eight at most.
  int per_group = 1, per_warp = 0;
  if (lanes) {
    int n_sm = 0;
    const int rc = sm_count(&n_sm);
    if (rc != LMK_OK) return rc;
    const int64_t resident = (int64_t)n_sm * kGsWarps * 8;
    per_group = (int)std::min<int64_t>(std::max<int64_t>(rows / (3 * resident), 1), std::min(p.H, 8));
    const int groups = (p.H + per_group - 1) / per_group;
    per_group = (p.H + groups - 1) / groups;
    grid = (unsigned)(((int64_t)p.B * groups * p.Lq + kGsWarps - 1) / kGsWarps);
    // shared memory of a warp: two rows, or what the chunked form of a crowded row takes
    per_warp = ((int)(smem / sizeof(float) / kGsWarps) + 7) & ~7;
    per_warp = std::max(per_warp, (kBackward ? 2 : 1) * 144 * n4);
    smem = sizeof(float) * (size_t)per_warp * kGsWarps;
  }
#define LMK_GS_RUN(kernel, ...)                                                                              \
  do {                                                                                                       \
    LMK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));          \
    kernel<<<grid, kGsWarps * 32, smem, st>>>(__VA_ARGS__);                                                  \
  } while (0)
#define LMK_GS_OVERLAPPED(kernel, ...)                                                                       \
  do {                                                                                                       \
    LMK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));          \
    LMK_CUDA(launch_overlapped(kernel, dim3(grid), dim3(kGsWarps * 32), smem, st, __VA_ARGS__));             \
  } while (0)
#define LMK_GS_LANES(T, causal)                                                                              \
  do {                                                                                                       \
    if (n4 <= 8) LMK_GS_OVERLAPPED((grouped_softmax_lanes_kernel<T, kBackward, causal, 32>), p, n_chunks, per_group, per_warp);   \
    else LMK_GS_OVERLAPPED((grouped_softmax_lanes_kernel<T, kBackward, causal, 64>), p, n_chunks, per_group, per_warp);                \
  } while (0)
#define LMK_GS_LAUNCH(T)                                                                                     \
  do {                                                                                                       \
    if (lanes && p.causal) LMK_GS_LANES(T, true);                                                            \
    else if (lanes) LMK_GS_LANES(T, false);                                                                  \
    else if (fast && p.causal) LMK_GS_RUN((grouped_softmax_rows_kernel<T, kBackward, true>), p, n_chunks);   \
    else if (fast) LMK_GS_RUN((grouped_softmax_rows_kernel<T, kBackward, false>), p, n_chunks);              \
    else LMK_GS_RUN((grouped_softmax_kernel<T, kBackward>), p);                                              \
  } while (0)
  if (dtype == LMK_F32) LMK_GS_LAUNCH(float);
  else if (dtype == LMK_F16) LMK_GS_LAUNCH(__half);
  else LMK_GS_LAUNCH(__nv_bfloat16);
#undef LMK_GS_LANES
#undef LMK_GS_OVERLAPPED
#undef LMK_GS_RUN
#undef LMK_GS_LAUNCH
  LMK_CUDA(cudaGetLastError());
  return LMK_OK;
}

int fill(GsParams& p, const void* x, const int64_t* xs, const uint8_t* is_mem, const int64_t* ms,
         const uint8_t* last, const int64_t* ls, const uint8_t* hidden, const int64_t* hs, int B, int H, int Lq,
         int Lk, int dtype, int guards, int max_groups) {
  LMK_CHECK_ARG(x && is_mem && last && xs && ms && ls, "grouped_softmax: null pointer");
  LMK_CHECK_ARG(!hidden || hs, "grouped_softmax: hidden mask without strides");
  LMK_CHECK_ARG(B >= 0 && H >= 0 && Lq >= 0 && Lk >= 0, "grouped_softmax: negative dimension");
  LMK_CHECK_ARG(dtype == LMK_F32 || dtype == LMK_F16 || dtype == LMK_BF16, "grouped_softmax: bad dtype %d", dtype);
  LMK_CHECK_ARG(max_groups >= 1 && max_groups <= 2048, "grouped_softmax: max_groups %d outside [1, 2048]", max_groups);
  p.x = x;
  p.is_mem = is_mem; p.last = last; p.hidden = hidden;
  for (int i = 0; i < 3; ++i) p.xs[i] = xs[i];
  for (int i = 0; i < 4; ++i) {
    p.ms[i] = ms[i];
    p.ls[i] = ls[i];
    p.hs[i] = hidden ? hs[i] : 0;
  }
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk; p.guards = guards; p.max_groups = max_groups;
  return LMK_OK;
}

}  // namespace
}  // namespace lmk

extern "C" int lmk_grouped_softmax_fwd(const void* x, const int64_t x_strides[3], const uint8_t* is_mem,
                                       const int64_t is_mem_strides[4], const uint8_t* last_section,
                                       const int64_t last_strides[4], const uint8_t* hidden,
                                       const int64_t hidden_strides[4], float* probs, float* group_prob,
                                       int max_mem_cnt, int B, int H, int Lq, int Lk, int dtype, int guards,
                                       int max_groups, void* stream) {
  lmk::GsParams p{};
  int rc = lmk::fill(p, x, x_strides, is_mem, is_mem_strides, last_section, last_strides, hidden, hidden_strides,
                     B, H, Lq, Lk, dtype, guards, max_groups);
  if (rc != LMK_OK) return rc;
  LMK_CHECK_ARG(probs != nullptr, "grouped_softmax_fwd: probs is null");
  LMK_CHECK_ARG(group_prob == nullptr || max_mem_cnt >= 2, "grouped_softmax_fwd: max_mem_cnt must be >= 2");
  p.probs = probs;
  p.group_prob = group_prob;
  p.max_mem_cnt = max_mem_cnt;
  return lmk::launch<false>(p, dtype, (cudaStream_t)stream);
}

static int run_bwd(const void* x, const int64_t* xs, const uint8_t* is_mem, const int64_t* ms, const uint8_t* last,
                   const int64_t* ls, const uint8_t* hidden, const int64_t* hs, const float* grad_probs, void* grad_x,
                   int typed, int B, int H, int Lq, int Lk, int dtype, int guards, int max_groups, void* stream) {
  lmk::GsParams p{};
  int rc = lmk::fill(p, x, xs, is_mem, ms, last, ls, hidden, hs, B, H, Lq, Lk, dtype, guards, max_groups);
  if (rc != LMK_OK) return rc;
  LMK_CHECK_ARG(grad_probs && grad_x, "grouped_softmax_bwd: null gradient pointer");
  p.gprobs = grad_probs;
  p.gx = grad_x;
  p.gx_as_x = typed && dtype != LMK_F32;
  return lmk::launch<true>(p, dtype, (cudaStream_t)stream);
}

extern "C" int lmk_grouped_softmax_bwd(const void* x, const int64_t x_strides[3], const uint8_t* is_mem,
                                       const int64_t is_mem_strides[4], const uint8_t* last_section,
                                       const int64_t last_strides[4], const uint8_t* hidden,
                                       const int64_t hidden_strides[4], const float* grad_probs, float* grad_x,
                                       int B, int H, int Lq, int Lk, int dtype, int guards, int max_groups,
                                       void* stream) {
  return run_bwd(x, x_strides, is_mem, is_mem_strides, last_section, last_strides, hidden, hidden_strides, grad_probs,
                 grad_x, 0, B, H, Lq, Lk, dtype, guards, max_groups, stream);
}

extern "C" int lmk_grouped_softmax_bwd_typed(const void* x, const int64_t x_strides[3], const uint8_t* is_mem,
                                             const int64_t is_mem_strides[4], const uint8_t* last_section,
                                             const int64_t last_strides[4], const uint8_t* hidden,
                                             const int64_t hidden_strides[4], const float* grad_probs, void* grad_x,
                                             int B, int H, int Lq, int Lk, int dtype, int guards, int max_groups,
                                             void* stream) {
  return run_bwd(x, x_strides, is_mem, is_mem_strides, last_section, last_strides, hidden, hidden_strides, grad_probs,
                 grad_x, 1, B, H, Lq, Lk, dtype, guards, max_groups, stream);
}

// Mask block + grouped softmax of the lm_benchmark call site (lm_benchmark/models/landmark.py:210-232) from one flag
// per (batch row, key): query i sees keys 0 .. i + Lk - Lq; hidden scores count as -inf.
static int fill_causal(lmk::GsParams& p, const void* x, const int64_t* xs, const uint8_t* is_mem_row, int64_t row_stride,
                       int B, int H, int Lq, int Lk, int dtype, int max_groups) {
  LMK_CHECK_ARG(x && xs && is_mem_row, "grouped_softmax_causal: null pointer");
  LMK_CHECK_ARG(B >= 0 && H >= 0 && Lq >= 0 && Lk >= Lq, "grouped_softmax_causal: need Lk >= Lq >= 0");
  LMK_CHECK_ARG(dtype == LMK_F32 || dtype == LMK_F16 || dtype == LMK_BF16, "grouped_softmax_causal: bad dtype %d", dtype);
  LMK_CHECK_ARG(max_groups >= 1 && max_groups <= 2048, "grouped_softmax_causal: max_groups %d outside [1, 2048]", max_groups);
  p.x = x;
  for (int i = 0; i < 3; ++i) p.xs[i] = xs[i];
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk; p.guards = 1; p.max_groups = max_groups;
  p.row_flags = is_mem_row; p.row_flags_stride = row_stride; p.causal = 1;
  return LMK_OK;
}

extern "C" int lmk_grouped_softmax_causal_fwd(const void* x, const int64_t x_strides[3], const uint8_t* is_mem_row,
                                              int64_t is_mem_stride, float* probs, int B, int H, int Lq, int Lk,
                                              int dtype, int max_groups, void* stream) {
  lmk::GsParams p{};
  int rc = fill_causal(p, x, x_strides, is_mem_row, is_mem_stride, B, H, Lq, Lk, dtype, max_groups);
  if (rc != LMK_OK) return rc;
  LMK_CHECK_ARG(probs != nullptr, "grouped_softmax_causal_fwd: probs is null");
  p.probs = probs;
  return lmk::launch<false>(p, dtype, (cudaStream_t)stream);
}

static int run_causal_bwd(const void* x, const int64_t* xs, const uint8_t* is_mem_row, int64_t is_mem_stride,
                          const float* grad_probs, void* grad_x, int typed, int B, int H, int Lq, int Lk, int dtype,
                          int max_groups, void* stream) {
  lmk::GsParams p{};
  int rc = fill_causal(p, x, xs, is_mem_row, is_mem_stride, B, H, Lq, Lk, dtype, max_groups);
  if (rc != LMK_OK) return rc;
  LMK_CHECK_ARG(grad_probs && grad_x, "grouped_softmax_causal_bwd: null gradient pointer");
  p.gprobs = grad_probs;
  p.gx = grad_x;
  p.gx_as_x = typed && dtype != LMK_F32;
  return lmk::launch<true>(p, dtype, (cudaStream_t)stream);
}

extern "C" int lmk_grouped_softmax_causal_bwd(const void* x, const int64_t x_strides[3], const uint8_t* is_mem_row,
                                              int64_t is_mem_stride, const float* grad_probs, float* grad_x, int B,
                                              int H, int Lq, int Lk, int dtype, int max_groups, void* stream) {
  return run_causal_bwd(x, x_strides, is_mem_row, is_mem_stride, grad_probs, grad_x, 0, B, H, Lq, Lk, dtype, max_groups,
                        stream);
}

extern "C" int lmk_grouped_softmax_causal_bwd_typed(const void* x, const int64_t x_strides[3], const uint8_t* is_mem_row,
                                                    int64_t is_mem_stride, const float* grad_probs, void* grad_x, int B,
                                                    int H, int Lq, int Lk, int dtype, int max_groups, void* stream) {
  return run_causal_bwd(x, x_strides, is_mem_row, is_mem_stride, grad_probs, grad_x, 1, B, H, Lq, Lk, dtype, max_groups,
                        stream);
}

extern "C" int lmk_cached_rows_supported(int D, int T, int P, int dtype) {
  return (dtype == LMK_BF16 || dtype == LMK_F16) && D == 128 && T >= 1 && P >= 1 && P + T <= 2000 &&
         lmk::cr_smem(T, P) + 2 * 64 * lmk::kCrVPitch <= lmk::kCrMaxSmem ? 1 : 0;      // as when the values had room of their own
}

extern "C" int lmk_cached_rows(const void* q, const void* k, const void* v, const int64_t q_strides[3], const int64_t k_strides[3],
                               const int64_t v_strides[3], const void* prefix_logits, const uint8_t* is_mem_row, int64_t is_mem_stride,
                               float* prefix_probs, void* out, int B, int H, int T, int P, int D, int max_groups, float sm_scale,
                               int dtype, void* stream) {
  using namespace lmk;
  LMK_CHECK_ARG(q && k && v && q_strides && k_strides && v_strides && prefix_logits && is_mem_row && prefix_probs && out,
                "cached_rows: null pointer");
  LMK_CHECK_ARG(B >= 1 && H >= 1 && (int64_t)B * H <= 65535, "cached_rows: bad sizes");
  LMK_CHECK_ARG(max_groups >= 1 && max_groups <= 2048, "cached_rows: max_groups %d outside [1, 2048]", max_groups);
  if (!lmk_cached_rows_supported(D, T, P, dtype))
    return fail(LMK_ERR_UNSUPPORTED, "cached_rows needs a 16-bit type, D=128 and 16 rows of P + T keys in shared memory "
                "(got dtype=%d D=%d T=%d P=%d)", dtype, D, T, P);
  LMK_CHECK_ARG((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) == 0, "cached_rows: pointers must be 16-byte aligned");
  CrParams p{};
  for (int i = 0; i < 3; ++i) {
    LMK_CHECK_ARG(q_strides[i] % 8 == 0 && k_strides[i] % 8 == 0 && v_strides[i] % 8 == 0,
                  "cached_rows: strides must be multiples of 8 elements");
    p.qs[i] = q_strides[i]; p.ks[i] = k_strides[i]; p.vs[i] = v_strides[i];
  }
  p.q = q; p.k = k; p.v = v; p.prefix = prefix_logits; p.flags = is_mem_row; p.flags_stride = is_mem_stride;
  p.probs = prefix_probs; p.out = out; p.H = H; p.T = T; p.P = P; p.G = max_groups; p.scale = sm_scale;
  p.status = device_status_word();
  const size_t smem = cr_smem(T, P);
  const bool wide = cr_pieces(P + T) > 8;
  const auto kernel = dtype == LMK_BF16 ? (wide ? cached_rows_kernel<__nv_bfloat16, 64> : cached_rows_kernel<__nv_bfloat16, 32>)
                                        : (wide ? cached_rows_kernel<__half, 64> : cached_rows_kernel<__half, 32>);
  LMK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  LMK_CUDA(launch_overlapped(kernel, dim3((T + kCrRows - 1) / kCrRows, B * H), dim3(kCrThreads), smem, (cudaStream_t)stream, p));
  return LMK_OK;
}
