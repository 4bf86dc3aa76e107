// 16-bit types two to a register: arithmetic with the roundings of the tensor formulation, and mma.sync m16n8k16 for contractions too
// small or too irregular for tcgen05 tiles.
#pragma once
#include <type_traits>
#include "common.cuh"

namespace lmk {
namespace {

template <typename T>
__device__ __forceinline__ float rnd(float x) { return to_f32(from_f32<T>(x)); }

// Two 16-bit values in one 32-bit register; every product and every sum is rounded to the type.
template <typename T> struct Pair16;
template <> struct Pair16<__nv_bfloat16> {
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  static __device__ __forceinline__ float2 f32(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
};
template <> struct Pair16<__half> {
  static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  static __device__ __forceinline__ float2 f32(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
};
template <> struct Pair16<float> {};      // named by kernels whose 16-bit branch is not compiled for fp32

// D += A B, m16n8k16.  A thread (g = lane / 4, t = lane % 4) holds the 16-byte vectors [32 c + 8 t, +8) of rows g and g + 8 of A
// and of row g of B^T; registers (0, 1) and (2, 3) of a vector serve as two k-steps.  A dot product does not depend on the
// order of the features, so the hardware's k index may stand for any four of them as long as both operands agree.
template <typename T>
__device__ __forceinline__ void mma16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <typename T>
__device__ __forceinline__ void mma_chunk(float (&d)[4], const uint4& a, const uint4& a8, const uint4& b) {
  mma16<T>(d, a.x, a8.x, a.y, a8.y, b.x, b.y);
  mma16<T>(d, a.z, a8.z, a.w, a8.w, b.z, b.w);
}

// Four 8 x 8 tiles of 16-bit values from shared memory, a lane's address being one of the 32 rows of 16 bytes.
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}

}  // namespace
}  // namespace lmk
