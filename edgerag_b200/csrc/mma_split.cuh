// Products of float operands on the bfloat16 tensor cores without rounding them to 16 bits.
//
// A float is the sum of three bfloat16 values exactly (8 bits of significand each), as long as the smallest piece is no
// denormal: x = a + b + c with a = bf16(x), b = bf16(x - a), c = bf16(x - a - b).  A product with a bfloat16 operand is then
// three products accumulated in float; one of two such operands takes the six whose terms are above 2^-24 of the result.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace erb {

__device__ __forceinline__ void ldmatrix4(uint32_t* r, const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldmatrix4t(uint32_t* r, const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// (the addresses of the first 16 lanes)
__device__ __forceinline__ void ldmatrix2t(uint32_t* r, const void* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The three pieces of two neighbouring floats, each piece as a pair of bfloat16.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t* piece) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
    piece[k] = *reinterpret_cast<const uint32_t*>(&b);
    x -= __uint_as_float(piece[k] << 16);
    y -= __uint_as_float(piece[k] & 0xffff0000u);
  }
}

// 16 bytes to shared memory without a register, zeros where the source is not to be read.
__device__ __forceinline__ void copy16_or_zero(void* dst, const void* src, bool real) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = real ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace erb
