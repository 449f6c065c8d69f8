// Two fp32 values in a 64-bit register and the packed arithmetic on them (one issue slot for two operations), and the unpacking
// of bf16 pairs: the kernels that give a thread neighbouring channels carry every fp32 quantity in this form.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace sb {

typedef unsigned long long f2;           // two packed fp32 values
__device__ __forceinline__ f2 f2_pack(float a, float b) { f2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ float2 f2_unpack(f2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) { f2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ f2 f2_bf(uint32_t w) { return f2_pack(lo_f(w), hi_f(w)); }
__device__ __forceinline__ uint32_t pack_bf2(f2 v) {
  const float2 t = f2_unpack(v);
  __nv_bfloat162 r = __floats2bfloat162_rn(t.x, t.y);
  return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
  __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&r);
}

// interleaved (x1, x2, v) triples of two neighbouring channels: three words (x1 x2 | v x1 | x2 v)
struct FeatPair { f2 x1, x2, v; };
__device__ __forceinline__ FeatPair feat_pair(uint32_t w0, uint32_t w1, uint32_t w2) {
  return FeatPair{f2_pack(lo_f(w0), hi_f(w1)), f2_pack(hi_f(w0), lo_f(w2)), f2_pack(lo_f(w1), hi_f(w2))};
}

}  // namespace sb
