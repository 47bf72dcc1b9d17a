// Arithmetic helpers shared by the attention kernels (mha_nvfp4.cu, mha_int8_fp8.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace ac4k {

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// max of three (one FMNMX3), and two fp32 operations in one instruction on an aligned register pair
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rc, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nmov.b64 rc, {%6, %7};\n"
      "fma.rn.f32x2 rd, ra, rb, rc;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\n"
      "mul.rn.f32x2 rd, ra, rb;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\n"
      "add.rn.f32x2 rd, ra, rb;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
// 128 columns of this warp's 16 rows of O in tensor memory (16x256b shape) times a[r], r = 0, 1 the thread's two rows
__device__ __forceinline__ void mha_rescale(uint32_t t_o, const float (&a)[2]) {
  uint32_t ro[64];
  ptx::tmem_ld_16x256b_x16(t_o, ro);
  ptx::tmem_ld_wait();
  ptx::tmem_pin(ro);
#pragma unroll
  for (int i = 0; i < 64; i += 2) {
    const float f = a[(i >> 1) & 1];
    const float2 v = fmul2(make_float2(__uint_as_float(ro[i]), __uint_as_float(ro[i + 1])), make_float2(f, f));
    ro[i] = __float_as_uint(v.x);
    ro[i + 1] = __float_as_uint(v.y);
  }
  ptx::tmem_st_16x256b_x16(t_o, ro);
  ptx::tmem_st_wait();
}
// Query tiles per CTA.  A pair of tiles shares the K and V tiles and fills each other's waits, but a launch of few CTAs leaves SMs
// idle: one tile per CTA where that ends sooner, counted in waves of CTAs.  A CTA with two tiles takes 1.4 times one with one (INT8,
// 4096 keys: 55 / 40 us a wave; NVFP4 61 / 43), and with an odd number of tiles every head's last CTA has one.  Kernel us, one tile /
// two, INT8 (NVFP4 alike): 9 heads x 2048 x 2048, one wave either way: 27 / 32; 12 heads, two waves against one: 47 / 33; 190 heads
// x 384 x 1024, four against three, every other CTA with one tile: 62 / 53; 98 heads, two against two: 31 / 33.
inline int mha_query_tiles(int64_t q_blocks, int64_t heads, int sms) {
  if (q_blocks < 2) return 1;
  const int64_t full = q_blocks / 2, ctas = full + (q_blocks & 1);       // of a head, two tiles each
  const int64_t waves2 = (heads * ctas + sms - 1) / sms, waves1 = (heads * q_blocks + sms - 1) / sms;
  return 10 * waves1 * ctas >= waves2 * (14 * full + 10 * (q_blocks & 1)) ? 2 : 1;
}
// O may be stored four columns at a time: its rows are contiguous and start on 8-byte boundaries
__device__ __forceinline__ bool mha_rows_vec4(const void *O, int64_t o_b, int64_t o_h, int64_t o_n, int64_t o_d, int Dv) {
  return o_d == 1 && (Dv & 3) == 0 && ((o_b | o_h | o_n) & 3) == 0 && (reinterpret_cast<uintptr_t>(O) & 7) == 0;
}
// One row's 32 columns c0 .. c0 + 31 of O from the four threads that hold it in the 16x256b shape: o[2 i + e] is column
// c0 + 8 i + 2 t4 + e.  Vector form: neighbouring threads swap words, so that the even one has four columns of the first
// eight of every sixteen and the odd one of the second, and the four of them write whole 32-byte sectors.
__device__ __forceinline__ void mha_store_row(__nv_bfloat16 *dst, const float (&o)[8], int c0, int t4, int Dv, int64_t o_d, bool vec,
                                              bool live) {
  if (vec) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h2 = __floats2bfloat162_rn(o[2 * i], o[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t *>(&h2);
    }
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, (t4 & 1) ? w[i] : w[i + 1], 1);
      const int col = c0 + 8 * i + ((t4 & 1) ? 6 + 2 * t4 : 2 * t4);
      if (live && col < Dv) *reinterpret_cast<uint2 *>(dst + col) = (t4 & 1) ? make_uint2(got, w[i + 1]) : make_uint2(w[i], got);
    }
  } else if (live) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int col = c0 + 8 * (i >> 1) + 2 * t4 + (i & 1);
      if (col < Dv) dst[(int64_t)col * o_d] = __float2bfloat16_rn(o[i]);
    }
  }
}
}  // namespace ac4k
