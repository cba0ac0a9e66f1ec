// Warp-level pieces of int8-KV decode attention, shared by the split-K kernel and the fused decode step: the two-part
// int8 split of the query, the int8 / fp16 tensor-core steps and the in-register dequantisation of V.
#pragma once

#include "common.cuh"

namespace uv {

constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_GAP = 6.0f;  // 2^6 * (largest fp16 scale 65504/127) still fits fp16

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// two bytes (already xor 0x80) selected from x -> half2 of the signed values: 0x64xx is 1024 + xx, minus 1152
__device__ __forceinline__ uint32_t bias_pair(uint32_t x, uint32_t sel) {
  uint32_t w = __byte_perm(x, 0x64646464u, sel);
  __half2 h = __hsub2(*reinterpret_cast<__half2*>(&w), __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<uint32_t*>(&h);
}

// Two-part symmetric int8 split of one query head slice held by a quad: q ~= s1*q1 + (s1/254)*q2 with
// |error| <= max|q| / 64516, so Q K^T runs on the int8 tensor-core path against the raw cache bytes.
template <int N>
__device__ __forceinline__ void split_q(const float (&qv)[N], uint32_t (&w1)[N / 4], uint32_t (&w2)[N / 4],
                                        float& f1, float& f2, float scale_log2) {
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) amax = fmaxf(amax, fabsf(qv[i]));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  const float s1 = amax > 0.f ? amax / 127.0f : 1.0f;
  const float inv1 = 1.0f / s1, inv2 = 254.0f / s1;
#pragma unroll
  for (int w = 0; w < N / 4; ++w) {
    uint32_t p1 = 0u, p2 = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float x = qv[4 * w + i];
      const float a = fminf(fmaxf(rintf(x * inv1), -127.f), 127.f);
      const float b = fminf(fmaxf(rintf((x - a * s1) * inv2), -127.f), 127.f);
      p1 |= ((uint32_t)(__float2int_rn(a) & 0xff)) << (8 * i);
      p2 |= ((uint32_t)(__float2int_rn(b) & 0xff)) << (8 * i);
    }
    w1[w] = p1, w2[w] = p2;
  }
  f1 = s1 * scale_log2;
  f2 = s1 * (1.0f / 254.0f) * scale_log2;
}

__device__ __forceinline__ void imma16832(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// first k-step of a tile: C = 0, so the accumulators need no clearing
__device__ __forceinline__ void imma16832_z(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                            uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

}  // namespace uv
