// FP32 values as pairs of FP16 numbers (gemm_pair.cu says what for): hi = fp16(v s), lo = fp16((v s - hi) 2^11).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace pg {
namespace {

constexpr float PAIR_LO = 2048.f, PAIR_LO_INV = 1.f / 2048.f;

__device__ __forceinline__ void split_pair2(float a, float b, float scale, uint32_t& hi, uint32_t& lo) {
  const float x = a * scale, y = b * scale;
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn((x - f.x) * PAIR_LO, (y - f.y) * PAIR_LO);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void store_pair2(uint16_t* hi, uint16_t* lo, float a, float b, float scale) {
  uint32_t h, l;
  split_pair2(a, b, scale, h, l);
  *reinterpret_cast<uint32_t*>(hi) = h;
  *reinterpret_cast<uint32_t*>(lo) = l;
}
__device__ __forceinline__ void store_pair4(uint16_t* hi, uint16_t* lo, float4 v, float scale) {
  uint2 h, l;
  split_pair2(v.x, v.y, scale, h.x, l.x);
  split_pair2(v.z, v.w, scale, h.y, l.y);
  *reinterpret_cast<uint2*>(hi) = h;
  *reinterpret_cast<uint2*>(lo) = l;
}

}  // namespace
}  // namespace pg
