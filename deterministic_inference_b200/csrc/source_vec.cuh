// Four consecutive elements of a Source at once, and of outputs: for the element-wise kernels of prompt
// portions, which are bound by the loads and stores they can issue and have in flight (a 2,048 x 3,072
// float32 matrix through an element-wise kernel: 16 us one element a thread and load, 12 us four; the split of
// 2,048 projection rows of 4,096 into heads 20 us, 11 us four).
#pragma once

#include "source.cuh"

// Can elements 4 i .. 4 i + 3 of the source be read with one load (of a split)?
static inline bool source_takes_vectors(const Source& s) {
  const uintptr_t p = reinterpret_cast<uintptr_t>(s.p);
  return s.kind == 1 ? p % 8 == 0 : p % 16 == 0 && (s.splits == 1 || s.stride % 4 == 0);
}
static inline bool vectors_start_at(const void* p, int dtype) {
  return reinterpret_cast<uintptr_t>(p) % (dtype == 1 ? 8 : 16) == 0;
}

__device__ __forceinline__ float4 bf16x4(uint2 x) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// elements i .. i + 3, i a multiple of 4; the splits are added in order, as by source_load
__device__ __forceinline__ float4 source_load4(const Source& s, long long i) {
  if (s.kind == 1) return bf16x4(*reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(s.p) + i));
  const float* f = reinterpret_cast<const float*>(s.p) + i;
  float4 v = *reinterpret_cast<const float4*>(f);
  for (int k = 1; k < s.splits; ++k) {
    const float4 a = *reinterpret_cast<const float4*>(f + (long long)k * s.stride);
    v.x = __fadd_rn(v.x, a.x);
    v.y = __fadd_rn(v.y, a.y);
    v.z = __fadd_rn(v.z, a.z);
    v.w = __fadd_rn(v.w, a.w);
  }
  return v;
}
template <typename T> __device__ __forceinline__ void store4(T* p, float4 v);
template <> __device__ __forceinline__ void store4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
}
__device__ __forceinline__ void store4_as(void* p, int dtype, long long i, float4 v) {
  if (dtype == 1) store4(reinterpret_cast<__nv_bfloat16*>(p) + i, v);
  else store4(reinterpret_cast<float*>(p) + i, v);
}
