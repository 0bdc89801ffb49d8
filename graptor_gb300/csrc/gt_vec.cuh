// Slice vectors of the register-blocked projectors: VW slices per lane as packed pairs, so
// that one fma.rn.f32x2 does two of them (each half rounds as a scalar fused multiply-add).
#pragma once
#include <cuda_runtime.h>

namespace gt {

typedef unsigned long long f32x2;  // two floats, the lower slice in the lower half

__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

__device__ __forceinline__ void fma2(f32x2 &acc, f32x2 w, f32x2 v) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w), "l"(v));
}

// VW = 8: two runs of 4 slices, the second off2 (128 or 0) after the first; 4, 2, 1: one run
template <int VW>
struct Vec {
  f32x2 v[VW / 2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < VW / 2; ++k) v[k] = 0ull;
  }
  __device__ __forceinline__ void load(const float *__restrict__ p, int off2) {
    if constexpr (VW >= 4) {
      const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2 *>(p));
      v[0] = a.x;
      v[1] = a.y;
      if constexpr (VW == 8) {
        const ulonglong2 b = __ldg(reinterpret_cast<const ulonglong2 *>(p + off2));
        v[2] = b.x;
        v[3] = b.y;
      }
    } else {
      v[0] = __ldg(reinterpret_cast<const f32x2 *>(p));
    }
  }
  // plain loads and stores of a lane's slices; vb: the second run lies inside the field
  static __device__ __forceinline__ void loadw(const float *p, float (&r)[VW], bool vb) {
    if constexpr (VW >= 4) {
      const float4 a = *reinterpret_cast<const float4 *>(p);
      r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
      if constexpr (VW == 8) {
        const float4 b = vb ? *reinterpret_cast<const float4 *>(p + 128) : make_float4(0.f, 0.f, 0.f, 0.f);
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
      }
    } else {
      const float2 a = *reinterpret_cast<const float2 *>(p);
      r[0] = a.x; r[1] = a.y;
    }
  }
  static __device__ __forceinline__ void store(float *p, const float (&r)[VW], bool vb) {
    if constexpr (VW >= 4) {
      *reinterpret_cast<float4 *>(p) = make_float4(r[0], r[1], r[2], r[3]);
      if constexpr (VW == 8) {
        if (vb) *reinterpret_cast<float4 *>(p + 128) = make_float4(r[4], r[5], r[6], r[7]);
      }
    } else {
      *reinterpret_cast<float2 *>(p) = make_float2(r[0], r[1]);
    }
  }
};

template <>
struct Vec<1> {
  float v;
  __device__ __forceinline__ void clear() { v = 0.f; }
  __device__ __forceinline__ void load(const float *__restrict__ p, int) { v = __ldg(p); }
  static __device__ __forceinline__ void loadw(const float *p, float (&r)[1], bool) { r[0] = *p; }
  static __device__ __forceinline__ void store(float *p, const float (&r)[1], bool) { *p = r[0]; }
};

template <int VW>
struct VecAcc {
  f32x2 v[VW / 2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < VW / 2; ++k) v[k] = 0ull;
  }
  __device__ __forceinline__ void fma(float w, const Vec<VW> &x) {
    const f32x2 ww = pack2(w, w);
#pragma unroll
    for (int k = 0; k < VW / 2; ++k) fma2(v[k], ww, x.v[k]);
  }
  __device__ __forceinline__ void get(float (&r)[VW]) const {
#pragma unroll
    for (int k = 0; k < VW / 2; ++k) unpack2(v[k], r[2 * k], r[2 * k + 1]);
  }
  __device__ __forceinline__ bool finite() const {
    float r[VW], z = 0.f;
    get(r);
#pragma unroll
    for (int k = 0; k < VW; ++k) z = __fmaf_rn(r[k], 0.f, z);  // 0, or NaN once an r is infinite or NaN
    return z == 0.f;
  }
};

template <>
struct VecAcc<1> {
  float v;
  __device__ __forceinline__ void zero() { v = 0.f; }
  __device__ __forceinline__ void fma(float w, const Vec<1> &x) { v = __fmaf_rn(w, x.v, v); }
  __device__ __forceinline__ void get(float (&r)[1]) const { r[0] = v; }
};

}  // namespace gt
