// Helpers shared by the warm-start network's translation units.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace gt {
int set_error(int code, const char *msg);
int cuda_error(cudaError_t e, const char *what, int line);
}  // namespace gt

#define NN_CK(expr, what)                                              \
  do {                                                                 \
    cudaError_t e_ = (expr);                                           \
    if (e_ != cudaSuccess) return gt::cuda_error(e_, what, __LINE__);   \
  } while (0)

namespace {

template <class T> __device__ __forceinline__ float ld(const T *p) { return (float)*p; }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16 *p) { return __bfloat162float(*p); }
template <class T> __device__ __forceinline__ void st(T *p, float v) { *p = (T)v; }
template <> __device__ __forceinline__ void st<__nv_bfloat16>(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

struct Shape {
  int B, D, H, W;
};

inline unsigned nblk(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace
