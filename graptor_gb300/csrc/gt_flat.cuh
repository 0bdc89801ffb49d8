// Device code of the flat and staged projectors (few slices per pixel), shared by their own
// kernels (gt_fwd.cu, gt_proj.cu) and the two-launch iteration of small problems (gt_small.cu).
#pragma once
#include <cuda_runtime.h>

#include "gt_common.cuh"
#include "gt_vec.cuh"

namespace gt {

// A kernel whose threads need several loads in flight gives __launch_bounds__ its second
// argument (1 block): without it ptxas aims at occupancy and orders the loads of a group one
// after another (the forward projection below: 72 instead of 114 registers, 14.4 instead of
// 10.4 us on 64^2 x 32; the back projection 32 instead of 64 registers, 25.9 instead of 12.3 us).

// t / n without the 64-bit division where 32 bits do
__device__ __forceinline__ long long div_pos(long long t, int n) {
  return t < (1ll << 32) ? (long long)((unsigned)t / (unsigned)n) : t / n;
}

// p + k * S (k >= 0): one 32 x 32 + 64 bit multiply-add, not a 64-bit product
__device__ __forceinline__ const float *at(const float *p, int k, int S) {
  return reinterpret_cast<const float *>(reinterpret_cast<const char *>(p) +
                                         (unsigned long long)(unsigned)k * (4u * (unsigned)S));
}

// one ray from the ray table, UNR entries in flight; the next group's entries are fetched
// while the current group's pixels are on their way
template <int VW, int UNR>
__device__ __forceinline__ void ray_sum(const float *__restrict__ img, size_t S, const int2 *__restrict__ ent, int n,
                                        int off2, VecAcc<VW> &acc) {
  int2 nx[UNR];
#pragma unroll
  for (int u = 0; u < UNR; ++u) nx[u] = n > 0 ? __ldg(ent + min(u, n - 1)) : make_int2(0, 0);
  int e = 0;
  for (; e + UNR <= n; e += UNR) {
    float w[UNR];
    Vec<VW> v[UNR];
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      v[u].load(img + (size_t)nx[u].x * S, off2);
      w[u] = __int_as_float(nx[u].y);
    }
#pragma unroll
    for (int u = 0; u < UNR; ++u) nx[u] = __ldg(ent + min(e + UNR + u, n - 1));
#pragma unroll
    for (int u = 0; u < UNR; ++u) acc.fma(w[u], v[u]);
  }
#pragma unroll
  for (int u = 0; u < UNR - 1; ++u) {  // the rest: its entries are in nx
    if (e + u < n) {
      Vec<VW> v;
      v.load(img + (size_t)nx[u].x * S, off2);
      acc.fma(__int_as_float(nx[u].y), v);
    }
  }
}

// K u and the data dual of bin b (j * nd + i), slices s0 ..; vb: see Vec::store
template <int VW>
__device__ __forceinline__ void data_step(const IterParams &P, int disc, const VecAcc<VW> &acc, long long b, int s0,
                                          bool vb) {
  const Dims d = P.d;
  const float sd = P.sigma_data;
  const size_t q = (size_t)b * d.S + s0;
  float a[VW], lam[VW], f[VW];
  acc.get(a);
  Vec<VW>::store(P.ku + q, a, vb);
  if (disc == DATA_NONE) return;
  Vec<VW>::loadw(P.lam + q, lam, vb);
  Vec<VW>::loadw(P.f + q, f, vb);
#pragma unroll
  for (int k = 0; k < VW; ++k) {
    const int s = VW == 8 ? s0 + (k < 4 ? k : 124 + k) : s0 + k;
    const float m = s < d.S ? __ldg(P.mu + s / d.Nz) : 0.f;
    if (disc == KL) {
      const float sv = lam[k] + sd * a[k];
      const float wv = sv - m;
      const float dv = wv * wv + 4.f * sd * f[k] * m;
      lam[k] = sv - 0.5f * (wv + sqrtf(dv));
    } else {
      lam[k] = (lam[k] + sd * (a[k] - f[k])) * m;
    }
  }
  Vec<VW>::store(P.lam + q, lam, vb);
}

// forward projection of thread t = (ray, VW slices)
template <int VW, int UNR>
__device__ __forceinline__ void fwd_flat_body(const IterParams &P, int disc, long long t) {
  const Dims d = P.d;
  const int ng = d.S / VW;
  if (t >= (long long)ng * d.nd * d.nang) return;
  const long long b = div_pos(t, ng);
  const int s0 = (int)(t - b * ng) * VW;
  const long long r0 = __ldg(P.ray_start + b);
  VecAcc<VW> acc;
  acc.zero();
  ray_sum<VW, UNR>(P.ubar + s0, d.S, P.ray_ent + r0, (int)(__ldg(P.ray_start + b + 1) - r0), 0, acc);
  data_step<VW>(P, disc, acc, b, s0, false);
}

// ---------------------------------------------------------------------------
// S = VW slices (1, 2 or 4): a thread per ray or pixel leaves most of the GPU idle and its chain
// of dependent loads bare.  The staged forms load for several rays or pixels at once into
// shared memory and add from there in order.
// ---------------------------------------------------------------------------
constexpr int FS_RAYS = 32;  // rays of a block (of 256 threads)
constexpr int BS_PIX = 8;    // pixels of a warp (lanes: 8 pixels x 4 angles)
constexpr int BS_ANG = 32;   // angles staged at a time

template <int VW>
struct FwdStage {
  static constexpr int CH = VW == 1 ? 128 : VW == 2 ? 96 : 64;  // entries of a ray staged at a time
  float w[FS_RAYS][CH + 1];
  Vec<VW> v[FS_RAYS][CH + 1];
};

template <int VW>
struct BpStage {
  float2 w[BS_ANG][BS_PIX];
  Vec<VW> a[BS_ANG][BS_PIX], b[BS_ANG][BS_PIX];
};

// forward projection of rays 32 bid .. (256 threads): the 8 warps stage CH entries of the 32
// rays in runs of 32 entries, warp 0 (lane = ray) adds them
template <int VW>
__device__ __forceinline__ void fwd_staged_body(const IterParams &P, int disc, long long bid, FwdStage<VW> &sh) {
  constexpr int CH = FwdStage<VW>::CH, RW = FS_RAYS / 8;
  const Dims d = P.d;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long rays = (long long)d.nd * d.nang, b0 = bid * FS_RAYS;
  const int2 *__restrict__ ent[RW];
  int n[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const long long b = b0 + warp * RW + r, bc = min(b, rays - 1);
    const long long r0 = __ldg(P.ray_start + bc);
    ent[r] = P.ray_ent + r0;
    n[r] = b < rays ? (int)(__ldg(P.ray_start + bc + 1) - r0) : 0;
  }
  const long long bl = min(b0 + lane, rays - 1);
  const int mine = b0 + lane < rays ? (int)(__ldg(P.ray_start + bl + 1) - __ldg(P.ray_start + bl)) : 0;
  const int nmax = __reduce_max_sync(0xffffffffu, mine);  // the same in every warp
  VecAcc<VW> acc;
  acc.zero();
  for (int c = 0; c < nmax; c += CH) {
    int2 e[RW][CH / 32];
    Vec<VW> v[RW][CH / 32];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int k = 0; k < CH / 32; ++k) {
        const int q = c + k * 32 + lane;
        e[r][k] = q < n[r] ? __ldg(ent[r] + q) : make_int2(-1, 0);  // past the end: 0 x 0 leaves a sum unchanged
      }
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int k = 0; k < CH / 32; ++k) {
        v[r][k].clear();
        if (e[r][k].x >= 0) v[r][k].load(P.ubar + (size_t)e[r][k].x * VW, 0);
      }
    __syncthreads();  // the chunk before has been added
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int k = 0; k < CH / 32; ++k) {
        sh.w[warp * RW + r][k * 32 + lane] = __int_as_float(e[r][k].y);
        sh.v[warp * RW + r][k * 32 + lane] = v[r][k];
      }
    __syncthreads();
    if (warp == 0) {
      const int m = min(CH, (nmax - c + 15) & ~15);
#pragma unroll 1
      for (int k = 0; k < m; k += 16)
#pragma unroll
        for (int q = 0; q < 16; ++q) acc.fma(sh.w[lane][k + q], sh.v[lane][k + q]);
    }
  }
  if (warp == 0 && b0 + lane < rays) data_step<VW>(P, disc, acc, b0 + lane, 0, false);
}

// back projection of pixels BS_PIX * wid ..: lane 0 .. BS_PIX - 1 gets its pixel and sum and true
template <int VW>
__device__ __forceinline__ bool bp_staged_body(const IterParams &P, long long wid, BpStage<VW> &sh, int &pix,
                                               float (&r)[VW]) {
  const Dims d = P.d;
  const int lane = threadIdx.x & 31, px = lane & (BS_PIX - 1), slot = lane / BS_PIX;
  constexpr int SLOTS = 32 / BS_PIX, NK = BS_ANG / SLOTS;
  if (wid * BS_PIX >= (long long)P.npix) return false;
  pix = (int)min(wid * BS_PIX + px, (long long)P.npix - 1);
  const int y = pix / d.N, x = pix - y * d.N;
  const float xf = (float)x, yf = (float)y, fnd = (float)d.nd;
  VecAcc<VW> acc;
  acc.zero();
  for (int j0 = 0; j0 < d.nang; j0 += BS_ANG) {
    Vec<VW> a[NK], b[NK];
    float p[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      const int j = j0 + k * SLOTS + slot;
      const float4 o = __ldg(P.ofs + min(j, d.nang - 1));
      const float tt = __fadd_rn(__fadd_rn(__fmul_rn(xf, o.x), __fmul_rn(yf, o.y)), o.z);
      const bool in = tt > -1.f && tt < fnd && j < d.nang;
      const float fl = floorf(tt);
      p[k] = in ? fminf(__fsub_rn(tt, fl), 0x1.fffffep-1f) : 0.f;
      const int il = (int)fl;
      const float *__restrict__ lj = P.lam + (size_t)j * d.nd * VW;
      a[k].clear();
      b[k].clear();
      // a tap off the detector stays 0: its product leaves the sum unchanged
      if (in && il >= 0) a[k].load(lj + (size_t)il * VW, 0);
      if (in && il <= d.nd - 2) b[k].load(lj + (size_t)(il + 1) * VW, 0);
    }
    __syncwarp();  // the angles before have been added
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      const int q = k * SLOTS + slot;
      sh.w[q][px] = make_float2(__fsub_rn(1.0f, p[k]), p[k]);
      sh.a[q][px] = a[k];
      sh.b[q][px] = b[k];
    }
    __syncwarp();
    if (lane < BS_PIX) {
#pragma unroll 8
      for (int q = 0; q < BS_ANG; ++q) {
        const float2 w = sh.w[q][lane];
        acc.fma(w.x, sh.a[q][lane]);
        acc.fma(w.y, sh.b[q][lane]);
      }
    }
  }
  acc.get(r);
  return lane < BS_PIX && wid * BS_PIX + lane < (long long)P.npix;
}

// back projection of thread t = (pixel, VW slices), UA angles at a time: their taps are loaded
// together, then added in angle order; false past the end
template <int VW, int UA>
__device__ __forceinline__ bool bp_flat_body(const IterParams &P, long long t, int &pix, int &s0, float (&r)[VW]) {
  const Dims d = P.d;
  const int ng = d.S / VW;
  if (t >= (long long)ng * d.N * d.N) return false;
  pix = (int)div_pos(t, ng);
  s0 = (int)(t - (long long)pix * ng) * VW;
  const int y = pix / d.N, x = pix - y * d.N;
  const float xf = (float)x, yf = (float)y, fnd = (float)d.nd;
  const size_t jstride = (size_t)d.nd * d.S;
  const float *__restrict__ lam = P.lam + s0;
  VecAcc<VW> acc;
  acc.zero();
  for (int j0 = 0; j0 < d.nang; j0 += UA) {
    Vec<VW> a[UA], b[UA];
    float p[UA];
#pragma unroll
    for (int u = 0; u < UA; ++u) {
      const int j = min(j0 + u, d.nang - 1);
      const float4 o = __ldg(P.ofs + j);
      const float tt = __fadd_rn(__fadd_rn(__fmul_rn(xf, o.x), __fmul_rn(yf, o.y)), o.z);
      const bool in = tt > -1.f && tt < fnd && j0 + u < d.nang;
      const float fl = floorf(tt);
      p[u] = in ? fminf(__fsub_rn(tt, fl), 0x1.fffffep-1f) : 0.f;
      const int il = (int)fl;
      const float *__restrict__ lj = lam + (size_t)j * jstride;
      a[u].clear();
      b[u].clear();
      // a tap off the detector stays 0: its product leaves the sum unchanged
      if (in && il >= 0) a[u].load(at(lj, il, d.S), 0);
      if (in && il <= d.nd - 2) b[u].load(at(lj, il + 1, d.S), 0);
    }
#pragma unroll
    for (int u = 0; u < UA; ++u) {
      acc.fma(__fsub_rn(1.0f, p[u]), a[u]);
      acc.fma(p[u], b[u]);
    }
  }
  acc.get(r);
  return true;
}

}  // namespace gt
