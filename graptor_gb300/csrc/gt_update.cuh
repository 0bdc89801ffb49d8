// Device code of the primal update shared by k_update (gt_kernels.cu) and the two-launch
// iteration of small problems (gt_small.cu).
#pragma once
#include <cuda_runtime.h>

#include "gt_common.cuh"
#include "gt_dual.cuh"

namespace gt {

// coherent vector loads / stores of UW consecutive slices (fields a kernel also writes)
template <int VW> __device__ __forceinline__ void ldw(const float *p, float (&r)[VW]) {
  if (VW == 4) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    r[0] = q.x; r[1 % VW] = q.y; r[2 % VW] = q.z; r[3 % VW] = q.w;
  } else if (VW == 2) {
    const float2 q = *reinterpret_cast<const float2 *>(p);
    r[0] = q.x; r[1 % VW] = q.y;
  } else {
    r[0] = p[0];
  }
}
template <int VW> __device__ __forceinline__ void stv(float *p, const float (&r)[VW]) {
  if (VW == 4) *reinterpret_cast<float4 *>(p) = make_float4(r[0], r[1 % VW], r[2 % VW], r[3 % VW]);
  else if (VW == 2) *reinterpret_cast<float2 *>(p) = make_float2(r[0], r[1 % VW]);
  else p[0] = r[0];
}

// update_u (3-D :706-729, 2-D :340-357) + update_p (3-D :734-757, 2-D :359-376) +
// extrapolation and swap (:1217-1221) for UW consecutive slices from s0.
// PART selects the halves: PART_U the u / ubar half (needs K* lambda), PART_P the
// p / pbar half (needs only the dual kernel's v and w), PART_ALL both.  Each half
// computes its values by the same operations whichever way it is launched.
enum { PART_ALL = 0, PART_U = 1, PART_P = 2 };
template <int DIM, bool TGV, int UW, int PART = PART_ALL>
__device__ __forceinline__ void primal_update(const IterParams &P, int x, int y, int s0, const float (&kstar)[UW]) {
  const Dims d = P.d;
  const size_t S = d.S, rowS = (size_t)d.N * S, vol = d.vol, i = ((size_t)y * d.N + x) * S + s0;
  // first / last slice of the channel; a padding slice (s >= C Nz) has no neighbours, so it stays zero
  bool fz[UW], lz[UW];
#pragma unroll
  for (int k = 0; k < UW; ++k) {
    const int z = (DIM == 3) ? (s0 + k) % d.Nz : 0;
    const bool pad = s0 + k >= d.C * d.Nz;
    fz[k] = pad || z == 0;
    lz[k] = pad || z == d.Nz - 1;
  }
  const float *__restrict__ v = P.v;

  if (PART != PART_P) {
  // divergence of v: backward differences (adjoint of the forward gradient)
  float a[UW], b[UW], am[UW], bm[UW], uo[UW], un[UW], ub[UW];
  ldw<UW>(v + i, a);
  ldw<UW>(v + vol + i, b);
  if (x > 0) ldw<UW>(v + i - S, am);
  if (y > 0) ldw<UW>(v + vol + i - rowS, bm);
  ldw<UW>(P.u + i, uo);
  float c[UW], cprev = 0.f;
  if (DIM == 3) {
    ldw<UW>(v + 2 * vol + i, c);
    if (!fz[0]) cprev = v[2 * vol + i - 1];
  }
  float lo[UW], lon[UW];  // the low parts of u (precise primal mode, P.ulo set)
  if (P.ulo) ldw<UW>(P.ulo + i, lo);
#pragma unroll
  for (int k = 0; k < UW; ++k) {
    float ak = a[k], bk = b[k];
    if (x == d.N - 1) ak = 0.f;
    if (x > 0) ak -= am[k];
    if (y == d.N - 1) bk = 0.f;
    if (y > 0) bk -= bm[k];
    float sum;
    if (DIM == 3) {
      float ck = c[k];
      if (lz[k]) ck = 0.f;
      if (!fz[k]) ck -= (k > 0 ? c[k - 1] : cprev);
      ck /= P.stepsize;
      sum = ak + bk + ck - P.norming * kstar[k];
    } else {
      sum = ak + bk - P.norming * kstar[k];
    }
    if (!P.ulo) {  // the reference's update (one rounding of u + tau sum)
      float r = uo[k] + P.tau * sum;
      if (r < 0.f) r = 0.f;
      un[k] = r;
      ub[k] = 2.0f * r - uo[k];
    } else {
      // u held as uo + lo (two floats): the step is added to the low part and
      // the pair renormalised by TwoSum (Knuth), so steps below half an ulp of u
      // are kept instead of absorbed
      const float t = lo[k] + P.tau * sum;
      const float r = __fadd_rn(uo[k], t);
      const float bv = __fsub_rn(r, uo[k]);
      const float e = __fadd_rn(__fsub_rn(uo[k], __fsub_rn(r, bv)), __fsub_rn(t, bv));
      const bool neg = r < 0.f || (r == 0.f && e < 0.f);
      un[k] = neg ? 0.f : r;
      lon[k] = neg ? 0.f : e;
      ub[k] = (2.0f * un[k] - uo[k]) + (2.0f * lon[k] - lo[k]);
    }
  }
  stv<UW>(P.ubar + i, ub);
  stv<UW>(P.u + i, un);
  if (P.ulo) stv<UW>(P.ulo + i, lon);
  }

  if (TGV && PART != PART_U) {
    const float *__restrict__ w = P.w;
    constexpr int K = DIM;
    // rows of the symmetric tensor: 3-D (w0 w3 w4), (w3 w1 w5), (w4 w5 w2); 2-D (w0 w2), (w2 w1)
    const int rx[3] = {0, DIM == 3 ? 3 : 2, 4}, ry[3] = {DIM == 3 ? 3 : 2, 1, 5}, rz[3] = {4, 5, 2};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float wa[UW], wan[UW], wb[UW], wbn[UW], po[UW], vk[UW], pn[UW], pb[UW];
      ldw<UW>(w + rx[k] * vol + i, wa);
      ldw<UW>(w + ry[k] * vol + i, wb);
      if (x < d.N - 1) ldw<UW>(w + rx[k] * vol + i + S, wan);
      if (y < d.N - 1) ldw<UW>(w + ry[k] * vol + i + rowS, wbn);
      ldw<UW>(P.p + k * vol + i, po);
      ldw<UW>(v + k * vol + i, vk);
      float wc[UW], wcnext = 0.f;
      if (DIM == 3) {
        ldw<UW>(w + rz[k] * vol + i, wc);
        if (!lz[UW - 1]) wcnext = w[rz[k] * vol + i + UW];
      }
#pragma unroll
      for (int e = 0; e < UW; ++e) {
        float A = -wa[e], B = -wb[e];
        if (x == 0) A = 0.f;
        if (x < d.N - 1) A += wan[e];
        if (y == 0) B = 0.f;
        if (y < d.N - 1) B += wbn[e];
        float r;
        if (DIM == 3) {
          r = p_step3(po[e], vk[e], wa[e], wan[e], wb[e], wbn[e], wc[e], e < UW - 1 ? wc[e + 1] : wcnext, x == 0,
                      x < d.N - 1, y == 0, y < d.N - 1, fz[e], !lz[e], P.tau, P.stepsize);
        } else {
          r = po[e] + P.tau * (vk[e] + A + B);
        }
        pn[e] = r;
        pb[e] = 2.0f * r - po[e];
      }
      stv<UW>(P.pbar + k * vol + i, pb);
      stv<UW>(P.p + k * vol + i, pn);
    }
  }
}

template <int DIM, bool TGV, int UW, int PART = PART_ALL>
__device__ __forceinline__ void update_body(const IterParams &P, long long bid) {
  const Dims d = P.d;
  const int nsg = d.S / UW;
  const long long t = bid * blockDim.x + threadIdx.x;
  if (t >= (long long)d.N * d.N * nsg) return;
  const int pix = (int)(t / nsg);
  const int s0 = (int)(t - (long long)pix * nsg) * UW;
  const int y = pix / d.N, x = pix - y * d.N;
  float ks[UW];
  if (PART != PART_P) ldw<UW>(P.kstar + (size_t)pix * d.S + s0, ks);
  primal_update<DIM, TGV, UW, PART>(P, x, y, s0, ks);
}

}  // namespace gt
