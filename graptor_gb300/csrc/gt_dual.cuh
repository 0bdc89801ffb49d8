// Device code of the dual update shared by the dual kernels (gt_kernels.cu) and the two-launch
// iteration of small problems (gt_small.cu).
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "gt_common.cuh"
#include "gt_round.cuh"

namespace gt {

// ===========================================================================
// ball projections
// ===========================================================================

// The nuclear-norm projections evaluate eigenvectors by formulas that cancel
// catastrophically when the off-diagonal entry is small, so their results depend
// on rounding: they are written with explicitly rounded operations (no fused
// multiply-add), in the reference's order, and with hypot / atan / cos / cube
// as evaluated in double and rounded once (as the host C library's float versions
// are, to within their last bit).  gt_round.cuh gives those values without FP64 but for
// about one call in 10^4, which is left to the functions here.
__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
static __device__ __noinline__ float hyp_exact(float a, float b) { return (float)sqrt((double)a * a + (double)b * b); }
static __device__ __noinline__ float cos_exact(float x) { return (float)cos((double)x); }
static __device__ __noinline__ float atan_exact(float y) { return (float)atan((double)y); }
static __device__ __noinline__ float cube_exact(float c) { return (float)((double)c * c * c); }

__device__ __forceinline__ float hyp(float a, float b) {
  float r;
  return hyp_round(a, b, r) ? r : hyp_exact(a, b);
}
__device__ __forceinline__ float cos_f(float x) {
  float r;
  return cos_round(x, r) ? r : cos_exact(x);
}
__device__ __forceinline__ float atan_f(float y) {
  float r;
  return atan_round(y, r) ? r : atan_exact(y);
}
__device__ __forceinline__ float cube_f(float c) {
  float r;
  return cube_round(c, r) ? r : cube_exact(c);
}

// nuclear 2-D (update_NormV_Nucl, radon_tgv_primal_dual_2d.py:124-204): spectral
// projection of the C x 2 matrix A of one pixel via the 2x2 matrix A^T A = [a b; b c].
__device__ __forceinline__ void nucl2d_matrix(float a, float b, float c, float ainv, float M[3]) {
  const float eps = 0.00001f;
  float s1, s2, S1, S2;
  const float o = c < a ? c : a;
  if (fm(b, b) / fm(o, o) > eps && fm(o, o) > 0.f) {
    const float dd = fa(a, c), e = fs(a, c);
    float f = fa(fm(fm(4.f, b), b), fm(e, e));
    f = f < 0.f ? 0.f : sqrtf(f);
    s2 = (fs(dd, f) > 0.f) ? sqrtf(fm(fs(dd, f), 0.5f)) : 0.f;
    s1 = (fa(dd, f) > 0.f) ? sqrtf(fm(fa(dd, f), 0.5f)) : 0.f;
    const float g = fm(fa(e, f), 0.5f), h = fm(fs(e, f), 0.5f);
    float q0 = fa(fm(g, a), fm(b, b)), q1 = fa(fm(g, b), fm(c, b));
    float q2 = fa(fm(h, a), fm(b, b)), q3 = fa(fm(h, b), fm(b, c));
    const float n1 = hyp(q0, q1), n2 = hyp(q2, q3);
    if (n1 > 0.f) { q0 = q0 / n1; q1 = q1 / n1; }
    if (n2 > 0.f) { q2 = q2 / n2; q3 = q3 / n2; }
    S1 = (fm(s1, ainv) > 1.f) ? 1.f / fm(s1, ainv) : 1.f;
    S2 = (fm(s2, ainv) > 1.f) ? 1.f / fm(s2, ainv) : 1.f;
    M[0] = fa(fm(fm(q0, q0), S1), fm(fm(q2, q2), S2));
    M[2] = fa(fm(fm(q1, q1), S1), fm(fm(q3, q3), S2));
    M[1] = fa(fm(fm(S1, q0), q1), fm(fm(S2, q2), q3));
  } else {
    s1 = sqrtf(a);
    s2 = sqrtf(c);
    S1 = (fm(ainv, s1) > 1.f) ? 1.f / fm(ainv, s1) : 1.f;
    S2 = (fm(ainv, s2) > 1.f) ? 1.f / fm(ainv, s2) : 1.f;
    M[0] = S1; M[2] = S2; M[1] = 0.f;
  }
}

// nuclear 3-D helpers (radon_tgv_primal_dual_3d.py:190-284), results by value
__device__ __forceinline__ void diag2d(float a, float b, float c, float X[6]) {
  const float eps = 0.001f;
  const float o = c < a ? c : a;
  if (fm(b, b) / fm(o, o) > eps && fm(o, o) > 0.f) {
    const float dd = fa(a, c), e = fs(a, c);
    float f = fa(fm(fm(4.f, b), b), fm(e, e));
    f = f < 0.f ? 0.f : sqrtf(f);
    X[1] = (fs(dd, f) > 0.f) ? fm(fs(dd, f), 0.5f) : 0.f;
    X[0] = (fa(dd, f) > 0.f) ? fm(fa(dd, f), 0.5f) : 0.f;
    const float h = fm(fs(e, f), 0.5f);
    float v0 = 1.f, v1 = -h / b;
    const float n1 = hyp(v0, v1);
    v0 = v0 / n1; v1 = v1 / n1;
    X[2] = v0; X[3] = v1; X[4] = v1; X[5] = -v0;
  } else {
    X[0] = a; X[1] = c; X[2] = 1.f; X[3] = 0.f; X[4] = 0.f; X[5] = -1.f;
  }
}

__device__ __forceinline__ void eig3d(float a, float b, float c, float d, float e, float f, float out[3]) {
  const float pi = (float)3.14159265359;
  float c2 = -fa(fa(a, b), c);
  const float c1 = fs(fs(fs(fa(fa(fm(a, b), fm(a, c)), fm(b, c)), fm(d, d)), fm(e, e)), fm(f, f));
  const float c0 = fs(fs(fa(fa(fm(fm(a, f), f), fm(fm(b, e), e)), fm(fm(c, d), d)), fm(fm(a, b), c)),
                      fm(fm(fm(2.f, d), e), f));
  float p = (float)((double)fm(c2, c2) - 3.0 * (double)c1);
  const float cube = cube_f(c2);
  const float q = fa(fs(fm(-13.5f, c0), cube), fm(fm(4.5f, c2), c1));
  const float inner = fm(27.f, fa(fm(fm(fm(0.25f, c1), c1), fs(p, c1)), fm(c0, fa(q, fm(6.75f, c0)))));
  float phi = fm(1.f / 3.f, atan_f(sqrtf(inner) / q));
  if (q < 0.f) phi = fa(phi, pi / 3.f);
  const float x1 = fm(2.f, cos_f(phi));
  const float x2 = fm(2.f, cos_f(fa(phi, fm(2.f, pi) / 3.f)));
  const float x3 = fm(2.f, cos_f(fs(phi, fm(2.f, pi) / 3.f)));
  p = sqrtf(p) / 3.f;
  c2 = c2 / 3.f;
  out[0] = fs(fm(p, x1), c2); out[1] = fs(fm(p, x2), c2); out[2] = fs(fm(p, x3), c2);
}

__device__ __forceinline__ void cross3(float a1, float a2, float a3, float b1, float b2, float b3, float o[3]) {
  o[0] = fs(fm(a2, b3), fm(a3, b2));
  o[1] = fs(fm(b1, a3), fm(a1, b3));
  o[2] = fs(fm(a1, b2), fm(a2, b1));
}

__device__ __forceinline__ float norm3(const float v[3]) { return sqrtf(fa(fa(fm(v[0], v[0]), fm(v[1], v[1])), fm(v[2], v[2]))); }

// nuclear 3-D (update_NormV_Nucl, radon_tgv_primal_dual_3d.py:290-520): returns the
// symmetric 3x3 projection matrix M (xx, yy, zz, xy, xz, yz) applied to every channel,
// for A^T A = [a r t; r b d; t d c].
static __device__ void nucl3d_matrix(float a, float b, float c, float r, float t, float d, float ainv, float M[6]) {
  const float epsdt = 0.0001f, epsr = 0.0001f, epsoo = 0.0001f / ainv;
  const float ndt = fa(fm(d, d), fm(t, t));
  float oo = b < a ? b : a;
  float sig[3], v0[3], v1[3], v2[3], X[6], u1 = 1.f, u2 = 0.f;
  if (ndt < fm(fm(epsdt, oo), oo) && oo > epsoo) {
    diag2d(a, r, b, X);
    sig[0] = X[0]; sig[1] = X[1];
    sig[2] = (fm(c, c) < ndt) ? 1.f / epsdt : c;
    v0[0] = X[2]; v0[1] = X[3]; v0[2] = 0.f;
    v1[0] = X[4]; v1[1] = X[5]; v1[2] = 0.f;
    v2[0] = 0.f; v2[1] = 0.f; v2[2] = 1.f;
  } else if (oo < epsoo) {
    if (a >= b) {
      sig[0] = b; v0[0] = 0.f; v0[1] = 1.f; v0[2] = 0.f;
      diag2d(a, t, c, X);
      sig[1] = X[0]; sig[2] = X[1];
      v1[0] = X[2]; v1[1] = 0.f; v1[2] = X[3];
      v2[0] = X[4]; v2[1] = 0.f; v2[2] = X[5];
    } else {
      sig[0] = a; v0[0] = 1.f; v0[1] = 0.f; v0[2] = 0.f;
      diag2d(b, d, c, X);
      sig[1] = X[0]; sig[2] = X[1];
      v1[0] = 0.f; v1[1] = X[2]; v1[2] = X[3];
      v2[0] = 0.f; v2[1] = X[4]; v2[2] = X[5];
    }
  } else {
    // rotate about z so that the (x, z) entry vanishes (3-D :434-452)
    const float t1 = fs(fm(b, t), fm(d, r)), t2 = fs(fm(a, d), fm(t, r));
    u1 = d / sqrtf(ndt);
    u2 = t / sqrtf(ndt);
    const float bn = fa(fm(d, fa(fm(b, d), fm(r, t))), fm(t, fa(fm(a, t), fm(d, r)))) / ndt;
    const float an = fa(fm(t, t1), fm(d, t2)) / ndt;
    const float rn = fa(fm(-d, t1), fm(t, t2)) / ndt;
    const float dn = sqrtf(ndt);
    oo = bn < c ? bn : c;
    if (fabsf(rn) < fm(epsr, oo)) {
      diag2d(bn, dn, c, X);
      sig[0] = an; sig[1] = X[0]; sig[2] = X[1];
      v0[0] = 1.f; v0[1] = 0.f; v0[2] = 0.f;
      v1[0] = 0.f; v1[1] = X[2]; v1[2] = X[3];
      v2[0] = 0.f; v2[1] = X[4]; v2[2] = X[5];
    } else {
      eig3d(an, bn, c, rn, 0.f, dn, sig);
      cross3(fs(an, sig[0]), rn, 0.f, rn, fs(bn, sig[0]), dn, v0);
      float n = norm3(v0);
      v0[0] /= n; v0[1] /= n; v0[2] /= n;
      cross3(v0[0], v0[1], v0[2], 0.f, dn, fs(c, sig[1]), v1);
      n = norm3(v1);
      v1[0] /= n; v1[1] /= n; v1[2] /= n;
      cross3(v0[0], v0[1], v0[2], v1[0], v1[1], v1[2], v2);
      n = norm3(v2);
      v2[0] /= n; v2[1] /= n; v2[2] /= n;
    }
  }
  // eigenvectors back in the original frame (:476-479)
  float w[3][3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const float *vv = m == 0 ? v0 : (m == 1 ? v1 : v2);
    w[m][0] = fa(fm(u1, vv[0]), fm(u2, vv[1]));
    w[m][1] = fa(fm(-u2, vv[0]), fm(u1, vv[1]));
    w[m][2] = vv[2];
  }
  float S[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const float sg = sig[m] > 0.f ? sqrtf(sig[m]) : 0.f;
    S[m] = (fm(sg, ainv) > 1.f) ? 1.f / fm(ainv, sg) : 1.f;
  }
  // M = W diag(S) W^T (:500-507)
  const int ii[6] = {0, 1, 2, 0, 0, 1}, jj[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int q = 0; q < 6; ++q)
    M[q] = fa(fa(fm(fm(S[0], w[0][ii[q]]), w[0][jj[q]]), fm(fm(S[1], w[1][ii[q]]), w[1][jj[q]])),
              fm(fm(S[2], w[2][ii[q]]), w[2][jj[q]]));
}

// squared norm of one channel's w in the reference's weighting:
//  3-D Frobenius  w0^2+w1^2+w2^2+(1.4142 w3)^2+1.4142^2 (w4^2+w5^2)   (3-D :583)
//  3-D uncorr.    w0^2+w1^2+w2^2+(1.4142 w3)^2+(1.4142 w4)^2+w5^2      (3-D :603)
//  2-D Frobenius  w0^2+w1^2+(2 w2)^2                                    (2-D :232)
//  2-D uncorr.    w0^2+w1^2+(1.4142 w2)^2                               (2-D :254)
template <int DIM, int CPL>
__device__ __forceinline__ float wnorm2(const float *w) {
  if (DIM == 3) {
    const float q3 = 1.4142f * w[3], q4 = 1.4142f * w[4];
    const float q5 = (CPL == UNCORR) ? w[5] : 1.4142f * w[5];
    return w[0] * w[0] + w[1] * w[1] + w[2] * w[2] + q3 * q3 + q4 * q4 + q5 * q5;
  } else {
    const float q2 = (CPL == UNCORR) ? 1.4142f * w[2] : 2.f * w[2];
    return w[0] * w[0] + w[1] * w[1] + q2 * q2;
  }
}

// One component of update_p (3-D :734-757) at one voxel-slice: the divergence of
// the symmetric tensor w by forward differences (wa, wb, wc the row's entries at the
// voxel, wan, wbn, wcn at its x / y / z successor; fx, fy, fz: first pixel / row /
// slice, hx, hy, hz: a successor exists), then p + tau (v + div w).  k_update and the
// fused dual kernel both compute p through this function, by the same operations.
__device__ __forceinline__ float p_step3(float po, float vk, float wa, float wan, float wb, float wbn, float wc,
                                         float wcn, bool fx, bool hx, bool fy, bool hy, bool fz, bool hz, float tau,
                                         float stepsize) {
  float A = -wa, B = -wb, Cz = -wc;
  if (fx) A = 0.f;
  if (hx) A += wan;
  if (fy) B = 0.f;
  if (hy) B += wbn;
  if (fz) Cz = 0.f;
  if (hz) Cz += wcn;
  Cz /= stepsize;
  return po + tau * (vk + A + B + Cz);
}

// projections of the dual variables onto the norm balls (NormV / NormW of the
// coupling): vv, ww of the nC channels of one voxel, in place.
template <int DIM, bool TGV, int CPL, int CMAX>
__device__ __forceinline__ void dual_project(const IterParams &P, const int nC, float (&vv)[CMAX][DIM],
                                             float (&ww)[CMAX][DIM == 3 ? 6 : 3]) {
  constexpr int K = DIM, KW = DIM == 3 ? 6 : 3;
  if (CPL == UNCORR) {
#pragma unroll
    for (int c = 0; c < CMAX; ++c) {
      if (c >= nC) break;
      float n2 = 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) n2 += vv[c][k] * vv[c][k];
      const float nv = sqrtf(n2) * P.ainv1;
      if (nv > 1.f) {
#pragma unroll
        for (int k = 0; k < K; ++k) vv[c][k] = vv[c][k] / nv;
      }
      if (TGV) {
        const float nw = sqrtf(wnorm2<DIM, UNCORR>(ww[c])) * P.ainv0;
        if (nw > 1.f) {
#pragma unroll
          for (int k = 0; k < KW; ++k) ww[c][k] = ww[c][k] / nw;
        }
      }
    }
  } else {
    if (CPL == FROB) {
      float n2 = 0.f;
#pragma unroll
      for (int c = 0; c < CMAX; ++c) {
        if (c >= nC) break;
#pragma unroll
        for (int k = 0; k < K; ++k) n2 += vv[c][k] * vv[c][k];
      }
      const float nv = sqrtf(n2) * P.ainv1;
      if (nv > 1.f) {
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (c >= nC) break;
#pragma unroll
          for (int k = 0; k < K; ++k) vv[c][k] = vv[c][k] / nv;
        }
      }
    } else {  // NUCL: spectral projection of the C x K matrix
      if (DIM == 2) {
        float a = 0.f, b = 0.f, cc = 0.f;
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (c >= nC) break;
          a = fa(a, fm(vv[c][0], vv[c][0])); b = fa(b, fm(vv[c][0], vv[c][1])); cc = fa(cc, fm(vv[c][1], vv[c][1]));
        }
        float M[3];
        nucl2d_matrix(a, b, cc, P.ainv1, M);
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (c >= nC) break;
          const float v0 = vv[c][0], v1 = vv[c][1];
          vv[c][0] = fa(fm(v0, M[0]), fm(v1, M[1]));
          vv[c][1] = fa(fm(v0, M[1]), fm(v1, M[2]));
        }
      } else {
        float a = 0.f, b = 0.f, cc = 0.f, r = 0.f, tt = 0.f, dd = 0.f;
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (c >= nC) break;
          const float X = vv[c][0], Y = vv[c][1], Z = vv[c][DIM - 1];
          a = fa(a, fm(X, X)); b = fa(b, fm(Y, Y)); cc = fa(cc, fm(Z, Z));
          r = fa(r, fm(X, Y)); tt = fa(tt, fm(X, Z)); dd = fa(dd, fm(Y, Z));
        }
        float M[6];
        nucl3d_matrix(a, b, cc, r, tt, dd, P.ainv1, M);
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (c >= nC) break;
          const float A = vv[c][0], B = vv[c][1], Cc = vv[c][DIM - 1];
          vv[c][0] = fa(fa(fm(A, M[0]), fm(B, M[3])), fm(Cc, M[4]));
          vv[c][1] = fa(fa(fm(A, M[3]), fm(B, M[1])), fm(Cc, M[5]));
          vv[c][DIM - 1] = fa(fa(fm(A, M[4]), fm(B, M[5])), fm(Cc, M[2]));
        }
      }
    }
    if (TGV) {  // w: Frobenius coupling for both FROB and NUCL (3-D :1118-1124)
      float n2 = 0.f;
#pragma unroll
      for (int c = 0; c < CMAX; ++c) {
        if (c >= nC) break;
        n2 += wnorm2<DIM, FROB>(ww[c]);
      }
      const float nw = sqrtf(n2) * P.ainv0;
      if (nw > 1.f) {
#pragma unroll
        for (int c = 0; c < CMAX; ++c) {
          if (c >= nC) break;
#pragma unroll
          for (int k = 0; k < KW; ++k) ww[c][k] = ww[c][k] / nw;
        }
      }
    }
  }

}

// ===========================================================================
// k_dual: update_v (3-D :615-634, 2-D :265-284), update_w (3-D :637-660,
// 2-D :286-304), NormV / NormW (3-D :290-610, 2-D :98-258)
// thread = one (pixel, z); it owns all C channels of that voxel.
// ===========================================================================
template <int DIM, bool TGV, int CPL, int CMAX>
__device__ __forceinline__ void dual_body(const IterParams &P, long long bid) {
  constexpr int K = DIM, KW = DIM == 3 ? 6 : 3;
  const Dims d = P.d;
  const long long t = bid * blockDim.x + threadIdx.x;
  if (t >= (long long)d.N * d.N * d.Nz) return;
  const int pix = (int)(t / d.Nz);
  const int z = (int)(t - (long long)pix * d.Nz);
  const int y = pix / d.N, x = pix - y * d.N;
  const size_t vol = d.vol, S = d.S, rowS = (size_t)d.N * S;
  const float sigma = P.sigma;
  const float *__restrict__ ub = P.ubar;
  const float *__restrict__ pb = P.pbar;
  const int nC = min(CMAX, d.C - P.cbase);  // channels of this launch (channel groups for uncorrelated C > 8)

  float vv[CMAX][K], ww[CMAX][KW];
#pragma unroll
  for (int c = 0; c < CMAX; ++c) {
    if (c >= nC) break;
    const size_t i = (size_t)pix * S + (size_t)(P.cbase + c) * d.Nz + z;
    // gradient of ubar: forward differences, zero at the last index
    const float mu = -ub[i];
    float g[3];
    g[0] = (x < d.N - 1) ? mu + ub[i + S] : 0.f;
    g[1] = (y < d.N - 1) ? mu + ub[i + rowS] : 0.f;
    if (DIM == 3) g[2] = ((z < d.Nz - 1) ? mu + ub[i + 1] : 0.f) / P.stepsize;
    float pc[3];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      pc[k] = TGV ? pb[k * vol + i] : 0.f;
      vv[c][k] = P.v[k * vol + i] + sigma * (g[k] - pc[k]);
    }
    if (TGV) {
      // symmetrised gradient of pbar: backward differences, zero at index 0
      float a[3], b[3], cz[3];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        a[k] = x > 0 ? pc[k] - pb[k * vol + i - S] : 0.f;
        b[k] = y > 0 ? pc[k] - pb[k * vol + i - rowS] : 0.f;
        if (DIM == 3) cz[k] = (z > 0 ? pc[k] - pb[k * vol + i - 1] : 0.f) / P.stepsize;
      }
      float e[6];
      if (DIM == 3) {
        e[0] = a[0]; e[1] = b[1]; e[2] = cz[2];
        e[3] = 0.5f * (a[1] + b[0]);
        e[4] = 0.5f * (a[2] + cz[0]);
        e[5] = 0.5f * (b[2] + cz[1]);
      } else {
        e[0] = a[0]; e[1] = b[1];
        e[2] = 0.5f * (a[1] + b[0]);
      }
#pragma unroll
      for (int k = 0; k < KW; ++k) ww[c][k] = P.w[k * vol + i] + sigma * e[k];
    }
  }

  dual_project<DIM, TGV, CPL, CMAX>(P, nC, vv, ww);

  // ---- store
#pragma unroll
  for (int c = 0; c < CMAX; ++c) {
    if (c >= nC) break;
    const size_t i = (size_t)pix * S + (size_t)(P.cbase + c) * d.Nz + z;
#pragma unroll
    for (int k = 0; k < K; ++k) P.v[k * vol + i] = vv[c][k];
    if (TGV) {
#pragma unroll
      for (int k = 0; k < KW; ++k) P.w[k * vol + i] = ww[c][k];
    }
  }
}

}  // namespace gt
