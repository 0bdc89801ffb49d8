// cos, atan and a few short expressions of floats, rounded once to float, without FP64 arithmetic
// (compiles for the host too).
//
// The nuclear-norm projection evaluates these in double and rounds once, and FP64 runs at 1/64 of
// the FP32 rate: that took most of its dual update.  Here
// a value is computed as an unevaluated sum h + l of two floats with a relative error below
// 2^-38 (bounds at each function), and accepted where every real number that close to h + l
// rounds to h (Ziv's test).  Otherwise, about once in 10^4 calls, the function returns false
// and the caller evaluates in double; so results are the same in all bits.  NaN goes through
// as NaN.  Dual update of 128^2 x 30 x 3: 64 -> 54 us after 100 iterations, 120 -> 58 us once
// the iterate is NaN, as the reference's projection can make it.
//
// Sums and products of such pairs: T. J. Dekker, "A floating-point technique for extending the
// available precision", Numer. Math. 18 (1971); the series are Taylor's.  Built with
// -fmad=false (-ffp-contract=off): every operation below rounds as written.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define GT_HD __device__ __forceinline__
#else
#define GT_HD inline
#endif

namespace gt {

struct F2 {
  float h, l;  // h + l, |l| <= half an ulp of h
};

GT_HD F2 f2_fast(float a, float b) {  // |a| >= |b| or a == 0
  const float s = a + b;
  return {s, b - (s - a)};
}

GT_HD F2 f2_sum(float a, float b) {
  const float s = a + b, t = s - a;
  return {s, (a - (s - t)) + (b - t)};
}

GT_HD F2 f2_mul(F2 a, F2 b) {
  const float p = a.h * b.h;
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  return f2_fast(p, e);
}

GT_HD F2 f2_add(F2 a, F2 b) {  // |a| >= |b|
  const F2 s = f2_fast(a.h, b.h);
  return f2_fast(s.h, s.l + (a.l + b.l));
}

// every real within 2^-38 |h| of h + l rounds to h
GT_HD bool f2_round(F2 v, float &r) {
  const float e = fabsf(v.h) * 0x1p-38f;
  r = v.h;
  return v.h + (v.l + e) == v.h && v.h + (v.l - e) == v.h;
}

// c^3 and sqrt(a^2 + b^2): relative errors below 2^-43.  Arguments whose low parts
// would underflow are scaled by a power of two, or declined.  NaN gives NaN: iterates of the
// nuclear projection can get there and stay.
GT_HD bool cube_round(float c, float &out) {
  const float a = fabsf(c);
  if (c != c) {
    out = c;
    return true;
  }
  if (!(a > 0x1p-41f && a < 0x1p33f)) return false;
  const bool small = a < 0x1p-15f;
  const F2 v{small ? c * 0x1p20f : c, 0.f};
  const bool ok = f2_round(f2_mul(f2_mul(v, v), v), out);
  if (small) out *= 0x1p-60f;
  return ok;
}

GT_HD bool hyp_round(float a, float b, float &out) {
  if (a != a || b != b) {
    out = a + b;
    return true;
  }
  const float m = fmaxf(fabsf(a), fabsf(b));
  const float k = m > 0x1p40f ? 0x1p-70f : m < 0x1p-28f ? 0x1p70f : 1.f;
  const F2 x{m * k, 0.f}, y{fminf(fabsf(a), fabsf(b)) * k, 0.f};
  const F2 s = f2_add(f2_mul(x, x), f2_mul(y, y));
  if (!(s.h > 0x1p-60f && s.h < 0x1p120f)) return false;
  const float r = sqrtf(s.h);
  const bool ok = f2_round(f2_fast(r, (fmaf(-r, r, s.h) + s.l) / (2.f * r)), out);
  out *= k < 1.f ? 0x1p70f : k > 1.f ? 0x1p-70f : 1.f;
  return ok && out > 0x1p-126f;
}

// |x| <= 3.9.  x = n pi/2 + r, |r| <= pi/4: x - n P1 is exact (n P1 within a factor 2 of x), the
// rest of n pi/2 to 2^-48 of r.  Both series are m (1 + z P(z)), z = r^2 <= 0.617; P's first
// three coefficients as pairs, its rest in float, where it is below 2^-18 of 1 (error 2^-40);
// the first term left out is below 2^-45.
GT_HD bool cos_round(float x, float &out) {
  if (x != x) {
    out = x;
    return true;
  }
  if (!(fabsf(x) <= 3.9f)) return false;
  const float n = rintf(x * 0x1.45f306p-1f);
  const F2 d = f2_sum(fmaf(-n, 0x1.921fb6p+0f, x), n * 0x1.777a5cp-25f);
  const F2 r = f2_fast(d.h, d.l + n * 0x1.ee59dap-50f);
  const int k = (int)n;
  const bool odd = k & 1;
  const F2 z = f2_mul(r, r);
  const float q = odd ? fmaf(z.h, fmaf(z.h, fmaf(z.h, -1.f / 1307674368000.f, 1.f / 6227020800.f), -1.f / 39916800.f),
                             1.f / 362880.f)
                      : fmaf(z.h, fmaf(z.h, fmaf(z.h, -1.f / 87178291200.f, 1.f / 479001600.f), -1.f / 3628800.f),
                             1.f / 40320.f);
  const F2 c2 = odd ? F2{-0x1.a01a02p-13f, 0x1.7f97fap-39f} : F2{-0x1.6c16c2p-10f, 0x1.27d27ep-35f};
  const F2 c1 = odd ? F2{0x1.111112p-7f, -0x1.ddddep-32f} : F2{0x1.555556p-5f, -0x1.555556p-30f};
  const F2 c0 = odd ? F2{-0x1.555556p-3f, 0x1.555556p-28f} : F2{-0.5f, 0.f};
  const float zq = z.h * q;
  F2 p = f2_fast(c2.h, c2.l + zq);
  p = f2_add(c1, f2_mul(z, p));
  p = f2_add(c0, f2_mul(z, p));
  F2 v = f2_add(F2{1.f, 0.f}, f2_mul(z, p));
  if (odd) v = f2_mul(r, v);
  if (k == 1 || k == 2 || k == -2) {
    v.h = -v.h;
    v.l = -v.l;
  }
  return f2_round(v, out);
}

// atan(k / 8)
#ifdef __CUDACC__
__device__
#endif
static const float ATAN8[18] = {0.f, 0.f, 0x1.fd5baap-4f, -0x1.54f424p-30f, 0x1.f5b76p-3f, -0x1.b4dfc8p-29f,
                                0x1.6f6194p-2f, 0x1.e4defp-30f, 0x1.dac67p-2f, 0x1.586ed4p-28f,
                                0x1.1e00bap-1f, 0x1.7bdfd6p-26f, 0x1.4978fap-1f, 0x1.934f7p-28f,
                                0x1.700a7cp-1f, 0x1.5e118cp-27f, 0x1.921fb6p+0f / 2, -0x1.777a5cp-26f};

// |y| > 1: pi/2 - atan(1 / |y|).  t in [0, 1]: atan(t) = atan(c) + atan(u), c = k / 8 nearest to t,
// u = (t - c) / (1 + t c), |u| <= 1/16 (t - c exact, the quotient to 2^-44).  atan(u) =
// u (1 + w (-1/3 + w B(w))), w = u^2 <= 2^-8: B in float is below 2^-18 of 1 (error 2^-41),
// the first term left out below 2^-43.
GT_HD bool atan_round(float y, float &out) {
  const float a = fabsf(y);
  if (!(a > 0.f)) {  // zero of either sign, NaN
    out = y;
    return true;
  }
  F2 t{a, 0.f};
  if (a > 1.f) {
    t.h = 1.f / a;
    t.l = fmaf(-t.h, a, 1.f) * t.h;  // a infinite: NaN, and the test below fails
  }
  const float k = rintf(t.h * 8.f), c = k * 0.125f;
  F2 num = f2_sum(t.h - c, t.l);
  const float tc = t.h * c;
  F2 den = f2_fast(1.f, tc);
  den = f2_fast(den.h, den.l + fmaf(t.l, c, fmaf(t.h, c, -tc)));
  const float inv = 1.f / den.h, u0 = num.h * inv;
  const float rem = fmaf(-u0, den.l, fmaf(-u0, den.h, num.h) + num.l);
  const F2 u = f2_fast(u0, rem * inv);
  const F2 w = f2_mul(u, u);
  const float b = fmaf(w.h, fmaf(w.h, -1.f / 11.f, 1.f / 9.f), -1.f / 7.f);
  const float wb = w.h * fmaf(w.h, b, 1.f / 5.f);
  const F2 g = f2_fast(-0x1.555556p-2f, 0x1.555556p-27f + wb);
  F2 v = f2_mul(u, f2_add(F2{1.f, 0.f}, f2_mul(w, g)));
  const int i = 2 * (int)k;
  if (i) v = f2_add(F2{ATAN8[i], ATAN8[i + 1]}, v);
  if (a > 1.f) v = f2_add(F2{0x1.921fb6p+0f, -0x1.777a5cp-25f}, F2{-v.h, -v.l});
  if (y < 0.f) {
    v.h = -v.h;
    v.l = -v.l;
  }
  return f2_round(v, out);
}

}  // namespace gt
