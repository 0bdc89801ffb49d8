// Detector coordinates of the FP64 operator-norm estimate in fixed point (compiles for the host too).
//
// t = x X + y Y + off is a 64-bit integer with FIX fraction bits.  X, Y and off keep 16 bits more
// (X = (X.hi + X.lo 2^-16) 2^-FIX, X.lo in [0, 2^16)), so that x and y do not multiply a
// rounding of X and Y at the last place: t is off by at most 2^-(FIX + 1) from its last rounding and
// (x + y + 1) 2^-(FIX + 17) from X, Y and off, a 64th of that for a 512^2 image.  In FP64 it is off by half
// an ulp of x X, of x X + y Y and of t, 2^-45 each from 2^8 on; fix_bits chooses FIX so that
// the fixed-point t is nowhere worse: errors of up to 1.2e-16 against 7e-14 for a 256^2 image and as many
// bins, 1.8e-15 against 1.3e-13 for 512^2.
#pragma once
#include <math.h>

#ifndef GT_HD
#ifdef __CUDACC__
#define GT_HD __device__ __forceinline__
#else
#define GT_HD inline
#endif
#endif

namespace gt {

// fraction bits for coordinates below t in magnitude (t 2^FIX < 2^62); 0: FP64
inline int fix_bits(long long t) { return t < (1 << 10) ? 52 : t < (1 << 14) ? 48 : t < (1 << 18) ? 44 : 0; }

struct FixNum {
  long long hi;
  unsigned lo;
};

template <int FIX>
GT_HD FixNum to_fix(double v) {
  const double s = v * (double)(1ll << FIX), f = floor(s);
  const unsigned q = (unsigned)((s - f) * 65536.0 + 0.5);  // 0 .. 2^16
  return {(long long)f + (q >> 16), q & 0xffffu};
}

struct FixAngle {
  long long X, Y, off;
  unsigned xl, yl, ol;  // their low parts; ol with half a unit of the last place for the rounding of t
};

GT_HD FixAngle fix_angle(FixNum X, FixNum Y, FixNum off) {
  return {X.hi, Y.hi, off.hi, X.lo, Y.lo, off.lo + 0x8000u};
}

// x X + y Y + off, rounded (hi); 0 <= x, y < 2^15: the low parts' sum stays below 2^32
GT_HD FixNum fix_at(const FixAngle &a, unsigned x, unsigned y) {
  const unsigned l = x * a.xl + y * a.yl + a.ol;
  const unsigned long long h = (unsigned long long)a.X * x + (unsigned long long)a.Y * y + a.off + (l >> 16);
  return {(long long)h, l << 16};  // lo: the rest of the low parts, as a fraction of 2^32
}

// one pixel along the row
GT_HD void fix_step(FixNum &t, const FixAngle &a) {
  const unsigned l = t.lo + (a.xl << 16);
  t.hi += a.X + (l < t.lo);
  t.lo = l;
}

}  // namespace gt
