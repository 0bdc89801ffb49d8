// Detector coordinates of the FP64 operator-norm estimate in fixed point (compiles for the host too).
//
// t = x X + y Y + off is a 64-bit integer with FIX fraction bits.  X, Y and off keep 32 bits more
// (X = (X.hi + X.lo 2^-32) 2^-FIX, X.lo in [0, 2^32)), so that x and y do not multiply a
// rounding of X and Y: t is off by at most 2^-(FIX + 1) from its last rounding and (x + y + 1)
// 2^-(FIX + 33) from X, Y and off.  In FP64 it is off by half an ulp of x X, of x X + y Y and of t,
// 2^-45 each from 2^8 on; fix_bits chooses FIX so that the fixed-point t is nowhere worse: errors of up to
// 1.2e-16 against 8e-14 for a 256^2 image and as many bins, 1.8e-15 against 1.3e-13 for 512^2.
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
  const long long q = (long long)((s - f) * 4294967296.0 + 0.5);  // 0 .. 2^32
  return {(long long)f + (q >> 32), (unsigned)q};
}

struct FixAngle {
  FixNum X, Y, off;  // off: half a unit of the last place added, for the rounding of t
};

template <int FIX>
GT_HD FixAngle fix_angle(double X, double Y, double off) {
  FixAngle a{to_fix<FIX>(X), to_fix<FIX>(Y), to_fix<FIX>(off)};
  const unsigned long long l = (unsigned long long)a.off.lo + 0x80000000ull;
  a.off.hi += (long long)(l >> 32);
  a.off.lo = (unsigned)l;
  return a;
}

// x X + y Y + off, rounded: hi; 0 <= x, y < 2^15
GT_HD FixNum fix_at(const FixAngle &a, int x, int y) {
  const unsigned long long l =
      (unsigned long long)(unsigned)x * a.X.lo + (unsigned long long)(unsigned)y * a.Y.lo + a.off.lo;
  return {x * a.X.hi + y * a.Y.hi + a.off.hi + (long long)(l >> 32), (unsigned)l};
}

// one pixel along the row
GT_HD void fix_step(FixNum &t, const FixNum &X) {
  const unsigned l = t.lo + X.lo;
  t.hi += X.hi + (l < t.lo);
  t.lo = l;
}

}  // namespace gt
