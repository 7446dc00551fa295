// The advective and diffusive terms of the momentum and temperature equations
// in 64-bit integers, for the form that is held to a tolerance rather than to
// the reference's operation order (src/fluid/update_velocity.c:11-192,
// src/temperature/update.c:11-87).
//
// GB300 issues one FP64 warp instruction per sub-partition every 70 to 80
// cycles, an integer addition every 1 to 2 and a 32 x 32 -> 64 multiply-add
// every 2 to 3: 38 of the 52 FP64 instructions of a cell's velocity update are
// the sums, differences and products of these terms, ~10 cycles each here.
//
// The terms are
//   A = - ax (sxm dxm + sxp dxp) - ay (sym dym + syp dyp)
//       + cp dxp - cm dxm + cy (dyp - dym),
// d the differences of the updated quantity f to its neighbours, s twice the
// velocities of the faces. The three values of f along a direction are taken at
// the largest exponent among them, as integers below 2^60: exact for values
// from 2^-7 of the largest one up, truncated at its 2^-60 below. So differences
// and second differences are exact for the most part; the two differences of a
// direction are shifted up together until the larger one has 62 bits, the second
// difference too, and the products' top 64 bits are formed from there. The
// velocities of a direction's faces have an exponent of their own. Each
// direction's advection and diffusion is a number with its own exponent until
// the final sum: on cells that are not square the coefficients of the two
// directions and their differences are the aspect and its square apart. (One
// exponent and one shift for both lost two bits for each doubling of the
// aspect: at 64 the error was 96 times the FP64 expressions', at 1/32 25 times.)
// cp and cm are equal, or (at a wall) one is twice the other, up to the rounding
// of the grid: what is left of cp dxp - cm dxm beside the second difference is a
// term of its own (ex), zero on a grid of equal spacings. No sum can overflow
// (bounds beside each line).
//
// Accuracy: the error of A is below that of the FP64 expressions, whose terms
// are rounded at 2^-53 each: 0.4 to 0.6 of it on square cells
// (tests/test_stencil_fixed.py), 0.8 or less at aspects from 1/512 to 512
// (tests/test_stencil_aspect.py; both against long double). Diffusion alone, on
// spacings that are powers of two, is the exact value rounded once either way.
#pragma once

#include "fft_fixed.cuh"

namespace sns {
namespace sfx {

// a in two signed words, a = hi 2^32 + lo; |a| <= 2^62
struct Split {
  int h, l;
};
FX_HD Split split(long long a) { return Split{fx::hi_part(a), fx::lo_part(a)}; }
// (a b + c d) 2^-64 rounded (the products of the low words, below half of the
// last bit, are left out); one product: |a|, |b| <= 2^62. Two: one factor of
// each at most 2^61.
FX_HD long long prod(Split a, Split b) {
  return fx::mw(a.h, b.h, fx::mw(a.l, b.h, fx::mw(a.h, b.l, 1ll << 31)) >> 32);
}
FX_HD long long prod2(Split a, Split b, Split c, Split d) {
  const long long m = fx::mw(c.l, d.h, fx::mw(c.h, d.l, fx::mw(a.l, b.h, fx::mw(a.h, b.l, 1ll << 31))));
  return fx::mw(a.h, b.h, fx::mw(c.h, d.h, m >> 32));
}
FX_HD unsigned long long bits_of(double d) {
  unsigned long long b;
#ifdef __CUDA_ARCH__
  b = (unsigned long long)__double_as_longlong(d);
#else
  __builtin_memcpy(&b, &d, 8);
#endif
  return b;
}
FX_HD int imax(int a, int b) { return a > b ? a : b; }
FX_HD int imin(int a, int b) { return a < b ? a : b; }

// v >> s, v << s; amounts of 64 and more shift everything out (as PTX's shr does)
FX_HD long long shr(long long v, int s) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
#else
  return v >> imin(s, 63);
#endif
}

// m 2^(e - 1082), |m| < 2^60: a double, its biased exponent e (a subnormal's m
// is half of what it is, far below any exponent in use)
struct Num {
  long long m;
  int e;
};
FX_HD Num num(double d) {
  const unsigned long long b = bits_of(d);
  const int e = (int)(b >> 52) & 0x7ff;
  const long long m = (long long)(((b & 0xfffffffffffffull) | (e ? 1ull << 52 : 0ull)) << 7), n = (long long)b >> 63;
  return Num{(m ^ n) - n, e};
}
// its integer at the exponent E >= e
FX_HD long long at(Num a, int E) { return shr(a.m, E - a.e); }

// exponents in use: 5 values whose largest one lies outside are left to FP64
// (all zeros are not: they are zeros at kExpLo)
constexpr int kExpLo = 1023 - 200, kExpHi = 1023 + 200;
FX_HD bool usable(int e) { return (unsigned)(e - kExpLo) <= (unsigned)(kExpHi - kExpLo) || e == 0; }

// v 2^e
struct Val {
  long long v;
  int e;
};
// their sum at the largest exponent; |v| < 2^63 together
FX_HD Val add(Val a, Val b) {
  const int t = a.e - b.e;
  return Val{shr(a.v, imax(-t, 0)) + shr(b.v, imax(t, 0)), imax(a.e, b.e)};
}
// (four at once: 512 x 1024 velocity update 31.6 us, two by two 32.8)
FX_HD Val add(Val a, Val b, Val c) {
  const int e = imax(imax(a.e, b.e), c.e);
  return Val{shr(a.v, e - a.e) + shr(b.v, e - b.e) + shr(c.v, e - c.e), e};
}
FX_HD Val add(Val a, Val b, Val c, Val d) {
  const int e = imax(imax(a.e, b.e), imax(c.e, d.e));
  return Val{shr(a.v, e - a.e) + shr(b.v, e - b.e) + (shr(c.v, e - c.e) + shr(d.v, e - d.e)), e};
}
// |v| < 2^63, e - 62 and e + 1 exponents of normal numbers
FX_HD double to_double(Val x) {
  const long long n = x.v >> 63;
  const unsigned long long a = (unsigned long long)((x.v ^ n) - n);
  const int lz = fx::clz64(a | 1ull) - 1;
  const unsigned long long r = ((a << lz) + 512) >> 10;  // 53 bits, or 2^53
  const unsigned long long bits =
      x.v == 0 ? 0 : ((unsigned long long)(62 + 1023 - 1 + x.e - lz) << 52) + r + ((unsigned long long)n << 63);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)bits);
#else
  double d;
  __builtin_memcpy(&d, &bits, 8);
  return d;
#endif
}

// a positive normal number m 2^(e - 63), m in [2^62, 2^63)
struct Coef {
  long long m;
  int e;
};
FX_HD bool coef_ok(double c) {
  const unsigned h = (unsigned)(bits_of(c) >> 52);  // negative numbers have bit 11 set
  return h - (unsigned)kExpLo <= (unsigned)(kExpHi - kExpLo);
}
FX_HD Coef coef(double c) {
  const unsigned long long b = bits_of(c);
  return Coef{(long long)(((b & 0xfffffffffffffull) | 1ull << 52) << 10), (int)(b >> 52) - 1022};
}
FX_HD Coef mul(Coef a, Coef b) {
  const long long h = prod(split(a.m >> 1), split(b.m >> 1));  // [2^58, 2^60]
  const int lz = fx::clz64((unsigned long long)h) - 1;
  return Coef{fx::shl(h, lz), a.e + b.e + 3 - lz};
}
FX_HD Coef quarter(Coef a) { return Coef{a.m, a.e - 2}; }
FX_HD long long down(long long m, int s) { return m >> imin(s, 63); }

// the coefficients, at an exponent for each direction: a cell of aspect a has
// 1/dx and 1/dy a factor of a apart, the diffusive coefficients a^2
struct Terms {
  Split ax, ay, cx, cy;
  int eax, eay, ecx, ecy;  // of the products' integers, without the exponents of s and f
  // cm is nearer to 2 cp (tm) or cp to 2 cm (tp) than they are to each other:
  // the second difference in x is dxp - dxm, or dxp / 2 - dxm, or dxp - dxm / 2
  bool tm, tp;
  Split ex;  // what is left of the x term, times dxp (tp) or dxm
  int ee;
};
// false: cp and cm too far apart (|ex| could exceed cx / 2), or exponents that
// a sum's double could not have
constexpr int kCoefExp = 300;
template <bool EQ>
FX_HD bool terms(Terms &k, Coef ax, Coef ay, Coef cp, Coef cm, Coef cy) {
  k.ax = split(-(ax.m >> 1));  // > -2^62
  k.ay = split(-(ay.m >> 1));
  k.eax = ax.e - 54 - 2044;
  k.eay = ay.e - 54 - 2044;
  // cp and cm at the larger exponent of the two, halved (< 2^62)
  const int eb = imax(cp.e, cm.e) + 1;
  const long long p = down(cp.m, eb - cp.e), m = down(cm.m, eb - cm.e);
  k.tm = m - p > (p >> 1);  // cm nearer to 2 cp than to cp
  k.tp = p - m > (m >> 1);
  // cp dxp - cm dxm = cx (second difference) + ex (dxp or dxm)
  Coef cx = k.tp ? cm : cp;
  if (k.tp | k.tm) cx.e += 1;
  if (!EQ) {
    const long long ex = k.tp ? p - 2 * m : k.tm ? 2 * p - m : p - m;
    const int up = fx::clz64((unsigned long long)(ex ^ (ex >> 63)) | 1ull) - 2;
    k.ex = split(fx::shl(ex, up));  // <= 2^62
    k.ee = eb - 59 - 1022 - up;
  }
  k.cx = split(cx.m >> 1);  // < 2^62
  k.cy = split(cy.m >> 1);
  k.ecx = cx.e - 58 - 1022;
  k.ecy = cy.e - 58 - 1022;
  auto in = [](Coef c) { return c.e >= -kCoefExp && c.e <= kCoefExp; };
  return m - p <= p + (p >> 1) && p - m <= m + (m >> 1) && in(ax) && in(ay) && in(cp) && in(cm) && in(cy);
}

// A, and the implicit directions' diffusion
struct Sum {
  Val A, G;
};
// the magnitude's bits, of the high word: differences below 2^-28 of the
// largest value stay where a shift by 30 brings them
FX_HD unsigned size(long long d) { return (unsigned)((int)(d >> 32) ^ (int)(d >> 63)); }
// the shift that brings such magnitudes (of 62 bits at most) below 2^62
FX_HD int room(unsigned m) {
#ifdef __CUDA_ARCH__
  return __clz((int)(m | 1u)) - 2;
#else
  return __builtin_clz(m | 1u) - 2;
#endif
}
// a direction's advective term s_m d_m + s_p d_p times the coefficient -a, from
// differences shifted up by g; |s| <= 2^61, |d| <= 2^62
FX_HD Val advective(Split dm, Split dp, int g, long long sm, long long sp, Split a, int e) {
  const long long t = fx::shl(prod2(split(sm), dm, split(sp), dp), 2);  // <= 2^62
  return Val{prod(split(t), a), e - 2 - g};                             // <= 2^60
}
FX_HD Val diffusive(long long d2, Split c, int e) {  // |d2| < 2^62
  const int g = fx::clz64((unsigned long long)(d2 ^ (d2 >> 63)) | 1ull) - 2;
  return Val{prod(split(fx::shl(d2, g)), c), e - g};  // <= 2^60
}
// differences of f along x and y and the velocities of the faces in that
// direction, at an exponent each; |s|, |d| <= 2^61
struct Line {
  long long dm, dp, sm, sp;
  int ed, es;
};
// EQ: equal spacings (ex = 0)
template <bool IMPX, bool IMPY, bool EQ>
FX_HD Sum sum(const Terms &k, const Line &X, const Line &Y) {
  const int gx = room(size(X.dm) | size(X.dp)), gy = room(size(Y.dm) | size(Y.dp));
  const Split xm = split(fx::shl(X.dm, gx)), xp = split(fx::shl(X.dp, gx));
  const Split ym = split(fx::shl(Y.dm, gy)), yp = split(fx::shl(Y.dp, gy));
  const Val ax = advective(xm, xp, gx, X.sm, X.sp, k.ax, k.eax + X.es + X.ed);
  const Val ay = advective(ym, yp, gy, Y.sm, Y.sp, k.ay, k.eay + Y.es + Y.ed);  // <= 2^60
  Val x = diffusive((k.tm ? X.dp >> 1 : X.dp) - (k.tp ? X.dm >> 1 : X.dm), k.cx, k.ecx + X.ed);
  const Val y = diffusive(Y.dp - Y.dm, k.cy, k.ecy + Y.ed);
  if (!EQ) x = add(x, Val{prod(k.tp ? xp : xm, k.ex), k.ee + X.ed - gx});  // <= 2^61
  // sums of at most 2^62 + 2^60
  if (IMPX && IMPY) return Sum{add(ax, ay), add(x, y)};
  if (IMPX) return Sum{add(ax, ay, y), x};
  if (IMPY) return Sum{add(ax, ay, x), y};
  return Sum{add(ax, ay, x, y), Val{0, 0}};
}

// the interpolation weights of a vertical velocity (in (0, 1)) times 2^62
struct Weights {
  Split m, p;
};
FX_HD Weights weights(double fm, double fp) {
  const Coef a = coef(fm), b = coef(fp);  // e <= 0
  return Weights{split(down(a.m, 1 - a.e)), split(down(b.m, 1 - b.e))};
}
FX_HD bool weights_ok(double fm, double fp) { return coef_ok(fm) && coef_ok(fp) && fm < 1.0 && fp < 1.0; }
// twice the weighted mean of a and b; EQ: both weights 1/2
template <bool EQ>
FX_HD long long twice_mean(const Weights &w, long long a, long long b) {
  if (EQ) return a + b;
  return fx::shl(prod(split(fx::shl(a, 2)), w.m) + prod(split(fx::shl(b, 2)), w.p), 1);
}

FX_HD int top(Num a, Num b) { return imax(a.e, b.e); }
FX_HD int top(Num a, Num b, Num c, Num d) { return imax(top(a, b), top(c, d)); }
// three values along a direction at the largest exponent of theirs
struct Three {
  long long m, c, p;
  int e;
};
FX_HD Three three(Num m, Num c, Num p) {
  const int e = imax(imax(top(m, p), c.e), kExpLo);
  return Three{at(m, e), at(c, e), at(p, e), e};
}

// the velocities that a cell reads (l: column x-1, r: x+1, m: row y-1, n: row
// y+1); false: out of range
struct Vels {
  Num ul, u0, u1, um0, um1, u0n, vl, v0, vr, vm, v0n, vln;
};
FX_HD bool vels(Vels &o, Num ul, Num u0, Num u1, Num um0, Num um1, Num u0n, Num vl, Num v0, Num vr, Num vm, Num v0n,
                Num vln) {
  o = Vels{ul, u0, u1, um0, um1, u0n, vl, v0, vr, vm, v0n, vln};
  return usable(imax(top(ul, u0, u1, um0), top(um1, u0n))) && usable(imax(top(vl, v0, vr, vm), top(v0n, vln)));
}
template <bool IMPX, bool IMPY, bool EQ>
FX_HD Sum sum_ux(const Terms &k, const Weights &w, const Vels &v) {
  const Three x = three(v.ul, v.u0, v.u1), y = three(v.um0, v.u0, v.u0n);
  const int e = imax(top(v.vl, v.v0, v.vln, v.v0n), kExpLo);
  return sum<IMPX, IMPY, EQ>(k, Line{x.c - x.m, x.p - x.c, x.m + x.c, x.c + x.p, x.e, x.e},
                             Line{y.c - y.m, y.p - y.c, twice_mean<EQ>(w, at(v.vl, e), at(v.v0, e)),
                                  twice_mean<EQ>(w, at(v.vln, e), at(v.v0n, e)), y.e, e});
}
template <bool IMPX, bool IMPY, bool EQ>
FX_HD Sum sum_uy(const Terms &k, const Vels &v) {
  const Three x = three(v.vl, v.v0, v.vr), y = three(v.vm, v.v0, v.v0n);
  const int e = imax(top(v.um0, v.u0, v.um1, v.u1), kExpLo);
  return sum<IMPX, IMPY, EQ>(
      k, Line{x.c - x.m, x.p - x.c, at(v.um0, e) + at(v.u0, e), at(v.um1, e) + at(v.u1, e), x.e, e},
      Line{y.c - y.m, y.p - y.c, y.m + y.c, y.c + y.p, y.e, y.e});
}
// temperature: left, here, right, below, above; the face velocities; false:
// out of range
template <bool IMPX, bool IMPY, bool EQ>
FX_HD bool sum_temp(Sum &r, const Terms &k, Num l, Num c, Num rt, Num d, Num u, Num ul, Num ur, Num vd, Num vu) {
  const Three x = three(l, c, rt), y = three(d, c, u);
  const int eu = top(ul, ur), ev = top(vd, vu), ex = imax(eu, kExpLo), ey = imax(ev, kExpLo);
  r = sum<IMPX, IMPY, EQ>(
      k, Line{x.c - x.m, x.p - x.c, fx::shl(at(ul, ex), 1), fx::shl(at(ur, ex), 1), x.e, ex},
      Line{y.c - y.m, y.p - y.c, fx::shl(at(vd, ey), 1), fx::shl(at(vu, ey), 1), y.e, ey});
  return usable(imax(top(l, c, rt, d), u.e)) && usable(eu) && usable(ev);
}

}  // namespace sfx
}  // namespace sns
