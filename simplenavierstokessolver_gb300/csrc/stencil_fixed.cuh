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
// velocities of the faces. The values of f that a cell reads are taken at the
// largest exponent among them, as integers below 2^60: exact for values from
// 2^-7 of the largest one up, truncated at its 2^-60 below. So differences and
// second differences are exact for the most part; the former are shifted up
// together until the largest has 62 bits, the latter too, and the products'
// top 64 bits are formed from there. The other velocity's values have an
// exponent of their own. cp and cm are equal, or (at a wall) one is twice the other, up to
// the rounding of the grid: what is left of cp dxp - cm dxm beside the second
// difference is a term of its own (ex), zero on a grid of equal spacings. No
// sum can overflow (bounds beside each line).
//
// Accuracy: the error of A is below that of the FP64 expressions, whose terms
// are rounded at 2^-53 each (tests/test_stencil_fixed.py measures both against
// long double: 0.4 to 0.6 of it).
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
// their sum at the larger exponent; |v| <= 2^62 together
FX_HD Val add(Val a, Val b) {
  const int t = a.e - b.e;
  return Val{shr(a.v, imax(-t, 0)) + shr(b.v, imax(t, 0)), imax(a.e, b.e)};
}
// |v| <= 2^62, e - 62 and e + 1 exponents of normal numbers
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

// the coefficients: the advective terms' at one exponent, the second
// differences' at another, or (where only one direction is implicit, and they
// go different ways) at one each
struct Terms {
  Split ax, ay, cx, cy;
  int ea, ecx, ecy;  // of the integers, without the exponents of s and f
  // cm is nearer to 2 cp (tm) or cp to 2 cm (tp) than they are to each other:
  // the second difference in x is dxp - dxm, or dxp / 2 - dxm, or dxp - dxm / 2
  bool tm, tp;
  Split ex;  // what is left of the x term, times dxp (tp) or dxm
  int ee;
};
// false: cp and cm too far apart (|ex| could exceed cx / 2), or exponents that
// a sum's double could not have
constexpr int kCoefExp = 300;
template <bool APART>
FX_HD bool terms(Terms &k, Coef ax, Coef ay, Coef cp, Coef cm, Coef cy) {
  const int ta = imax(ax.e, ay.e) + 1;
  k.ax = split(down(ax.m, ta - ax.e));  // <= 2^62
  k.ay = split(down(ay.m, ta - ay.e));
  k.ea = ta - 55 - 2044;
  // cp and cm at the larger exponent of the two, halved (< 2^62)
  const int eb = imax(cp.e, cm.e) + 1;
  const long long p = down(cp.m, eb - cp.e), m = down(cm.m, eb - cm.e);
  k.tm = m - p > (p >> 1);  // cm nearer to 2 cp than to cp
  k.tp = p - m > (m >> 1);
  // cp dxp - cm dxm = cx (second difference) + ex (dxp or dxm)
  Coef cx = k.tp ? cm : cp;
  if (k.tp | k.tm) cx.e += 1;
  const long long ex = k.tp ? p - 2 * m : k.tm ? 2 * p - m : p - m;
  const int up = fx::clz64((unsigned long long)(ex ^ (ex >> 63)) | 1ull) - 2;
  k.ex = split(fx::shl(ex, up));  // <= 2^62
  k.ee = eb - 59 - 1022 - up;
  const int tx = (APART ? cx.e : imax(cx.e, cy.e)) + 2, ty = APART ? cy.e + 2 : tx;
  k.cx = split(down(cx.m, tx - cx.e));  // <= 2^61
  k.cy = split(down(cy.m, ty - cy.e));
  k.ecx = tx - 59 - 1022;
  k.ecy = ty - 59 - 1022;
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
// f's differences at the exponent ef, s at exponents whose largest one is ec,
// by tx and ty above those of sx and sy; |s|, |d| <= 2^61. EQ: equal spacings
// (ex = 0)
template <bool IMPX, bool IMPY, bool EQ>
FX_HD Sum sum(const Terms &k, int ef, int ec, int tx, int ty, long long dxm, long long dxp, long long dym,
              long long dyp, long long sxm, long long sxp, long long sym, long long syp) {
  const int g = room(size(dxm) | size(dxp) | size(dym) | size(dyp));
  const Split xm = split(fx::shl(dxm, g)), xp = split(fx::shl(dxp, g));
  const Split ym = split(fx::shl(dym, g)), yp = split(fx::shl(dyp, g));
  const long long sx = shr(prod2(split(sxm), xm, split(sxp), xp), tx);  // <= 2^60
  const long long sy = shr(prod2(split(sym), ym, split(syp), yp), ty);
  const Val adv{-prod2(split(sx), k.ax, split(sy), k.ay), k.ea + ec + ef - g};  // <= 2^59
  const long long d1 = (k.tm ? dxp >> 1 : dxp) - (k.tp ? dxm >> 1 : dxm), d2 = dyp - dym;  // < 2^62
  constexpr bool APART = IMPX != IMPY;
  const int g1 = room(APART ? size(d1) : size(d1) | size(d2)), g2 = APART ? room(size(d2)) : g1;
  const Split e1 = split(fx::shl(d1, g1)), e2 = split(fx::shl(d2, g2));
  Val x{0, k.ecx + ef - g1}, y{0, k.ecy + ef - g2};
  if (!APART) {
    x.v = prod2(e1, k.cx, e2, k.cy);  // <= 2^60
  } else {
    x.v = prod(e1, k.cx);
    y.v = prod(e2, k.cy);
  }
  if (!EQ) x = add(x, Val{prod(k.tp ? xp : xm, k.ex), k.ee + ef - g});  // <= 2^60 + 2^60
  Sum r;
  r.G = Val{0, 0};
  if (IMPX && IMPY) {
    r.A = adv;
    r.G = x;
  } else if (IMPX) {
    r.A = add(adv, y);
    r.G = x;
  } else if (IMPY) {
    r.A = add(adv, x);
    r.G = y;
  } else {
    r.A = add(adv, x);
  }
  return r;
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

FX_HD int exponent(Num a, Num b, Num c, Num d, Num e) { return imax(imax(imax(a.e, b.e), imax(c.e, d.e)), e.e); }

// the velocities that a cell reads (l: column x-1, r: x+1, m: row y-1, n: row
// y+1), at one exponent each; false: out of range
struct Vels {
  long long ul, u0, u1, um0, um1, u0n, vl, v0, vr, vm, v0n, vln;
  int eu, ev, ec, tu, tv;  // ec: the larger one, by tu and tv above theirs
};
FX_HD bool vels(Vels &o, Num ul, Num u0, Num u1, Num um0, Num um1, Num u0n, Num vl, Num v0, Num vr, Num vm, Num v0n,
                Num vln) {
  const int a = imax(exponent(ul, u0, u1, um0, um1), u0n.e), b = imax(exponent(vl, v0, vr, vm, v0n), vln.e);
  const int eu = imax(a, kExpLo), ev = imax(b, kExpLo);
  o = Vels{at(ul, eu), at(u0, eu), at(u1, eu), at(um0, eu), at(um1, eu),       at(u0n, eu),      at(vl, ev),
           at(v0, ev), at(vr, ev), at(vm, ev), at(v0n, ev), at(vln, ev),       eu,               ev,
           imax(eu, ev), imax(ev - eu, 0), imax(eu - ev, 0)};
  return usable(a) && usable(b);
}
template <bool IMPX, bool IMPY, bool EQ>
FX_HD Sum sum_ux(const Terms &k, const Weights &w, const Vels &v) {
  return sum<IMPX, IMPY, EQ>(k, v.eu, v.ec, v.tu, v.tv, v.u0 - v.ul, v.u1 - v.u0, v.u0 - v.um0, v.u0n - v.u0, v.ul + v.u0,
                         v.u0 + v.u1, twice_mean<EQ>(w, v.vl, v.v0), twice_mean<EQ>(w, v.vln, v.v0n));
}
template <bool IMPX, bool IMPY, bool EQ>
FX_HD Sum sum_uy(const Terms &k, const Vels &v) {
  return sum<IMPX, IMPY, EQ>(k, v.ev, v.ec, v.tu, v.tv, v.v0 - v.vl, v.vr - v.v0, v.v0 - v.vm, v.v0n - v.v0, v.um0 + v.u0,
                         v.um1 + v.u1, v.vm + v.v0, v.v0 + v.v0n);
}
// temperature: left, here, right, below, above; the face velocities; false:
// out of range
template <bool IMPX, bool IMPY, bool EQ>
FX_HD bool sum_temp(Sum &r, const Terms &k, Num l, Num c, Num rt, Num d, Num u, Num ul, Num ur, Num vd, Num vu) {
  const int ef = exponent(l, c, rt, d, u), ev = imax(imax(ul.e, ur.e), imax(vd.e, vu.e));
  const int E = imax(ef, kExpLo), ec = imax(ev, kExpLo);
  const long long C = at(c, E);
  r = sum<IMPX, IMPY, EQ>(k, E, ec, 0, 0, C - at(l, E), at(rt, E) - C, C - at(d, E), at(u, E) - C,
                          fx::shl(at(ul, ec), 1), fx::shl(at(ur, ec), 1), fx::shl(at(vd, ec), 1),
                          fx::shl(at(vu, ec), 1));
  return usable(ef) && usable(ev);
}

}  // namespace sfx
}  // namespace sns
