// Host-side numerics shared by the plain path (sns_api.cpp) and the batched
// FP32-stencil engine (batch_api.cpp). Compiled without floating-point
// contraction: these values feed kernels that must reproduce the reference's
// rounding.
#pragma once

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <vector>

namespace sns {

constexpr double kPiRef = 3.1415926535897932;  // include/common.h:7 of the reference

// src/param/init.c:124-195: face/centre coordinates and spacings (0-based
// arrays: xf[i-1] = XF(i), xc[i] = XC(i), dxf[i-1] = DXF(i), dxc[i-1] = DXC(i))
inline void make_grid(int itot, int jtot, double lx, double ly, double stretch_in, double *xf, double *xc,
                      double *dxf, double *dxc, double *yf, double *yc, double *dy) {
  int stretch = (int)stretch_in;
  if (stretch < 0) stretch = 0;
  if (stretch >= itot / 2) {
    const double dx = lx / itot;
    for (int i = 1; i <= itot + 1; i++) xf[i - 1] = 1. * (i - 1) * dx;
  } else {
    for (int i = 1; i <= itot + 1; i++) xf[i - 1] = cos(kPiRef * (1. * (i - 1) + stretch) / (itot + 2. * stretch));
    const double mn = xf[0], mx = xf[itot];
    for (int i = 1; i <= itot + 1; i++) xf[i - 1] = lx * (xf[i - 1] - mn) / (mx - mn);
  }
  xf[0] = 0.;
  xf[itot] = lx;
  for (int i = 1; i <= itot; i++) dxf[i - 1] = xf[i] - xf[i - 1];
  xc[0] = xf[0];
  for (int i = 1; i <= itot; i++) xc[i] = 0.5 * (xf[i - 1] + xf[i]);
  xc[itot + 1] = xf[itot];
  for (int i = 1; i <= itot + 1; i++) dxc[i - 1] = xc[i] - xc[i - 1];
  *dy = ly / jtot;
  if (yf)
    for (int j = 1; j <= jtot + 1; j++) yf[j - 1] = 1. * (j - 1) * (*dy);
  if (yc)
    for (int j = 1; j <= jtot; j++) yc[j - 1] = 0.5 * (2 * j - 1) * (*dy);
}

// Thomas forward elimination of a constant matrix (src/linalg.c:11-24), the
// RHS-independent part: normalised upper diagonal and 1/pivot, with 1/pivot
// = +0 marking the |pivot| < DBL_EPSILON rows that the reference zeroes.
inline void factorize(int n, const double *l, const double *d, const double *u, double *inv, double *up) {
  up[0] = u[0] / d[0];
  inv[0] = 0.0;
  for (int i = 1; i <= n - 1; i++) {
    double v = d[i] - l[i] * up[i - 1];
    if (std::fabs(v) < DBL_EPSILON) {
      up[i] = 0.;
      inv[i] = 0.;
    } else {
      v = 1. / v;
      up[i] = v * u[i];
      inv[i] = v;
    }
  }
}

// Rows of a Thomas sweep after which a change of its starting value has shrunk
// below 2^-80 of it (the last 2^-27 let the roundings of two sweeps meet), in
// either direction and from any row: a change of the previous value reaches
// the next one times l_i inv_i (elimination) or up_i (substitution). n where
// some row does not shrink it.
constexpr double kForgotten = 0x1p-80;
inline int warm_rows(int n, const double *l, const double *inv, const double *up) {
  int worst = 0;
  for (int dir = 0; dir < 2; dir++) {
    double prod = 1.0;
    int first = 1;  // the window first .. i
    for (int i = 1; i < n; i++) {
      const int a = dir ? n - 1 - i : i;
      const double c = std::fabs(dir ? up[a] : l[a] * inv[a]);
      if (!(c < 1.0)) return n;
      if (c < kForgotten) {  // forgotten in this row
        prod = 1.0;
        first = i + 1;
        worst = std::max(worst, 1);
        continue;
      }
      prod *= c;
      while (first < i) {  // the shortest window that still shrinks enough
        const int b = dir ? n - 1 - first : first;
        const double shorter = prod / std::fabs(dir ? up[b] : l[b] * inv[b]);
        if (!(shorter < kForgotten)) break;
        prod = shorter;
        first++;
      }
      worst = std::max(worst, i - first + 1);
    }
  }
  return worst;
}

// exp(-2 pi i t/n) with the CPU FFT's rule: exact at multiples of pi/2, libm
// cos/sin evaluated only on [0, pi/4]
inline void twiddle(int n, int t, double *re, double *im) {
  const long t4 = 4L * t;
  const long q = t4 / n;
  const long r = t4 - q * (long)n;
  double c, s;
  if (2 * r <= n) {
    const double a = (3.14159265358979323846 * (double)r) / (2.0 * (double)n);
    c = std::cos(a);
    s = std::sin(a);
  } else {
    const double a = (3.14159265358979323846 * (double)(n - r)) / (2.0 * (double)n);
    c = std::sin(a);
    s = std::cos(a);
  }
  double cq, sq;
  switch (q & 3) {
    case 0: cq = c; sq = s; break;
    case 1: cq = -s; sq = c; break;
    case 2: cq = -c; sq = -s; break;
    default: cq = s; sq = -c; break;
  }
  *re = cq;
  *im = -sq;
}

inline std::vector<double> twiddle_table(int n) {
  std::vector<double> tw(2 * (size_t)n);
  for (int t = 0; t < n; t++) twiddle(n, t, &tw[2 * t], &tw[2 * t + 1]);
  return tw;
}

// Division by a divisor known in advance (Brisebarre, Muller, Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", IEEE Trans. Computers 53(8), 2004): with zh = RN(1/y)
// and zl close to 1/y - zh, RN(x zh + RN(x zl)), a product and a fused
// multiply-add, is RN(x/y) for every x (no over- or underflow) unless x/y lies
// very close to the midpoint of two neighbouring doubles. Before its last
// rounding that sum is off by at most 2 2^-54 ulp of the quotient with
// zl = RN(1/y - zh) (RN(x zl): 2^-54, as |x zl| < 1 ulp; zl: 2^-54) and by
// (2 + 2 k) 2^-54 ulp with a zl k ulps further. With 53-bit integer
// significands X and Y a midpoint M (odd, 54 bits) is |X 2^53 - M Y| / 2Y ulp
// away if X >= Y, |X 2^54 - M Y| / 2Y if X < Y, so only numerators X for which
// that integer is at most 2 + 2 k can fail. They solve M Y = -D (mod 2^53 or
// 2^54), a few X per D: all are formed here and tried, for zl and, where it
// fails (one divisor in 200), its neighbours up to k = 3.
// Returns false when no zl passes (or y is not normal and positive).
inline bool invariant_divisor(double y, double *zh_out, double *zl_out) {
  int ey;
  if (!(y > 0.0) || !std::isnormal(y)) return false;
  const uint64_t Y = (uint64_t)std::ldexp(std::frexp(y, &ey), 53);
  const double ys = (double)Y, zh = 1.0 / ys;
  const int t = __builtin_ctzll(Y);  // Y = 2^t Yo
  const uint64_t Yo = Y >> t;
  uint64_t yinv = Yo;  // inverse of Yo modulo 2^64 by Newton's iteration
  for (int k = 0; k < 5; k++) yinv *= 2 - Yo * yinv;
  const double zl0 = std::fma(-zh, ys, 1.0) / ys;  // the residual is exact
  // whether the pair (zh, zl) divides every X with a midpoint at most Dmax away
  auto divides = [&](double zl, int Dmax) {
    for (int w = 53; w <= 54; w++)  // X >= Y, X < Y
      for (int D = -Dmax; D <= Dmax; D++) {
        // M Y = -D (mod 2^w) needs 2^t | D
        if (D == 0 || t > 3 || D % (1 << t)) continue;
        // M = -(D / 2^t) / Yo modulo 2^(w - t), odd, in [2^53, 2^54)
        const uint64_t mod = 1ull << (w - t), lo = 1ull << 53;
        const uint64_t m0 = ((uint64_t)(-(int64_t)(D / (1 << t))) * yinv) & (mod - 1);
        for (uint64_t M = m0 >= lo ? m0 : m0 + (lo - m0 + mod - 1) / mod * mod; M < 2 * lo; M += mod) {
          if (!(M & 1)) continue;
          const __int128 n = (__int128)M * Y + D;
          if (n <= 0 || (n & (((__int128)1 << w) - 1)) != 0) continue;
          const uint64_t X = (uint64_t)(n >> w);
          if (X >> 52 != 1 || (w == 53) != (X >= Y)) continue;
          const double x = (double)X;
          if (std::fma(x, zh, x * zl) != x / ys) return false;
        }
      }
    return true;
  };
  for (int k = 0; k < 7; k++) {  // zl0, then one, two, three ulps up and down
    double zl = zl0;
    for (int i = 0; i < (k + 1) / 2; i++) zl = std::nextafter(zl, k % 2 ? 1.0 : -1.0);
    if (divides(zl, 2 + 2 * ((k + 1) / 2))) {
      *zh_out = std::ldexp(zh, 53 - ey);
      *zl_out = std::ldexp(zl, 53 - ey);
      return true;
    }
  }
  return false;
}

// exp(-2 pi i t / n), t < n (a power of two), scaled by 2^62 and split for the
// fixed-point DFT (fft_fixed.cuh, Tw; n >= 8): four words per t, real high and low,
// imaginary high and low, the low ones in (-2^31, 2^31). Sine and cosine of an
// angle in [0, pi/4] by their Taylor series in 112-bit fixed point, so the
// words are the same on every host.
inline std::vector<int32_t> fixed_twiddles(int n) {
  typedef unsigned __int128 u128;
  auto mulq = [](u128 a, u128 b) -> u128 {  // a b / 2^112 (truncated), a, b <= 2^112
    a <<= 8;
    b <<= 8;
    const u128 m = ((u128)1 << 64) - 1, ah = a >> 64, al = a & m, bh = b >> 64, bl = b & m;
    const u128 mid = ah * bl, mid2 = al * bh;
    return ah * bh + (mid >> 64) + (mid2 >> 64) + (((mid & m) + (mid2 & m) + ((al * bl) >> 64)) >> 64);
  };
  const u128 one = (u128)1 << 112;
  const u128 pi4 = ((u128)0xC90FDAA22168C234ull << 48) | (0xC4C6628B80DC1CD1ull >> 16);  // pi/4 in units of 2^-112
  auto sincos = [&](int num, u128 *s, u128 *c) {  // angle (pi/4) num / n, num <= n
    const u128 x = pi4 / (unsigned)n * (unsigned)num, x2 = mulq(x, x);
    u128 ts = x, tc = one, ss = x, cc = one;
    for (int k = 1; k < 16 && tc; k++) {
      tc = mulq(tc, x2) / (unsigned)((2 * k - 1) * (2 * k));
      ts = mulq(ts, x2) / (unsigned)((2 * k) * (2 * k + 1));
      if (k & 1) {
        cc -= tc;
        ss -= ts;
      } else {
        cc += tc;
        ss += ts;
      }
    }
    *s = ss;
    *c = cc;
  };
  // one octant: angles (pi/2) r / n, r = 4 t' <= n / 2 (r = 0, n / 2 alone below n = 8)
  const int noct = n / 8 + 1;
  std::vector<int64_t> so(noct), co(noct);
  for (int k = 0; k < noct; k++) {
    u128 s, c;
    sincos(8 * k, &s, &c);
    so[k] = (int64_t)((s + ((u128)1 << 49)) >> 50);
    co[k] = (int64_t)((c + ((u128)1 << 49)) >> 50);
  }
  std::vector<int32_t> out(4 * (size_t)n);
  for (int t = 0; t < n; t++) {
    const long q = 4L * t / n, r = 4L * t - q * n;  // quadrant and (pi/2) r / n inside it
    const bool low = 2 * r <= n;
    const int64_t si = low ? so[r / 4] : co[(n - r) / 4], ci = low ? co[r / 4] : so[(n - r) / 4];
    int64_t re = 0, im = 0;
    switch (q & 3) {
      case 0: re = ci; im = -si; break;
      case 1: re = -si; im = -ci; break;
      case 2: re = -ci; im = si; break;
      default: re = si; im = ci; break;
    }
    auto split = [](int64_t v, int32_t *h, int32_t *l) {
      if ((int32_t)(uint32_t)v == INT32_MIN) v++;  // keeps the low part's negative representable
      *l = (int32_t)(uint32_t)v;
      *h = (int32_t)((v - *l) / (int64_t)4294967296);
    };
    split(re, &out[4 * (size_t)t], &out[4 * (size_t)t + 1]);
    split(im, &out[4 * (size_t)t + 2], &out[4 * (size_t)t + 3]);
  }
  return out;
}

// Fourier eigenvalue of mode J of the periodic second difference
// (src/fluid/compute_potential.c:112-115)
inline double poisson_eigenvalue(double dy, int jtot, int J) {
  return -4. / pow(dy, 2.) * pow(sin(kPiRef * (J) / (1. * jtot)), 2.);
}

// ------------------------------------------------ partition method (PCR)
// A tridiagonal line of n rows is split into kPartSeg segments of m = n /
// kPartSeg rows, one per lane of a warp. Row e = k m + m - 1, the last of
// segment k, is its interface unknown; the m - 1 rows before it are the
// segment's interior. With the interface values known, an interior is the
// solution y of its own block (zero boundary values) plus multiples of two
// spikes: x_i = y_i + v_i x_{e(k-1)} + w_i x_{e(k)}. Substituting into the
// interface rows gives a tridiagonal system of kPartSeg unknowns, solved by
// parallel cyclic reduction in kPartLevels levels of warp shuffles.
// Everything here is independent of the right-hand side and computed once.
constexpr int kPartSeg = 32;
constexpr int kPartLevels = 5;  // log2(kPartSeg)

// doubles per line of the factor block written by partition_factors_tri
inline size_t partition_stride(int n) { return 4 * (size_t)n + 2 * kPartLevels * kPartSeg + kPartSeg; }

// Factors of one line of n rows with sub-diagonal a_i, diagonal d_i and
// super-diagonal c_i. periodic: row 0 couples to row n-1 through a_0 and row
// n-1 to row 0 through c_{n-1}, so the interface system is cyclic (lane k
// couples to lanes k -+ 2^lev modulo kPartSeg at every level; after the last
// level both couplings fold into the diagonal); otherwise a_0 and c_{n-1} are
// ignored and the couplings past either end are zero. pin_last: the singular
// mean mode of the Poisson lines, whose last unknown the reference's Thomas
// solve sets to zero (its last pivot vanishes, src/linalg.c:36-38). Output
// (doubles): inv[n] up[n] v[n] w[n] (interior Thomas factors and spikes by
// row) alpha[kPartLevels][kPartSeg] beta[kPartLevels][kPartSeg] rD[kPartSeg].
// interleave: the four row arrays hold row k m + r at index r kPartSeg + k,
// so that the 32 lanes, each walking its own segment, touch 32 consecutive
// words at every step.
inline void partition_factors_tri(int n, const double *a_in, const double *d, const double *c_in, bool periodic,
                                  bool pin_last, bool interleave, double *out) {
  const int m = n / kPartSeg;
  std::vector<double> a(a_in, a_in + n), c(c_in, c_in + n);
  if (!periodic) {
    a[0] = 0.0;
    c[n - 1] = 0.0;
  }
  std::vector<double> inv(n, 0.0), up(n, 0.0), v(n, 0.0), w(n, 0.0);
  double *alpha = out + 4 * (size_t)n, *beta = alpha + kPartLevels * kPartSeg, *rD = beta + kPartLevels * kPartSeg;
  std::vector<double> L(kPartSeg), D(kPartSeg), U(kPartSeg);
  for (int k = 0; k < kPartSeg; k++) {
    const int s = k * m, e = s + m - 1;
    // interior block rows s..e-1
    inv[s] = 1.0 / d[s];
    up[s] = c[s] * inv[s];
    for (int i = s + 1; i < e; i++) {
      inv[i] = 1.0 / (d[i] - a[i] * up[i - 1]);
      up[i] = c[i] * inv[i];
    }
    auto solve = [&](std::vector<double> &r) {  // r over rows s..e-1 (index i - s)
      r[0] *= inv[s];
      for (int i = s + 1; i < e; i++) r[i - s] = inv[i] * (r[i - s] - a[i] * r[i - s - 1]);
      for (int i = e - 2; i >= s; i--) r[i - s] -= up[i] * r[i - s + 1];
    };
    std::vector<double> rv(m - 1, 0.0), rw(m - 1, 0.0);
    rv[0] = -a[s];
    rw[m - 2] = -c[e - 1];
    solve(rv);
    solve(rw);
    for (int i = s; i < e; i++) {
      v[i] = rv[i - s];
      w[i] = rw[i - s];
    }
  }
  for (int k = 0; k < kPartSeg; k++) {
    const int s = k * m, e = s + m - 1;
    const double ae = a[e], ce = c[e];
    L[k] = ae * v[e - 1];
    D[k] = ae * w[e - 1] + d[e];
    U[k] = 0.0;
    if (periodic || k < kPartSeg - 1) {
      const int s1 = (s + m) % n;  // the next segment's first interior row
      D[k] += ce * v[s1];
      U[k] = ce * w[s1];
    }
  }
  if (pin_last) {
    L[kPartSeg - 1] = 0.0;
    D[kPartSeg - 1] = 1.0;
    U[kPartSeg - 1] = 0.0;
  }
  for (int lev = 0; lev < kPartLevels; lev++) {
    const int dd = 1 << lev;
    std::vector<double> L2(kPartSeg), D2(kPartSeg), U2(kPartSeg);
    for (int k = 0; k < kPartSeg; k++) {
      const bool has_m = periodic || k - dd >= 0, has_p = periodic || k + dd < kPartSeg;
      const int km = (k - dd + kPartSeg) % kPartSeg, kp = (k + dd) % kPartSeg;
      const double al = has_m ? -L[k] / D[km] : 0.0;
      const double be = has_p ? -U[k] / D[kp] : 0.0;
      alpha[lev * kPartSeg + k] = al;
      beta[lev * kPartSeg + k] = be;
      L2[k] = has_m ? al * L[km] : 0.0;
      U2[k] = has_p ? be * U[kp] : 0.0;
      D2[k] = D[k] + (has_m ? al * U[km] : 0.0) + (has_p ? be * L[kp] : 0.0);
    }
    L = L2;
    D = D2;
    U = U2;
  }
  // cyclic: the last level leaves L and U on the unknown itself
  for (int k = 0; k < kPartSeg; k++) rD[k] = periodic ? 1.0 / (D[k] + L[k] + U[k]) : 1.0 / D[k];
  for (int i = 0; i < n; i++) {
    const size_t o = interleave ? (size_t)(i % m) * kPartSeg + i / m : (size_t)i;
    out[o] = inv[i];
    out[n + o] = up[i];
    out[2 * (size_t)n + o] = v[i];
    out[3 * (size_t)n + o] = w[i];
  }
}

// stage layout of the length-jtot/2 complex FFT: radix 2 first when
// log2(jtot/2) is odd, then radix 4
inline void fft_layout(int jtot, int *nst, int *first2) {
  int p = 0;
  while ((1 << p) < jtot / 2) p++;
  *first2 = p & 1;
  *nst = (p & 1) + p / 2;
}

}  // namespace sns
