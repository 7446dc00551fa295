// Real DFTs along y in 64-bit block fixed point, for the forms whose Poisson
// solve is held to a tolerance rather than to the reference's operation order
// (src/fluid/compute_potential.c:69-92 and :146-157).
//
// GB300 issues one FP64 warp instruction per sub-partition every 70 to 80
// cycles, an integer addition every 1 to 2 and a 32 x 32 -> 64 multiply-add
// every 2 to 3. A complex butterfly of 64-bit integers is 2 instructions per
// real addition and 6 multiply-adds per real product by a twiddle, so the
// transform leaves the FP64 pipe, which the temperature update running beside
// it (plain path) and the other kernels need.
//
// A column's values are scaled by the power of two that brings its largest
// one just below 2^59. A pass adds at most 8 values (|z| up to 2^59.5), which
// stays below 2^63; its results' largest magnitude decides by how many bits
// the next pass shifts the column, with rounding (block floating point, per
// column, so that a column's result depends on nothing else). The factors of
// all shifts go into the exponent of the results.
//
// Accuracy: products and shifts are rounded at 2^-59 or less of the column's
// largest value of the pass. Over transforms of 8 to 4096 complex values the
// error is 0.2 to 0.6 of that of the FP64 transform it replaces (0.7 for
// delta columns of 8192 rows and, with radix 2, 64 rows inverted), for noise, smooth, single-mode, delta
// and wide-range columns (tests/test_fft_fixed.py and, for radix 4, 0.1 to 0.73,
// tests/test_fft_radix4.py measure both against an
// extended-precision DFT).
//
// Stockham passes of radix V = 8, 4 or 2 (then one of radix 4 or 2), V values per
// thread: thread t of a block handles column t mod C, group t / C of M / V. The
// radix-8 form moves the data through shared memory fewer times, the radix-4
// and radix-2 forms have two and four times the warps, each with fewer
// instructions (rules and both sides' times where the forms are launched).
// Shared memory holds element i of column c at c stride + i + i / 8 (elements
// of 16 bytes; one of padding per 8 spreads each pass's accesses over all
// banks, the columns' stride the lanes of different columns).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace sns {
namespace fx {

struct C64 {
  long long x, y;
};
// a twiddle (wr, wi) scaled by 2^62, each word split into a high part and a
// low part in (-2^31, 2^31) (fixed_twiddles in host_common.h)
struct Tw {
  int rh, rl, ih, il;
};

constexpr int kTopBits = 59;  // magnitudes below 2^kTopBits enter a pass

FX_HD int clz64(unsigned long long v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

FX_HD int hi_part(long long a) { return (int)(a >> 32) + (int)((unsigned)a >> 31); }
FX_HD int lo_part(long long a) { return (int)(unsigned)a; }
FX_HD long long mw(int a, int b, long long c) { return (long long)a * b + c; }
FX_HD long long shl(long long a, int n) { return (long long)((unsigned long long)a << n); }

FX_HD C64 add(C64 a, C64 b) { return C64{a.x + b.x, a.y + b.y}; }
FX_HD C64 sub(C64 a, C64 b) { return C64{a.x - b.x, a.y - b.y}; }
// a * (-i) (forward) or a * (+i) (inverse)
template <bool FWD>
FX_HD C64 rot(C64 a) {
  return FWD ? C64{a.y, -a.x} : C64{-a.y, a.x};
}

// u w (forward) or u conj(w) (inverse) from the words u4 = 4 u, |u4| <= 2^62:
// top 64 bits of the products with w's words, rounded (the product of the low
// parts, below a quarter of the last bit, is left out). The middle sum stays
// below 3.5 2^61.
template <bool FWD>
FX_HD C64 mul4(C64 u4, Tw w) {
  const int xh = hi_part(u4.x), xl = lo_part(u4.x), yh = hi_part(u4.y), yl = lo_part(u4.y);
  const int ph = FWD ? w.ih : -w.ih, pl = FWD ? w.il : -w.il;  // x times +wi: imaginary part
  const int nh = FWD ? -w.ih : w.ih, nl = FWD ? -w.il : w.il;  // y times -wi: real part
  const long long half = 1ll << 31;
  const long long qr = mw(yl, nh, mw(yh, nl, mw(xl, w.rh, mw(xh, w.rl, half))));
  const long long qi = mw(xl, ph, mw(xh, pl, mw(yl, w.rh, mw(yh, w.rl, half))));
  return C64{mw(xh, w.rh, mw(yh, nh, qr >> 32)), mw(yh, w.rh, mw(xh, ph, qi >> 32))};
}
template <bool FWD>
FX_HD C64 mul(C64 u, Tw w) {  // |u.x|, |u.y| <= 2^60
  return mul4<FWD>(C64{shl(u.x, 2), shl(u.y, 2)}, w);
}
// 4 v / 2^s (truncated: a quarter of the last bit at most)
FX_HD long long quad(long long v, int s) { return s < 2 ? shl(v, 2 - s) : v >> (s - 2); }
FX_HD C64 quad(C64 v, int s) { return C64{quad(v.x, s), quad(v.y, s)}; }

// a / sqrt(2), |a| <= 2^61 (the constant is scaled by 2^63)
FX_HD long long mul_sqrt_half(long long a) {
  constexpr int rh = 0x5A82799A, rl = (int)(0xFCEF3242u - 0x100000000ll);
  const long long b = shl(a, 1);
  const int bh = hi_part(b), bl = lo_part(b);
  return mw(bh, rh, mw(bl, rh, mw(bh, rl, 1ll << 31)) >> 32);
}

template <bool FWD>
FX_HD void dft4(C64 &v0, C64 &v1, C64 &v2, C64 &v3) {
  const C64 s0 = add(v0, v2), s1 = sub(v0, v2), s2 = add(v1, v3), s3 = rot<FWD>(sub(v1, v3));
  v0 = add(s0, s2);
  v2 = sub(s0, s2);
  v1 = add(s1, s3);
  v3 = sub(s1, s3);
}

// 8-point DFT in place: v[n] -> X[k]; n = j + 4 m: the even outputs are the
// 4-point DFT of v_j + v_j+4, the odd ones that of w8^j (v_j - v_j+4)
template <bool FWD>
FX_HD void dft8(C64 *v) {
  C64 a0 = add(v[0], v[4]), a1 = add(v[1], v[5]), a2 = add(v[2], v[6]), a3 = add(v[3], v[7]);
  C64 b0 = sub(v[0], v[4]), b1 = sub(v[1], v[5]), b2 = rot<FWD>(sub(v[2], v[6])), b3 = sub(v[3], v[7]);
  if (FWD) {
    b1 = C64{mul_sqrt_half(b1.x + b1.y), mul_sqrt_half(b1.y - b1.x)};
    b3 = C64{mul_sqrt_half(b3.y - b3.x), mul_sqrt_half(-b3.x - b3.y)};
  } else {
    b1 = C64{mul_sqrt_half(b1.x - b1.y), mul_sqrt_half(b1.x + b1.y)};
    b3 = C64{mul_sqrt_half(-b3.x - b3.y), mul_sqrt_half(b3.x - b3.y)};
  }
  dft4<FWD>(a0, a1, a2, a3);
  dft4<FWD>(b0, b1, b2, b3);
  v[0] = a0;
  v[2] = a1;
  v[4] = a2;
  v[6] = a3;
  v[1] = b0;
  v[3] = b1;
  v[5] = b2;
  v[7] = b3;
}

// one group of 8 values of a pass of radix R: twiddles and butterflies
template <int R, bool FWD>
FX_HD void butterfly(C64 *u) {
  if constexpr (R == 8) {
    dft8<FWD>(u);
  } else if constexpr (R == 4) {
    dft4<FWD>(u[0], u[1], u[2], u[3]);
  } else {
    const C64 t = u[0];
    u[0] = add(t, u[1]);
    u[1] = sub(t, u[1]);
  }
}

// (v + 2^(s-1)) >> s
FX_HD long long round_shift(long long v, int s) { return s > 0 ? (v + (1ll << (s - 1))) >> s : v; }
FX_HD C64 round_shift(C64 v, int s) { return C64{round_shift(v.x, s), round_shift(v.y, s)}; }
// bits of the magnitudes (as |v| or |v| - 1), of their high words
FX_HD unsigned mag(C64 v) {
  const int a = (int)(v.x >> 32), b = (int)(v.y >> 32);
  return (unsigned)(a ^ (a >> 31)) | (unsigned)(b ^ (b >> 31));
}
// shift that brings magnitudes with these bits below 2^kTopBits
FX_HD int shift_of(unsigned m) {
  const int s = (64 - kTopBits) - clz64((unsigned long long)m << 32);
  return s > 0 ? s : 0;
}

FX_HD unsigned exponent_key(double d) {
#ifdef __CUDA_ARCH__
  return (unsigned)(__double2hiint(d) & 0x7fffffff) >> 20;
#else
  unsigned long long b;
  __builtin_memcpy(&b, &d, 8);
  return (unsigned)(b >> 52) & 0x7ff;
#endif
}
// d 2^(1081 - E) rounded to an integer; E: a biased exponent of kTiny or more
// and at least d's: magnitudes up to 2^59. (A subnormal d is below the last
// bit.)
constexpr int kTiny = 128;
FX_HD long long quantise(double d, int E) {
  unsigned long long b;
#ifdef __CUDA_ARCH__
  b = (unsigned long long)__double_as_longlong(d);
#else
  __builtin_memcpy(&b, &d, 8);
#endif
  const int e = (int)(b >> 52) & 0x7ff;
  const unsigned long long m = ((b & 0xfffffffffffffull) | 1ull << 52) << 7;
  const int s = E - e;
  const long long q = (long long)(((m >> (s < 63 ? s : 63)) + 1) >> 1), n = (long long)b >> 63;
  return (q ^ n) - n;
}
// the same for a float; E at least its double exponent
FX_HD long long quantise(float f, int E) {
  unsigned b;
#ifdef __CUDA_ARCH__
  b = __float_as_uint(f);
#else
  __builtin_memcpy(&b, &f, 4);
#endif
  const int e = (int)(b >> 23) & 0xff;
  const unsigned long long m = (unsigned long long)(((b & 0x7fffffu) | (e ? 1u << 23 : 0u)) << 4) << 32;  // 60 bits
  const int s = E - ((e ? e : 1) + 896);
  const long long q = (long long)(((m >> (s < 63 ? s : 63)) + 1) >> 1), n = (long long)((int)b >> 31);
  return (q ^ n) - n;
}
// 0 for 0, a float's biased exponent as a double, 0x7ff for infinities and NaN
FX_HD unsigned exponent_key(float f) {
  unsigned b;
#ifdef __CUDA_ARCH__
  b = __float_as_uint(f);
#else
  __builtin_memcpy(&b, &f, 4);
#endif
  const unsigned e = (b >> 23) & 0xff;
  return e == 255u ? 0x7ffu : (b & 0x7fffffffu) == 0u ? 0u : (e ? e : 1u) + 896u;
}
// a column whose largest exponent is below kTiny is taken times 2^512 (exact)
FX_HD double lift(double d, bool tiny) { return tiny ? d * 0x1p512 : d; }
FX_HD int column_scale(unsigned top, bool *tiny, int *eoff) {
  *tiny = top < (unsigned)kTiny;
  if (*tiny) {
    *eoff -= 512;
    // the exponent of the largest value times 2^512, at most (a subnormal's is lower)
    return (int)top + 512;
  }
  return (int)top;
}
// v 2^e
FX_HD double to_double(long long v, int e) {
  if (v == 0) return 0.0;
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const int lz = clz64(a);
  const unsigned long long m = a << lz;
  const unsigned long long r = (m >> 11) + ((m >> 10) & 1ull);  // 53 bits, or 2^53
  const int be = 63 + 1023 + e - lz;
  const bool in_range = be > 0 && be < 2047;
  const unsigned long long bits =
      ((unsigned long long)((in_range ? be : 1023) - 1) << 52) + r + (v < 0 ? 1ull << 63 : 0ull);
  double d;
#ifdef __CUDA_ARCH__
  d = __longlong_as_double((long long)bits);
  if (!in_range) d = ldexp(d, be - 1023);
#else
  __builtin_memcpy(&d, &bits, 8);
  if (!in_range) d = __builtin_ldexp(d, be - 1023);
#endif
  return d;
}

// v 2^e times scale as two FP64 instructions: f = scale 2^e where that is a
// normal number
struct Factor {
  double f, scale;
  int e;
  bool ok;
};
FX_HD Factor factor(double scale, int e) {
  Factor r;
  r.scale = scale;
  r.e = e;
#ifdef __CUDA_ARCH__
  const int k = (__double2hiint(scale) >> 20) + e;  // negative for a negative scale
  r.ok = __double2hiint(scale) >> 20 > 0 && __double2hiint(scale) >> 20 < 2047 && k > 0 && k < 2047;
  r.f = r.ok ? __hiloint2double(__double2hiint(scale) + e * (1 << 20), __double2loint(scale)) : 0.0;
#else
  r.f = __builtin_ldexp(scale, e);
  r.ok = __builtin_isnormal(r.f) && scale > 0.0;
#endif
  return r;
}
FX_HD double scaled(long long v, const Factor &f) { return f.ok ? (double)v * f.f : to_double(v, f.e) * f.scale; }

// split step of the forward real FFT for the bin pair (k, M-k), 0 < k <= M/2,
// magnitudes below 2^59: 2 X[k] and 2 X[M-k] from A = Z[k], B = Z[M-k];
// w = exp(-2 pi i k / 2M)
FX_HD void split(C64 A, C64 B, Tw w, C64 &xk, C64 &xm) {
  // (Z[k] + conj Z[M-k]) + w (Z[k] - conj Z[M-k]) / i
  const long long sre = A.x + B.x, dim = A.y - B.y, dre = A.x - B.x, sim = A.y + B.y;
  const C64 t = mul<true>(C64{sim, -dre}, w);
  xk = C64{sre + t.x, dim + t.y};
  xm = C64{sre - t.x, t.y - dim};
}
// its inverse: 2 Z[k], 2 Z[M-k] from A = X[k], B = X[M-k]
FX_HD void merge(C64 A, C64 B, Tw w, C64 &zk, C64 &zm) {
  const long long er = A.x + B.x, ei = A.y - B.y;
  const C64 o = mul<false>(C64{A.x - B.x, A.y + B.y}, w);
  zk = C64{er - o.y, ei + o.x};
  zm = C64{er + o.y, o.x - ei};
}

// elements of 16 bytes a column takes: M and its padding, and what brings the
// stride to 8 / C modulo 8, so that the C columns' lanes fall on different banks
FX_HD int column_stride(int M, int lgC) {
  const int want = lgC < 3 ? 8 >> lgC : 1, n = M + (M >> 3);
  return n + ((want - n) & 7);
}

#ifdef __CUDACC__
constexpr int kMaxWarps = 32, kMaxCols = 16;
// per warp and column: the largest exponent, or the bits of a pass's magnitudes
struct Slots {
  unsigned s[2][kMaxWarps * kMaxCols];
};

// a thread's place: column c (of C = 2^lgC), group j of nv = M / V
template <int V>
struct Place {
  int C, M, nv, c, j, base;
  bool on;  // the block may have more threads than C M / V
  int par;  // slot buffer the next put writes
  Slots *sl;
  __device__ __forceinline__ Place(int lgC_, int M_, Slots *s)
      : C(1 << lgC_), M(M_), nv(M_ / V), c(threadIdx.x & (C - 1)), j(threadIdx.x >> lgC_),
        base(c * column_stride(M_, lgC_)), on(j < nv), par(0), sl(s) {}
  __device__ __forceinline__ int at(int i) const { return base + i + (i >> 3); }
  // a value per thread to the other threads of its column; read after a barrier
  template <bool MAX>
  __device__ __forceinline__ void put(unsigned v) {
    if (!on) v = 0u;
    for (int off = C; off < 32; off <<= 1) {
      const unsigned o = __shfl_xor_sync(0xffffffffu, v, off);
      v = MAX ? max(v, o) : v | o;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane < C) sl->s[par][w * C + lane] = v;
    par ^= 1;
  }
  // the column's result of the last put
  template <bool MAX>
  __device__ __forceinline__ unsigned get() const {
    unsigned v = 0u;
    const int nw = (int)(blockDim.x + 31) >> 5;
    for (int w = 0; w < nw; ++w) {
      const unsigned o = sl->s[par ^ 1][w * C + c];
      v = MAX ? max(v, o) : v | o;
    }
    return v;
  }
};

__device__ __forceinline__ Tw ldtw(const Tw *tw, int t) {
  const int4 v = __ldg(reinterpret_cast<const int4 *>(tw) + t);
  return Tw{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ C64 ldz(const C64 *z, int i) {
  const longlong2 v = *reinterpret_cast<const longlong2 *>(z + i);
  return C64{v.x, v.y};
}
__device__ __forceinline__ void stz(C64 *z, int i, C64 v) {
  *reinterpret_cast<longlong2 *>(z + i) = make_longlong2(v.x, v.y);
}

__device__ __forceinline__ double2 ldd(const C64 *z, int i) { return *reinterpret_cast<const double2 *>(z + i); }
__device__ __forceinline__ void std2(C64 *z, int i, double2 v) { *reinterpret_cast<double2 *>(z + i) = v; }

// The code below is short rather than unrolled: a warp runs it once per
// launch, and fetching instructions took most of the time of a version with
// every loop unrolled (about 4800 instructions a warp; warps stalled without
// an instruction 4 to 7 cycles per issue).

// One radix-V pass of span Ns: butterfly j reads elements j + r nv, shifts
// them by the bits the column needs (added to S), multiplies by the pass's
// twiddles and owns outputs (j - k) V + k + r Ns, k = j mod Ns. The last pass
// (Ns = nv) works in place.
template <int V, bool FWD>
__device__ __forceinline__ void pass_full(Place<V> &p, C64 *z, int Ns, const Tw *tw, int &S) {
  const int s = shift_of(p.template get<false>());
  S += s;
  const bool last = Ns == p.nv;
  const int k = p.j & (Ns - 1);
  C64 v[V];
  unsigned m = 0u;
  if (p.on) {
#pragma unroll
    for (int r = 0; r < V; ++r) v[r] = ldz(z, p.at(p.j + r * p.nv));
    if (Ns > 1) {
      const int step = (p.nv / Ns) * 2 * k;
      v[0] = round_shift(v[0], s);
#pragma unroll
      for (int r = 1; r < V; ++r) v[r] = mul4<FWD>(quad(v[r], s), ldtw(tw, r * step));
    } else if (s > 0) {
#pragma unroll
      for (int r = 0; r < V; ++r) v[r] = round_shift(v[r], s);
    }
    butterfly<V, FWD>(v);
#pragma unroll
    for (int r = 0; r < V; ++r) m |= mag(v[r]);
  }
  p.template put<false>(m);
  if (!last) __syncthreads();
  if (p.on) {
    const int base = (p.j - k) * V + k;
#pragma unroll
    for (int r = 0; r < V; ++r) stz(z, p.at(base + r * Ns), v[r]);
  }
}
// the last pass of lengths that are no power of V, radix R = 4 or 2 (span
// M / R): in place, V / R butterflies per thread
template <int V, int R, bool FWD>
__device__ __forceinline__ void pass_last(Place<V> &p, C64 *z, const Tw *tw, int &S) {
  const int s = shift_of(p.template get<false>());
  S += s;
  unsigned m = 0u;
  if (p.on) {
#pragma unroll 1
    for (int b = p.j; b < p.M / R; b += p.nv) {
      C64 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        v[r] = ldz(z, p.at(b + r * (p.M / R)));
        v[r] = r ? mul4<FWD>(quad(v[r], s), ldtw(tw, 2 * r * b)) : round_shift(v[r], s);
      }
      butterfly<R, FWD>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        m |= mag(v[r]);
        stz(z, p.at(b + r * (p.M / R)), v[r]);
      }
    }
  }
  p.template put<false>(m);
}
// every pass; on entry the column's magnitudes were put and a barrier passed;
// on return each thread's own elements j + r nv hold the result (a barrier
// makes the others' visible)
template <int V, bool FWD>
__device__ __forceinline__ void passes(Place<V> &p, C64 *z, const Tw *tw, int &S) {
  int Ns = 1;
#pragma unroll 1
  for (; Ns <= p.nv; Ns *= V) {
    if (Ns > 1) __syncthreads();
    pass_full<V, FWD>(p, z, Ns, tw, S);
  }
  if (Ns == p.M) return;
  __syncthreads();
  if (V == 8 && 4 * Ns == p.M) {
    pass_last<V, 4, FWD>(p, z, tw, S);
  } else {
    pass_last<V, 2, FWD>(p, z, tw, S);
  }
}

// What forward() reads. load(c, mm, raw): rows 2 mm and 2 mm + 1 of the
// block's column c into 16 bytes, and a key of 0 or the largest biased exponent
// that the magnitudes stay below 2^(key - 1022) with (0x7ff: not finite);
// fixed(raw, E, tiny): the two values times 2^(1081 - E) as integers (times
// 2^512 before that when tiny). kUnroll: loads in flight per thread.
template <typename F>
struct Doubles {
  F f;  // f(c, mm, d): d[0], d[1]
  static constexpr int kUnroll = 8;
  __device__ __forceinline__ unsigned load(int c, int mm, double2 &raw) const {
    double d[2];
    f(c, mm, d);
    raw = make_double2(d[0], d[1]);
    return max(exponent_key(d[0]), exponent_key(d[1]));
  }
  __device__ __forceinline__ C64 fixed(double2 d, int E, bool tiny) const {
    return C64{quantise(lift(d.x, tiny), E), quantise(lift(d.y, tiny), E)};
  }
};
template <typename F>
__device__ __forceinline__ Doubles<F> doubles(F f) {
  return Doubles<F>{f};
}

// Forward real DFT of a block's columns (M = jtot / 2 complex values each,
// M >= 8, C M / V threads or more) of the values that `in` gives times
// 2^eoff. out(c, k, X): 2 X[k] of the unnormalised transform (FFTW's
// conventions), k = 0 .. M. A column with a NaN or an infinity gives NaN.
template <int V, typename In, typename Out>
__device__ __forceinline__ void forward(C64 *z, Slots *slots, int lgC, int M, const Tw *tw, int eoff, In in, Out out) {
  Place<V> p(lgC, M, slots);
  unsigned top = 0u;
  if (p.on) {
    constexpr int U = In::kUnroll < V ? In::kUnroll : V;
#pragma unroll 1
    for (int r0 = 0; r0 < V; r0 += U) {
      double2 d[U];
#pragma unroll
      for (int r = 0; r < U; ++r) top = max(top, in.load(p.c, p.j + (r0 + r) * p.nv, d[r]));
#pragma unroll
      for (int r = 0; r < U; ++r) std2(z, p.at(p.j + (r0 + r) * p.nv), d[r]);
    }
  }
  p.template put<true>(top);
  __syncthreads();
  bool tiny;
  const int E = column_scale(p.template get<true>(), &tiny, &eoff);
  if (p.on) {  // each thread its own elements, which its first butterfly reads
#pragma unroll 1
    for (int i = p.j; i < M; i += p.nv) stz(z, p.at(i), in.fixed(ldd(z, p.at(i)), E, tiny));
  }
  p.template put<false>(0u);
  __syncthreads();
  int S = 0;
  passes<V, true>(p, z, tw, S);
  __syncthreads();
  const int s = shift_of(p.template get<false>());
  if (!p.on) return;
  const int e = S + s + E + eoff - 1081;
  const bool bad = E >= 0x7ff;
#pragma unroll 1
  for (int k = p.j; k <= M / 2; k += p.nv) {  // k = M / 2 is its own partner
    const C64 A = round_shift(ldz(z, p.at(k)), s), B = round_shift(ldz(z, p.at((M - k) & (M - 1))), s);
    C64 xk, xm;
    if (k == 0) {
      xk = C64{2 * (A.x + A.y), 0};
      xm = C64{2 * (A.x - A.y), 0};
    } else {
      split(A, B, ldtw(tw, k), xk, xm);
    }
    double2 o = make_double2(to_double(xk.x, e), to_double(xk.y, e));
    double2 q = make_double2(to_double(xm.x, e), to_double(xm.y, e));
    if (bad) o.x = o.y = q.x = q.y = __longlong_as_double(0x7ff8000000000000ll);
    out(p.c, k, o);
    if (2 * k != M) out(p.c, M - k, q);
  }
}

// Inverse: in(c, k): X[k] (the imaginary parts of X[0] and X[M] are ignored);
// out(c, mm, d): rows 2 mm and 2 mm + 1, the unnormalised inverse (of 2 X, as
// the merge gives 2 Z) times `scale`.
template <int V, typename In, typename Out>
__device__ __forceinline__ void inverse(C64 *z, Slots *slots, int lgC, int M, const Tw *tw, double scale, In in,
                                        Out out) {
  Place<V> p(lgC, M, slots);
  unsigned top = 0u;
  if (p.on) {
    // the pairs (k, M-k) of this thread, kept as they are until the column's
    // largest exponent is known; X[0] and X[M] share element 0
    double2 a[V / 2], b[V / 2];
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      a[i] = in(p.c, p.j + i * p.nv);
      b[i] = in(p.c, M - (p.j + i * p.nv));
    }
    if (p.j == 0) {
      a[0].y = b[0].x;
      b[0] = in(p.c, M >> 1);
    }
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      top = max(max(max(top, exponent_key(a[i].x)), max(exponent_key(a[i].y), exponent_key(b[i].x))),
                exponent_key(b[i].y));
      const int k = p.j + i * p.nv;
      std2(z, p.at(k), a[i]);
      std2(z, p.at(k ? M - k : M >> 1), b[i]);
    }
  }
  p.template put<true>(top);
  __syncthreads();
  bool tiny;
  int eoff = 0;
  const int E = column_scale(p.template get<true>(), &tiny, &eoff);
  unsigned m = 0u;
  if (p.on) {
    auto Q = [&](double2 d) { return C64{quantise(lift(d.x, tiny), E), quantise(lift(d.y, tiny), E)}; };
#pragma unroll 1
    for (int k = p.j; k <= M / 2; k += p.nv) {
      const int k2 = (M - k) & (M - 1);
      const C64 A = Q(ldd(z, p.at(k))), B = Q(ldd(z, p.at(k2)));
      C64 zk, zm;
      if (k == 0) {
        zk = zm = C64{A.x + A.y, A.x - A.y};
      } else {
        merge(A, B, ldtw(tw, k), zk, zm);
      }
      m |= mag(zk) | mag(zm);
      if (2 * k != M) stz(z, p.at(k2), zm);
      stz(z, p.at(k), zk);
    }
  }
  p.template put<false>(m);
  __syncthreads();
  int S = 0;
  passes<V, false>(p, z, tw, S);
  if (!p.on) return;
  const Factor f = factor(scale, S + E + eoff - 1081);
  const bool bad = E >= 0x7ff;
#pragma unroll 1
  for (int i = p.j; i < M; i += p.nv) {
    const C64 v = ldz(z, p.at(i));
    double d[2] = {scaled(v.x, f), scaled(v.y, f)};
    if (bad) d[0] = d[1] = __longlong_as_double(0x7ff8000000000000ll);
    out(p.c, i, d);
  }
}
#endif  // __CUDACC__

}  // namespace fx
}  // namespace sns
