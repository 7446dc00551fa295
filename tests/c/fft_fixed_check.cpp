// The fixed-point real DFT (csrc/fft_fixed.cuh) run on the CPU: the kernels'
// own arithmetic (quantisation, passes, shifts, split steps, conversions) in
// their order, one column at a time, against a DFT in long double, beside the
// FP64 radix-8 transform it stands for (the same passes in double). With an
// argument: passes of radix 2, to jtot 256. For each
// length and kind of column prints: jtot, kind, forward error of the fixed
// and of the FP64 transform, inverse errors of both (relative 2-norms).
#include <cstdio>
#include <cstring>
#include <complex>
#include <random>

#include "fft_fixed.cuh"
#include "host_common.h"

using namespace sns;
using namespace sns::fx;
typedef std::complex<double> cd;
typedef std::complex<long double> cl;

static std::vector<Tw> tw;
static std::vector<double> twd;

template <int R, bool FWD>
static void pass_fixed(std::vector<C64> &z, int M, int Ns, int &S, unsigned &m) {
  std::vector<C64> o(M);
  const int s = shift_of(m), nb = M / R;
  S += s;
  m = 0;
  for (int b = 0; b < nb; b++) {
    C64 u[8];
    const int k = b & (Ns - 1), step = 2 * (M / (Ns * R)) * k;
    for (int r = 0; r < R; r++) {
      u[r] = z[b + r * nb];
      u[r] = Ns > 1 && r ? mul4<FWD>(quad(u[r], s), tw[r * step]) : round_shift(u[r], s);
    }
    butterfly<R, FWD>(u);
    for (int r = 0; r < R; r++) {
      m |= mag(u[r]);
      o[(b - k) * R + k + r * Ns] = u[r];
    }
  }
  z.swap(o);
}
static bool radix2;  // two values per thread: passes of radix 2
template <bool FWD>
static void fixed_fft(std::vector<C64> &z, int M, int &S, unsigned &m) {
  int Ns = 1, rem = M;
  for (; radix2 && rem >= 2; rem >>= 1, Ns <<= 1) pass_fixed<2, FWD>(z, M, Ns, S, m);
  for (; rem >= 8; rem >>= 3, Ns <<= 3) pass_fixed<8, FWD>(z, M, Ns, S, m);
  if (rem == 4) pass_fixed<4, FWD>(z, M, Ns, S, m);
  if (rem == 2) pass_fixed<2, FWD>(z, M, Ns, S, m);
}
static void forward_fixed(const std::vector<double> &d, std::vector<cd> &X) {  // 2 X
  const int n = (int)d.size(), M = n / 2;
  unsigned top = 0;
  for (double v : d) top = std::max(top, exponent_key(v));
  bool tiny;
  int eoff = 0;
  const int E = column_scale(top, &tiny, &eoff);
  std::vector<C64> z(M);
  for (int i = 0; i < M; i++) z[i] = C64{quantise(lift(d[2 * i], tiny), E), quantise(lift(d[2 * i + 1], tiny), E)};
  int S = 0;
  unsigned m = 0;
  fixed_fft<true>(z, M, S, m);
  const int s = shift_of(m), e = S + s + E + eoff - 1081;
  X.resize(M + 1);
  for (int k = 0; k <= M / 2; k++) {
    const C64 A = round_shift(z[k], s), B = round_shift(z[(M - k) % M], s);
    if (k == 0) {
      X[0] = to_double(2 * (A.x + A.y), e);
      X[M] = to_double(2 * (A.x - A.y), e);
      continue;
    }
    C64 xk, xm;
    split(A, B, tw[k], xk, xm);
    X[k] = cd(to_double(xk.x, e), to_double(xk.y, e));
    if (2 * k != M) X[M - k] = cd(to_double(xm.x, e), to_double(xm.y, e));
  }
}
static void inverse_fixed(const std::vector<cd> &X, double scale, std::vector<double> &d) {
  const int M = (int)X.size() - 1;
  unsigned top = 0;
  for (const cd &x : X) top = std::max(top, std::max(exponent_key(x.real()), exponent_key(x.imag())));
  bool tiny;
  int eoff = 0;
  const int E = column_scale(top, &tiny, &eoff);
  auto Q = [&](double v) { return quantise(lift(v, tiny), E); };
  std::vector<C64> z(M);
  unsigned m = 0;
  for (int k = 0; k <= M / 2; k++) {
    const C64 A{Q(X[k].real()), k ? Q(X[k].imag()) : 0}, B{Q(X[M - k].real()), k ? Q(X[M - k].imag()) : 0};
    C64 zk{A.x + B.x, A.x - B.x}, zm{0, 0};
    if (k) merge(A, B, tw[k], zk, zm);
    z[k] = zk;
    if (k && 2 * k != M) z[M - k] = zm;
    m |= mag(zk) | mag(zm);
  }
  int S = 0;
  fixed_fft<false>(z, M, S, m);
  const Factor f = factor(scale, S + E + eoff - 1081);
  d.resize(2 * M);
  for (int i = 0; i < M; i++) {
    d[2 * i] = scaled(z[i].x, f);
    d[2 * i + 1] = scaled(z[i].y, f);
  }
}
// the same passes in double
static void fp64_fft(std::vector<cd> &z, bool fwd) {
  const int M = (int)z.size();
  auto W = [&](int t) {
    const cd w(twd[2 * t], twd[2 * t + 1]);
    return fwd ? w : std::conj(w);
  };
  int Ns = 1;
  for (int rem = M; rem > 1;) {
    const int R = rem >= 8 ? 8 : rem, nb = M / R;
    std::vector<cd> o(M);
    for (int b = 0; b < nb; b++) {
      const int k = b & (Ns - 1), step = 2 * (M / (Ns * R)) * k;
      cd u[8];
      for (int r = 0; r < R; r++) u[r] = z[b + r * nb] * W(r * step);
      // radix-2 stages with the 8th roots
      for (int h = R / 2; h >= 1; h /= 2)
        for (int g = 0; g < R; g += 2 * h)
          for (int i = 0; i < h; i++) {
            const cd a = u[g + i], c = u[g + i + h];
            u[g + i] = a + c;
            u[g + i + h] = (a - c) * W(2 * M / (2 * h) * i);
          }
      for (int r = 0; r < R; r++) {
        int p = 0;
        for (int i = 1, x = r; i < R; i *= 2, x >>= 1) p = 2 * p + (x & 1);
        o[(b - k) * R + k + r * Ns] = u[p];
      }
    }
    z.swap(o);
    Ns *= R;
    rem /= R;
  }
}
static void forward_fp64(const std::vector<double> &d, std::vector<cd> &X) {
  const int M = (int)d.size() / 2;
  std::vector<cd> z(M);
  for (int i = 0; i < M; i++) z[i] = cd(d[2 * i], d[2 * i + 1]);
  fp64_fft(z, true);
  X.resize(M + 1);
  for (int k = 0; k <= M; k++) {
    const cd A = z[k % M], B = std::conj(z[(M - k) % M]), w(twd[2 * k % (4 * M)], twd[(2 * k + 1) % (4 * M)]);
    X[k] = (A + B) + w * (A - B) * cd(0, -1);
  }
}
static void inverse_fp64(const std::vector<cd> &X, double scale, std::vector<double> &d) {
  const int M = (int)X.size() - 1;
  std::vector<cd> z(M);
  for (int k = 0; k < M; k++) {
    cd A = X[k], B = std::conj(X[M - k]);
    if (k == 0) {
      A = A.real();
      B = B.real();
    }
    const cd w(twd[2 * k], -twd[2 * k + 1]);
    z[k] = (A + B) + w * (A - B) * cd(0, 1);
  }
  fp64_fft(z, false);
  d.resize(2 * M);
  for (int i = 0; i < M; i++) {
    d[2 * i] = z[i].real() * scale;
    d[2 * i + 1] = z[i].imag() * scale;
  }
}
// long double complex DFT (recursive radix 2)
static void dft_ld(std::vector<cl> &z, int sign) {
  const int n = (int)z.size();
  if (n == 1) return;
  std::vector<cl> a(n / 2), b(n / 2);
  for (int i = 0; i < n / 2; i++) {
    a[i] = z[2 * i];
    b[i] = z[2 * i + 1];
  }
  dft_ld(a, sign);
  dft_ld(b, sign);
  for (int k = 0; k < n / 2; k++) {
    const long double t = sign * 2.0L * 3.14159265358979323846264338327950288L * k / n;
    const cl w(cosl(t), sinl(t));
    z[k] = a[k] + w * b[k];
    z[k + n / 2] = a[k] - w * b[k];
  }
}

int main(int argc, char **) {
  radix2 = argc > 1;
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(-1, 1);
  for (int n = 16; n <= (radix2 ? 256 : 8192); n *= 2) {
    const int M = n / 2;
    const std::vector<int32_t> t = fixed_twiddles(n);
    tw.resize(n);
    std::memcpy(tw.data(), t.data(), sizeof(Tw) * n);
    twd = twiddle_table(n);
    for (int kind = 0; kind < 6; kind++) {
      double e[4] = {0, 0, 0, 0}, nf = 0, ni = 0;
      for (int rep = 0; rep < 4; rep++) {
        std::vector<double> d(n);
        const double size = std::ldexp(1.0, rep == 3 ? -960 : (int)(g() % 200) - 100);
        const int at = (int)(g() % n), mode = 1 + (int)(g() % (M - 1));
        const double ph = U(g);
        for (int i = 0; i < n; i++) {
          const double x = 6.283185307179586 * i / n;
          double v = U(g);                                            // 0: noise
          if (kind == 1) v = std::sin(3 * x + ph) + 1e-6 * U(g);      // smooth, little noise
          if (kind == 2) v = std::cos(mode * x + ph);                 // one mode
          if (kind == 3) v = i == at ? 1.0 : 0.0;                     // delta
          if (kind == 4) v = U(g) * std::exp(-30.0 * (i / (double)n)); // wide range
          if (kind == 5) v = 1.0 + 1e-3 * U(g);                       // a mean and little else
          d[i] = v * size;
        }
        std::vector<cl> z(n);
        for (int i = 0; i < n; i++) z[i] = d[i];
        dft_ld(z, -1);
        std::vector<cd> Xf, Xd;
        forward_fixed(d, Xf);
        forward_fp64(d, Xd);
        long double sf = 0, sd = 0, s0 = 0;
        for (int k = 0; k <= M; k++) {
          sf += std::norm(cl(Xf[k]) - 2.0L * z[k]);
          sd += std::norm(cl(Xd[k]) - 2.0L * z[k]);
          s0 += std::norm(2.0L * z[k]);
        }
        e[0] += (double)(sf / s0);
        e[1] += (double)(sd / s0);
        // inverse: the spectrum of a Poisson solution, X / (1 + k^2)
        std::vector<cd> P(M + 1);
        for (int k = 0; k <= M; k++) P[k] = Xd[k] / (1.0 + 1.0 * k * k);
        P[0] = P[0].real();
        P[M] = P[M].real();
        const double scale = 1.2345678912345 / n;
        std::vector<double> pf, pd;
        inverse_fixed(P, scale, pf);
        inverse_fp64(P, scale, pd);
        for (int k = 0; k < n; k++) z[k] = k <= M ? cl(P[k]) : std::conj(cl(P[n - k]));
        dft_ld(z, 1);
        sf = sd = s0 = 0;
        for (int i = 0; i < n; i++) {
          const long double r = 1.0L * z[i].real() * scale;
          sf += (pf[i] - r) * (pf[i] - r);
          sd += (pd[i] - r) * (pd[i] - r);
          s0 += r * r;
        }
        e[2] += (double)(sf / s0);
        e[3] += (double)(sd / s0);
        nf++;
        ni++;
      }
      std::printf("%d %d %.3g %.3g %.3g %.3g\n", n, kind, std::sqrt(e[0] / nf), std::sqrt(e[1] / nf),
                  std::sqrt(e[2] / ni), std::sqrt(e[3] / ni));
    }
  }
  return 0;
}
