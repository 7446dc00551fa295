// fft_fixed_check.cpp for passes of radix 4 (four values per thread), with a last
// one of radix 2 where the length asks for it: jtot 16 to 4096.
#define main fft_fixed_check_main
#include "fft_fixed_check.cpp"
#undef main

template <bool FWD>
static int radix4(std::vector<C64> &z, int M, unsigned &m) {
  int S = 0, Ns = 1, rem = M;
  for (; rem >= 4; rem /= 4, Ns *= 4) pass_fixed<4, FWD>(z, M, Ns, S, m);
  if (rem == 2) pass_fixed<2, FWD>(z, M, Ns, S, m);
  return S;
}
struct Column {  // its largest exponent
  bool tiny;
  int eoff = 0, E;
  explicit Column(const std::vector<double> &v) {
    unsigned top = 0;
    for (double x : v) top = std::max(top, exponent_key(x));
    E = column_scale(top, &tiny, &eoff);
  }
  long long q(double v) const { return quantise(lift(v, tiny), E); }
};

int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(-1, 1);
  for (int n = 16; n <= 4096; n *= 2) {
    const int M = n / 2;
    const std::vector<int32_t> t = fixed_twiddles(n);
    tw.resize(n);
    std::memcpy(tw.data(), t.data(), sizeof(Tw) * n);
    twd = twiddle_table(n);
    for (int kind = 0; kind < 6; kind++) {
      long double e[4] = {0, 0, 0, 0};
      for (int rep = 0; rep < 4; rep++) {
        const double size = std::ldexp(1.0, rep == 3 ? -960 : (int)(g() % 200) - 100), ph = U(g);
        const int at = (int)(g() % n), mode = 1 + (int)(g() % (M - 1));
        std::vector<double> d(n);
        for (int i = 0; i < n; i++) {
          const double x = 6.283185307179586 * i / n, r = U(g);
          const double v[6] = {r, std::sin(3 * x + ph) + 1e-6 * r, std::cos(mode * x + ph), i == at ? 1.0 : 0.0,
                               r * std::exp(-30.0 * i / n), 1.0 + 1e-3 * r};
          d[i] = v[kind] * size;
        }
        auto add_errors = [&](long double *err, auto &&fixed, auto &&fp64, auto &&want, int count) {
          long double sf = 0, sd = 0, s0 = 0;
          for (int k = 0; k < count; k++) {
            sf += std::norm(cl(fixed[k]) - want(k));
            sd += std::norm(cl(fp64[k]) - want(k));
            s0 += std::norm(want(k));
          }
          err[0] += sf / s0;
          err[1] += sd / s0;
        };
        // forward: 2 X
        const Column c(d);
        std::vector<C64> z(M);
        for (int i = 0; i < M; i++) z[i] = C64{c.q(d[2 * i]), c.q(d[2 * i + 1])};
        unsigned m = 0;
        const int S = radix4<true>(z, M, m), s = shift_of(m), ex = S + s + c.E + c.eoff - 1081;
        std::vector<cd> Xf(M + 1), Xd;
        for (int k = 0; k <= M / 2; k++) {
          const C64 A = round_shift(z[k], s), B = round_shift(z[(M - k) % M], s);
          C64 xk{2 * (A.x + A.y), 0}, xm{2 * (A.x - A.y), 0};
          if (k) split(A, B, tw[k], xk, xm);
          Xf[k] = cd(to_double(xk.x, ex), to_double(xk.y, ex));
          if (2 * k != M) Xf[M - k] = cd(to_double(xm.x, ex), to_double(xm.y, ex));
        }
        forward_fp64(d, Xd);
        std::vector<cl> w(d.begin(), d.end());
        dft_ld(w, -1);
        add_errors(e, Xf, Xd, [&](int k) { return 2.0L * w[k]; }, M + 1);
        // inverse: the spectrum of a Poisson solution
        std::vector<cd> P(M + 1);
        for (int k = 0; k <= M; k++) P[k] = Xd[k] / (1.0 + 1.0 * k * k);
        P[0] = P[0].real();
        P[M] = P[M].real();
        const double scale = 1.2345678912345 / n;
        std::vector<double> parts;
        for (const cd &x : P) parts.insert(parts.end(), {x.real(), x.imag()});
        const Column ci(parts);
        m = 0;
        for (int k = 0; k <= M / 2; k++) {
          const C64 A{ci.q(P[k].real()), ci.q(P[k].imag())}, B{ci.q(P[M - k].real()), ci.q(P[M - k].imag())};
          C64 zk{A.x + B.x, A.x - B.x}, zm{0, 0};
          if (k) merge(A, B, tw[k], zk, zm);
          z[k] = zk;
          if (k && 2 * k != M) z[M - k] = zm;
          m |= mag(zk) | mag(zm);
        }
        const Factor f = factor(scale, radix4<false>(z, M, m) + ci.E + ci.eoff - 1081);
        std::vector<double> pf(n), pd;
        for (int i = 0; i < n; i++) pf[i] = scaled(i % 2 ? z[i / 2].y : z[i / 2].x, f);
        inverse_fp64(P, scale, pd);
        for (int k = 0; k < n; k++) w[k] = k <= M ? cl(P[k]) : std::conj(cl(P[n - k]));
        dft_ld(w, 1);
        add_errors(e + 2, pf, pd, [&](int i) { return cl(w[i].real() * scale); }, n);
      }
      std::printf("%d %d %.3Lg %.3Lg %.3Lg %.3Lg\n", n, kind, sqrtl(e[0] / 4), sqrtl(e[1] / 4), sqrtl(e[2] / 4),
                  sqrtl(e[3] / 4));
    }
  }
  return 0;
}
