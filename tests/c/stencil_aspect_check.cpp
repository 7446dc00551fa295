// The fixed-point advective and diffusive terms (csrc/stencil_fixed.cuh) on
// cells that are not square, on the CPU: errors of the integers and of the FP64
// expressions that they stand for (src/fluid/update_velocity.c:11-192,
// src/temperature/update.c:11-87), both against long double. Grids of N columns,
// dy = dx times each aspect on the command line; walls; neighbour distances that
// are equal, or equal but for the rounding of a grid or 2^-10; fields: 0 smooth,
// 1 noise, 2 smooth with u a thousandth of v, 3 the same the other way round,
// 4 and 5 smooth along x or y alone.
// Prints for each scheme (bit 0: implicit x, bit 1: implicit y), quantity (0 ux,
// 1 uy, 2 T) and sum (0: A, 1: the implicit diffusion) the relative 2-norms of
// both errors.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "stencil_fixed.cuh"

using namespace sns;
using namespace sns::sfx;
constexpr int W = 34, H = 10, N = 512;

struct Grid {
  double rx, ry, rm, rp, nu;
};
// A and the implicit diffusion, as the FP64 path forms them
template <typename F, int IX, int IY>
static void expression(const Grid &g, F c, F l, F r, F d, F u, F vm, F vp, F wm, F wp, F *out) {
  const F rx = g.rx, ry = g.ry, rm = g.rm, rp = g.rp, nu = g.nu, h = 0.5;
  const F gxm = (c - l) * rm, gxp = (r - c) * rp, gym = (c - d) * ry, gyp = (u - c) * ry;
  const F fx = (nu * (gxp - gxm)) * rx, fy = (nu * (gyp - gym)) * ry;
  out[0] = (-(h * rx / rm * vm * gxm) - (h * rx / rp * vp * gxp)) + (-(h * wm) * gym - (h * wp) * gyp);
  if (!IX) out[0] += fx;
  if (!IY) out[0] += fy;
  out[1] = (IX ? fx : F(0)) + (IY ? fy : F(0));
}

template <bool EQ, int IX, int IY>
static int check(double aspect) {
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> un(-1, 1);
  for (int kind = 0; kind < 6; kind++) {
    const double dx = 1.0 / (EQ ? N : N / 8 * 7), dy = dx * aspect;
    double e2[3][2][3] = {};
    for (int rep = 0; rep < 48; rep++) {
      static double f[3][H][W];
      const int x0 = rep % 4 == 0 ? 0 : (int)((rng() >> 1) % (N - 40)), y0 = (int)((rng() >> 1) % 4096);
      double ph[12];
      for (double &p : ph) p = 3.0 * un(rng);
      for (int k = 0; k < 3; k++)
        for (int j = 0; j < H; j++)
          for (int i = 0; i < W; i++) {
            const double x = kind == 5 ? 0.3 : (x0 + i) * dx, y = kind == 4 ? 0.3 : (y0 + j) * dy;
            double v = 0;
            if (kind != 1)
              for (int m = 1; m <= 3; m++) v += std::sin(3.14159 * m * x) * std::cos(6.28 * m * y + ph[3 * k + m]) / m;
            else
              v = un(rng);
            if ((kind == 2 && k == 0) || (kind == 3 && k == 1)) v *= 1e-3;
            f[k][j][i] = k == 2 ? (kind != 1 ? 0.5 - x + 0.1 * v : 0.5 * v) : 0.3 * v;
          }
      const Weights w = weights(0.5, 0.5);
      for (int i = 1; i + 1 < W; i++) {
        Grid g{1.0 / dx, 1.0 / dy, 1.0 / dx, 1.0 / dx, 1.0 / std::sqrt(kind == 1 ? 1e9 : 1e7)};
        if (i == 1 && rep % 2 == 0) g.rm *= 2;
        if (i + 2 == W && rep % 2 == 0) g.rp *= 2;
        if (!EQ) {
          g.rm *= 1 + std::ldexp(un(rng), rep % 3 ? -46 : -10);
          g.rp *= 1 + std::ldexp(un(rng), rep % 3 ? -46 : -10);
        }
        const Coef rx = coef(g.rx), ry = coef(g.ry), n = coef(g.nu), nx = mul(n, rx);
        Terms K;
        if (!terms<false>(K, quarter(rx), quarter(ry), mul(nx, coef(g.rp)), mul(nx, coef(g.rm)), mul(n, mul(ry, ry))))
          return 1;
        for (int j = 1; j + 1 < H; j++) {
          auto at = [&](int k, int dj, int di) { return f[k][j + dj][i + di]; };
          auto M = [&](int k, int dj, int di) { return num(at(k, dj, di)); };
          for (int q = 0; q < 3; q++) {
            auto whole = [&](auto t, auto *out) {
              typedef decltype(t) F;
              auto a = [&](int k, int dj, int di) { return F(at(k, dj, di)); };
              auto mean = [&](F x, F y) { return F(0.5) * x + F(0.5) * y; };
              const F vm = q == 0 ? mean(a(0, 0, -1), a(0, 0, 0)) : q == 1 ? mean(a(0, -1, 0), a(0, 0, 0)) : a(0, 0, 0);
              const F vp = q == 0 ? mean(a(0, 0, 0), a(0, 0, 1)) : q == 1 ? mean(a(0, -1, 1), a(0, 0, 1)) : a(0, 0, 1);
              const F wm = q == 0 ? mean(a(1, 0, -1), a(1, 0, 0)) : q == 1 ? mean(a(1, -1, 0), a(1, 0, 0)) : a(1, 0, 0);
              const F wp = q == 0 ? mean(a(1, 1, -1), a(1, 1, 0)) : q == 1 ? mean(a(1, 0, 0), a(1, 1, 0)) : a(1, 1, 0);
              expression<F, IX, IY>(g, a(q, 0, 0), a(q, 0, -1), a(q, 0, 1), a(q, -1, 0), a(q, 1, 0), vm, vp, wm, wp, out);
            };
            long double want[2];
            double fp[2];
            whole((long double)0, want);
            whole(0.0, fp);
            Sum t;
            Vels v;
            if (!vels(v, M(0, 0, -1), M(0, 0, 0), M(0, 0, 1), M(0, -1, 0), M(0, -1, 1), M(0, 1, 0), M(1, 0, -1),
                      M(1, 0, 0), M(1, 0, 1), M(1, -1, 0), M(1, 1, 0), M(1, 1, -1)))
              return 2;
            if (q == 0) {
              t = sum_ux<IX, IY, EQ>(K, w, v);
            } else if (q == 1) {
              t = sum_uy<IX, IY, EQ>(K, v);
            } else if (!sum_temp<IX, IY, EQ>(t, K, M(2, 0, -1), M(2, 0, 0), M(2, 0, 1), M(2, -1, 0), M(2, 1, 0),
                                             M(0, 0, 0), M(0, 0, 1), M(1, 0, 0), M(1, 1, 0))) {
              return 2;
            }
            const double fix[2] = {to_double(t.A), IX || IY ? to_double(t.G) : 0.0};
            for (int s = 0; s < 2; s++) {
              e2[q][s][0] += std::pow((double)(fix[s] - want[s]), 2);
              e2[q][s][1] += std::pow((double)(fp[s] - want[s]), 2);
              e2[q][s][2] += std::pow((double)want[s], 2);
            }
          }
        }
      }
    }
    for (int q = 0; q < 3; q++)
      for (int s = 0; s < (IX || IY ? 2 : 1); s++) {
        const double norm = e2[q][s][2] > 0 ? e2[q][s][2] : 1;
        printf("%d %d %g %d %d %d %.3e %.3e\n", (int)EQ, IX + 2 * IY, aspect, kind, q, s,
               std::sqrt(e2[q][s][0] / norm), std::sqrt(e2[q][s][1] / norm));
      }
  }
  return 0;
}

template <bool EQ>
static int schemes(double a) {
  return check<EQ, 0, 0>(a) | check<EQ, 1, 0>(a) | check<EQ, 0, 1>(a) | check<EQ, 1, 1>(a);
}

int main(int argc, char **argv) {
  int rc = 0;
  for (int i = 1; i < argc; i++) rc |= schemes<true>(atof(argv[i])) | schemes<false>(atof(argv[i]));
  return rc;
}
