// The fixed-point advective and diffusive terms (csrc/stencil_fixed.cuh) run on
// the CPU, against the same sums in long double, beside the FP64 expressions
// that they stand for (src/fluid/update_velocity.c:11-192,
// src/temperature/update.c:11-87). Tiles of 32 x 8 cells of a grid of N columns
// with square cells, or (not EQ) nearly so, some of them beside a wall; for
// each N, kind of field (0 and 2 smooth, 1 noise, 3 noise over 2^60) and
// quantity (0 ux, 1 uy, 2 T, 3 diffusion of T alone) prints the relative
// 2-norms of both errors.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "stencil_fixed.cuh"

using namespace sns;
using namespace sns::sfx;
constexpr int W = 34, H = 10;

// A of f with the face velocities vm, vp, wm, wp as the FP64 path forms it; rx:
// 1 / the cell's width, rm, rp: 1 / the distances to its x neighbours (the
// advective coefficient and the gradient's spacing multiply to rx / 2)
template <typename F>
static F expression(F c, F l, F r, F d, F u, F vm, F vp, F wm, F wp, F rx, F rm, F rp, F ry, F nu, bool adv) {
  const F gxm = (c - l) * rm, gxp = (r - c) * rp, gym = (c - d) * ry, gyp = (u - c) * ry;
  F A = 0;
  if (adv) {
    A = (-(F(0.5) * rx / rm * vm * gxm) - (F(0.5) * rx / rp * vp * gxp)) +
        (-(F(0.5) * wm) * gym - (F(0.5) * wp) * gyp);
  }
  return A + (nu * (gxp - gxm)) * rx + (nu * (gyp - gym)) * ry;
}

template <bool EQ>
static int check(int argc, char **argv) {
  const int lo = atoi(argv[1]), hi = atoi(argv[2]);
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> un(-1, 1);
  for (int N = lo; N <= hi; N *= 2)
    for (int kind = 0; kind < 4; kind++) {
      const double dx = 1.0 / (EQ ? N : N / 8 * 7), rx = 1.0 / dx, nu = 1.0 / std::sqrt(1e9 * (kind == 2 ? 1e-4 : 1.0));
      double e2[4][3] = {};
      for (int rep = 0; rep < 64; rep++) {
        static double f[3][H][W];
        const int x0 = rep % 4 == 0 ? 0 : (int)((rng() >> 1) % (unsigned)(N > 64 ? N - 40 : 1)), y0 = (int)((rng() >> 1) % 4096);
        double ph[12];
        for (double &p : ph) p = 3.0 * un(rng);
        for (int k = 0; k < 3; k++)
          for (int j = 0; j < H; j++)
            for (int i = 0; i < W; i++) {
              const double x = (x0 + i) * dx, y = (y0 + j) * dx;
              double v = 0;
              if (kind == 0 || kind == 2)  // smooth, zero at the wall
                for (int m = 1; m <= 3; m++) v += std::sin(3.14159 * m * x) * std::cos(6.28 * m * y + ph[3 * k + m]) / m;
              else if (kind == 1)  // noise
                v = un(rng);
              else  // wide range
                v = un(rng) * std::ldexp(1.0, (int)(rng() % 60) - 50);
              f[k][j][i] = k == 2 ? (kind == 0 || kind == 2 ? 0.5 - x + 0.1 * v : 0.5 * v) : 0.3 * v;
            }
        const Coef r = coef(rx), n = coef(nu), cy = mul(n, mul(r, r));
        const Weights w = weights(0.5, 0.5);
        for (int i = 1; i + 1 < W; i++) {
          // neighbour distances: a wall to the left or right, or (not EQ) the rounding of a grid
          double rm = rx, rp = rx;
          if (i == 1 && rep % 2 == 0) rm = 2 * rx;
          if (i + 2 == W && rep % 2 == 0) rp = 2 * rx;
          if (!EQ) {
            rm *= 1 + std::ldexp(un(rng), rep % 3 ? -46 : -10);
            rp *= 1 + std::ldexp(un(rng), rep % 3 ? -46 : -10);
          }
          Terms K;
          if (!terms<false>(K, quarter(r), quarter(r), mul(mul(n, r), coef(rp)), mul(mul(n, r), coef(rm)), cy)) return 1;
          for (int j = 1; j + 1 < H; j++)
            for (int q = 0; q < 4; q++) {
              const int k = q < 3 ? q : 2;
              auto at = [&](int kk, int dj, int di) { return f[kk][j + dj][i + di]; };
              // face velocities: ux: u in x, v of the columns x-1, x above and below; uy: the other way round
              auto face = [&](auto t, int s) {
                typedef decltype(t) F;
                switch (4 * k + s) {
                  case 0: return F(at(0, 0, -1)) * F(0.5) + F(at(0, 0, 0)) * F(0.5);
                  case 1: return F(at(0, 0, 0)) * F(0.5) + F(at(0, 0, 1)) * F(0.5);
                  case 2: return F(0.5) * F(at(1, 0, -1)) + F(0.5) * F(at(1, 0, 0));
                  case 3: return F(0.5) * F(at(1, 1, -1)) + F(0.5) * F(at(1, 1, 0));
                  case 4: return F(at(0, -1, 0)) * F(0.5) + F(at(0, 0, 0)) * F(0.5);
                  case 5: return F(at(0, -1, 1)) * F(0.5) + F(at(0, 0, 1)) * F(0.5);
                  case 6: return F(0.5) * F(at(1, -1, 0)) + F(0.5) * F(at(1, 0, 0));
                  case 7: return F(0.5) * F(at(1, 0, 0)) + F(0.5) * F(at(1, 1, 0));
                  case 8: return F(at(0, 0, 0));
                  case 9: return F(at(0, 0, 1));
                  case 10: return F(at(1, 0, 0));
                  default: return F(at(1, 1, 0));
                }
              };
              auto whole = [&](auto t) {
                typedef decltype(t) F;
                return expression<F>(at(k, 0, 0), at(k, 0, -1), at(k, 0, 1), at(k, -1, 0), at(k, 1, 0), face(t, 0),
                                     face(t, 1), face(t, 2), face(t, 3), rx, rm, rp, rx, nu, q < 3);
              };
              const long double want = whole((long double)0);
              const double fp = whole(0.0);
              auto M = [&](int kk, int dj, int di) { return num(at(kk, dj, di)); };
              const Num l = M(k, 0, -1), c = M(k, 0, 0), rt = M(k, 0, 1), d = M(k, -1, 0), u = M(k, 1, 0);
              Sum t;
              Vels v;
              if (!vels(v, M(0, 0, -1), M(0, 0, 0), M(0, 0, 1), M(0, -1, 0), M(0, -1, 1), M(0, 1, 0), M(1, 0, -1),
                        M(1, 0, 0), M(1, 0, 1), M(1, -1, 0), M(1, 1, 0), M(1, 1, -1)))
                return 2;
              if (k == 0) {
                t = sum_ux<false, false, EQ>(K, w, v);
              } else if (k == 1) {
                t = sum_uy<false, false, EQ>(K, v);
              } else if (!(q == 2 ? sum_temp<false, false, EQ>(t, K, l, c, rt, d, u, M(0, 0, 0), M(0, 0, 1), M(1, 0, 0),
                                                           M(1, 1, 0))
                                  : sum_temp<true, true, EQ>(t, K, l, c, rt, d, u, M(0, 0, 0), M(0, 0, 1), M(1, 0, 0),
                                                         M(1, 1, 0)))) {
                return 2;
              }
              const double fix = to_double(q < 3 ? t.A : t.G);
              e2[q][0] += std::pow((double)(fix - want), 2);
              e2[q][1] += std::pow((double)(fp - want), 2);
              e2[q][2] += std::pow((double)want, 2);
            }
        }
      }
      for (int q = 0; q < 4; q++)
        printf("%d %d %d %d %.3e %.3e\n", (int)EQ, N, kind, q, std::sqrt(e2[q][0] / e2[q][2]), std::sqrt(e2[q][1] / e2[q][2]));
    }
  return 0;
}

int main(int argc, char **argv) { return check<true>(argc, argv) | check<false>(argc, argv); }
