// Set-up kernels: what admitting a case or switching forms computes once per
// grid cell or per Fourier mode. Compiled without contraction, every operation
// in the order of its host counterpart (host_common.h, batch_api.cpp), so the
// values are the host's bit for bit.
#include <algorithm>
#include <cstdint>

#include "host_common.h"
#include "setup_internal.h"

namespace sns {
namespace {

// partition_factors_tri (host_common.h) of the Poisson lines: a warp per mode,
// a lane per segment; divisions and serial chains of nx/32 rows bound it. In
// host loops they were most of an admission (256 x 512: 1.7 ms, now 0.08 ms
// in all) and of the first switch to the parallel form (2048 x 4096: 97 ms,
// now 0.5).
__global__ void __launch_bounds__(128) k_partition_factors(const PoissonLines p) {
  const int lane = threadIdx.x & 31, J = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (J >= p.nh) return;  // the whole warp
  const int n = p.n, m = n / kPartSeg, s = lane * m, e = s + m - 1;
  const double eig = p.eig[J];
  auto at = [&](int i) -> size_t { return p.interleave ? (size_t)(i % m) * kPartSeg + i / m : (size_t)i; };
  // row i of the mode's line; the ends' raw couplings stay in the diagonal (Neumann closure)
  auto A = [&](int i) { return p.lo[at(i)]; };
  auto Cc = [&](int i) { return p.hi[at(i)]; };
  auto Dg = [&](int i) {
    const double l = i == 0 ? p.l_first : A(i), u = i == n - 1 ? p.u_last : Cc(i);
    double d = -l - u + eig;
    if (i == 0) d += p.l_first;
    if (i == n - 1) d += p.u_last;
    return d;
  };
  double *out = p.out + p.stride * (size_t)J;
  double *inv = out, *g = out + n, *up = p.with_g ? g + n : g, *v = up + n, *w = v + n;
  double *alpha = w + n, *beta = alpha + kPartLevels * kPartSeg, *rD = beta + kPartLevels * kPartSeg;
  // interior block rows s .. e-1: factors, and the spikes' forward pass beside them
  double iv = 1.0 / Dg(s), u = Cc(s) * iv;
  double rv = -A(s) * iv, rw = m == 2 ? -Cc(e - 1) * iv : 0.0;
  inv[at(s)] = iv;
  if (p.with_g) g[at(s)] = A(s) * iv;
  up[at(s)] = u;
  v[at(s)] = rv;
  w[at(s)] = rw;
  for (int i = s + 1; i < e; ++i) {
    const double a = A(i), c = Cc(i);
    iv = 1.0 / (Dg(i) - a * u);
    u = c * iv;
    rv = iv * (0.0 - a * rv);
    rw = iv * ((i == e - 1 ? -c : 0.0) - a * rw);
    inv[at(i)] = iv;
    if (p.with_g) g[at(i)] = a * iv;
    up[at(i)] = u;
    v[at(i)] = rv;
    w[at(i)] = rw;
  }
  const double ve = rv, we = rw;  // rows e-1: unchanged by the back substitution
  for (int i = e - 2; i >= s; --i) {
    const double ui = up[at(i)];
    rv = v[at(i)] - ui * rv;
    rw = w[at(i)] - ui * rw;
    v[at(i)] = rv;
    w[at(i)] = rw;
  }
  // the interface row: an interior-less value for the host's zeroed rows
  inv[at(e)] = 0.0;
  if (p.with_g) g[at(e)] = A(e) * 0.0;
  up[at(e)] = 0.0;
  v[at(e)] = 0.0;
  w[at(e)] = 0.0;
  // interface equations (the next segment's first interior row from the next lane)
  const double ae = A(e), ce = Cc(e);
  const double v1 = __shfl_down_sync(0xffffffffu, rv, 1), w1 = __shfl_down_sync(0xffffffffu, rw, 1);
  double L = ae * ve, D = ae * we + Dg(e), U = 0.0;
  if (lane < kPartSeg - 1) {
    D += ce * v1;
    U = ce * w1;
  }
  if (J == 0 && lane == kPartSeg - 1) {  // the mean mode: last unknown pinned to 0
    L = 0.0;
    D = 1.0;
    U = 0.0;
  }
  for (int lev = 0; lev < kPartLevels; ++lev) {
    const int d = 1 << lev;
    const double Lm = __shfl_up_sync(0xffffffffu, L, d), Dm = __shfl_up_sync(0xffffffffu, D, d),
                 Um = __shfl_up_sync(0xffffffffu, U, d), Lp = __shfl_down_sync(0xffffffffu, L, d),
                 Dp = __shfl_down_sync(0xffffffffu, D, d), Up = __shfl_down_sync(0xffffffffu, U, d);
    const bool hm = lane >= d, hp = lane + d < kPartSeg;
    const double al = hm ? -L / Dm : 0.0, be = hp ? -U / Dp : 0.0;
    alpha[lev * kPartSeg + lane] = al;
    beta[lev * kPartSeg + lane] = be;
    D = D + (hm ? al * Um : 0.0) + (hp ? be * Lp : 0.0);
    L = hm ? al * Lm : 0.0;
    U = hp ? be * Up : 0.0;
  }
  rD[lane] = 1.0 / D;
}

__device__ __forceinline__ void split_pair(double v, float *hi, float *lo) {
  const float h = (float)v;
  *hi = h;
  *lo = (float)(v - (double)h);
}

// the seeded initial temperature of a batched case (batch_api.cpp,
// initial_temperature): SplitMix64's k-th value from its counter
__global__ void __launch_bounds__(256) k_seeded_temperature(int nx, size_t cells, unsigned long long seed,
                                                            const double *__restrict__ xc, double xm, double xp,
                                                            float *__restrict__ hi, float *__restrict__ lo) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < cells; k += (size_t)gridDim.x * blockDim.x) {
    unsigned long long z = seed + (k + 1) * 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    const double r = (double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5;
    split_pair((xp - xm) * xc[k % nx] + xm + 0.1 * r, hi + k, lo + k);
  }
}

__global__ void __launch_bounds__(256) k_split(size_t n, const double *__restrict__ in, float *__restrict__ hi,
                                               float *__restrict__ lo) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
    split_pair(in[k], hi + k, lo + k);
}

int blocks_for(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 152 * 8); }

}  // namespace

cudaError_t launch_partition_factors(const PoissonLines &p, cudaStream_t st) {
  k_partition_factors<<<(p.nh + 3) / 4, 128, 0, st>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_seeded_temperature(int nx, int ny, unsigned long long seed, const double *xc, double xm, double xp,
                                      float *hi, float *lo, cudaStream_t st) {
  const size_t n = (size_t)nx * ny;
  k_seeded_temperature<<<blocks_for(n), 256, 0, st>>>(nx, n, seed, xc, xm, xp, hi, lo);
  return cudaGetLastError();
}

cudaError_t launch_split(size_t n, const double *in, float *hi, float *lo, cudaStream_t st) {
  k_split<<<blocks_for(n), 256, 0, st>>>(n, in, hi, lo);
  return cudaGetLastError();
}

}  // namespace sns
