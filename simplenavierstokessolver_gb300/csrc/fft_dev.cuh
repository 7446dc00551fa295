// Device real FFT along y shared by the plain FP64 path and the FP32-stencil
// form (same algorithm and operation order as the CPU FFT of the oracle:
// radix-2/4 decimation in time on z[m] = x[2m] + i x[2m+1], in place in
// shared memory, then the real-FFT split step; FFTW's conventions).
// Translation units compiled with --fmad=false reproduce the CPU FFT bit for
// bit; others may contract multiply-adds.
#pragma once

#include <type_traits>

namespace sns {
namespace fft {

// the threads that work on one group of columns: the whole block, or (Part) a
// part of it that meets at a named barrier of its own
struct Block {
  __device__ __forceinline__ int tid() const { return threadIdx.x; }
  __device__ __forceinline__ int size() const { return blockDim.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
};
struct Part {
  int t, n, bar;
  __device__ __forceinline__ int tid() const { return t; }
  __device__ __forceinline__ int size() const { return n; }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(n) : "memory"); }
};

// slot of element idx before the in-place decimation-in-time stages: digit
// reversal over the stage radices (2 first when log2(M) is odd, then 4s)
__device__ __forceinline__ int fft_slot(int idx, int M, int nst, int first2) {
  int rest = idx, span = M, slot = 0;
  for (int s = nst - 1; s >= 0; --s) {
    if (s == 0 && first2) {
      span >>= 1;
      slot += (rest & 1) * span;
      rest >>= 1;
    } else {
      span >>= 2;
      slot += (rest & 3) * span;
      rest >>= 2;
    }
  }
  return slot;
}

// One radix-4 butterfly by 4 adjacent lanes, each with one input, its twiddle
// and one output: 10 FP64 instructions on the way instead of 34, the same
// operations on the same operands. Every lane of the warp takes part (`on`: its
// result is stored).
template <bool FWD>
__device__ __forceinline__ void butterfly4(double2 *z, bool on, int base, int L, int k, int tstep, const double2 *tw) {
  const int r = threadIdx.x & 3;
  double2 v = z[base + r * L];
  if (L > 1) {
    const double2 w = tw[r * k * tstep];
    const double xr = FWD ? v.x * w.x - v.y * w.y : v.x * w.x + v.y * w.y;
    const double xi = FWD ? v.x * w.y + v.y * w.x : v.y * w.x - v.x * w.y;
    if (r) v = make_double2(xr, xi);  // the first input has no twiddle
  }
  // inputs 0 and 2, 1 and 3: t0 = v0 + v2, t2 = v1 + v3, t1 = v0 - v2, t3 = v1 - v3
  const double px = __shfl_xor_sync(0xffffffffu, v.x, 2), py = __shfl_xor_sync(0xffffffffu, v.y, 2);
  double2 t = make_double2(px + (r < 2 ? v.x : -v.x), py + (r < 2 ? v.y : -v.y));
  if (r == 3) t = FWD ? make_double2(t.y, -t.x) : make_double2(-t.y, t.x);
  // t0 + t2, t0 - t2, t1 + t3, t1 - t3: outputs 0, 2, 1, 3
  const double qx = __shfl_xor_sync(0xffffffffu, t.x, 1), qy = __shfl_xor_sync(0xffffffffu, t.y, 1);
  const double2 o = make_double2(qx + (r & 1 ? -t.x : t.x), qy + (r & 1 ? -t.y : t.y));
  if (on) z[base + (r == 1 ? 2 : r == 2 ? 1 : r) * L] = o;
}

// One in-place DIT stage on `cols` columns of length M held in shared memory;
// the same floating-point operations as dit_stage() of the CPU FFT.
// Part: where a stage has at most 32 butterflies (one warp), four lanes take
// one, so that all four sub-partitions have a warp. Fused Poisson launch, us:
// 64 x 128 34.9 -> 33.0, 128 x 256 51.2 -> 49.0; with 64 butterflies it would
// be 40 instructions on each against 34 on two: 400 x 512 118.6 -> 119.6.
template <bool FWD, typename Team = Block>
__device__ __forceinline__ void fft_stages(double2 *z, int cols, int M, int N, int nst, int first2,
                                           const double2 *tw, const Team team = Team()) {
  int L = 1, lg = 0;
  for (int st = 0; st < nst; ++st) {
    const int R = (st == 0 && first2) ? 2 : 4;
    const int span = R * L, tstep = N / span, nb = M / R;
    if constexpr (std::is_same_v<Team, Part>) {
      const int n = cols * nb, t = team.tid() >> 2;
      if (R == 4 && n <= 32 && 4 * n <= team.size()) {
        if ((team.tid() & ~31) < 4 * n) {  // whole warps
          const int b = min(t, n - 1), c = b / nb, bb = b - c * nb, k = bb & (L - 1);
          butterfly4<FWD>(z, t < n, c * M + (bb >> lg) * span + k, L, k, tstep, tw);
        }
        team.sync();
        L *= R;
        lg += 2;
        continue;
      }
    }
    for (int b = team.tid(); b < cols * nb; b += team.size()) {
      const int c = b / nb, bb = b - c * nb;
      const int k = bb & (L - 1);
      const int base = c * M + (bb >> lg) * span + k;
      double vr[4], vi[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r < R) {
          const double2 v = z[base + r * L];
          vr[r] = v.x;
          vi[r] = v.y;
        }
      }
      if (L > 1) {
#pragma unroll
        for (int r = 1; r < 4; ++r) {
          if (r < R) {
            const double2 w = tw[r * k * tstep];
            const double xr = vr[r], xi = vi[r];
            if (FWD) {
              vr[r] = xr * w.x - xi * w.y;
              vi[r] = xr * w.y + xi * w.x;
            } else {
              vr[r] = xr * w.x + xi * w.y;
              vi[r] = xi * w.x - xr * w.y;
            }
          }
        }
      }
      if (R == 2) {
        z[base] = make_double2(vr[0] + vr[1], vi[0] + vi[1]);
        z[base + L] = make_double2(vr[0] - vr[1], vi[0] - vi[1]);
      } else {
        const double t0r = vr[0] + vr[2], t0i = vi[0] + vi[2];
        const double t1r = vr[0] - vr[2], t1i = vi[0] - vi[2];
        const double t2r = vr[1] + vr[3], t2i = vi[1] + vi[3];
        const double t3r = vr[1] - vr[3], t3i = vi[1] - vi[3];
        const double sr = FWD ? t3i : -t3i;
        const double si = FWD ? -t3r : t3r;
        z[base] = make_double2(t0r + t2r, t0i + t2i);
        z[base + L] = make_double2(t1r + sr, t1i + si);
        z[base + 2 * L] = make_double2(t0r - t2r, t0i - t2i);
        z[base + 3 * L] = make_double2(t1r - sr, t1i - si);
      }
    }
    team.sync();
    L *= R;
    lg += (R == 2) ? 1 : 2;
  }
}


// split step of the forward real FFT for bin pair (k, M-k) of one column,
// k in [0, M/2]: X[k] from the half-length complex spectrum Z (natural order)
// (bins of one column at out[J * os])
__device__ __forceinline__ void rfft_post(const double2 *zc, double2 *out, int M, int k, const double2 *tw,
                                          size_t os = 1) {
  if (k == 0) {
    const double2 z0 = zc[0];
    out[0] = make_double2(z0.x + z0.y, 0.0);
    out[(size_t)M * os] = make_double2(z0.x - z0.y, 0.0);
  } else {
    const double2 A = zc[k], B = zc[M - k];
    const double sre = A.x + B.x, dim = A.y - B.y, dre = A.x - B.x, sim = A.y + B.y;
    const double er = 0.5 * sre, ei = 0.5 * dim;
    const double orr = 0.5 * sim, oi = -(0.5 * dre);
    const double2 w = tw[k];
    const double wor = w.x * orr - w.y * oi;
    const double woi = w.x * oi + w.y * orr;
    out[(size_t)k * os] = make_double2(er + wor, ei + woi);
    if (2 * k != M) out[(size_t)(M - k) * os] = make_double2(er - wor, woi - ei);
  }
}

// inverse split step for bin pair (k, M-k): Z slots (digit-reversed) from X
// (bins of one column at in[J * is]);
// imaginary parts of X[0] and X[M] are ignored (FFTW c2r convention)
// CG: load the input through L2 only (data written by other blocks of the running kernel)
template <bool CG = false>
__device__ __forceinline__ void rfft_pre(const double2 *in, double2 *zc, int M, int k, const double2 *tw, int nst,
                                         int first2, size_t is = 1) {
  auto ld = [](const double2 *p) -> double2 {
    if constexpr (CG) {
      return __ldcg(p);
    } else {
      return *p;
    }
  };
  if (k == 0) {
    const double x0r = ld(in).x, xmr = ld(in + (size_t)M * is).x;
    zc[0] = make_double2(x0r + xmr, x0r - xmr);
  } else {
    const double2 A = ld(in + (size_t)k * is), B = ld(in + (size_t)(M - k) * is);
    const double er = A.x + B.x, ei = A.y - B.y, dr = A.x - B.x, di = A.y + B.y;
    const double2 w = tw[k];
    const double orr = dr * w.x + di * w.y;
    const double oi = di * w.x - dr * w.y;
    zc[fft_slot(k, M, nst, first2)] = make_double2(er - oi, ei + orr);
    if (2 * k != M) zc[fft_slot(M - k, M, nst, first2)] = make_double2(er + oi, orr - ei);
  }
}

}  // namespace fft
}  // namespace sns
