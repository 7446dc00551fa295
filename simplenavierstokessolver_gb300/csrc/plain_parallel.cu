// Parallel form of the plain FP64 step's line solves and DFTs on GB300.
//
// The reference solves each Fourier mode's x-line with a serial Thomas
// recurrence (src/fluid/compute_potential.c:109-136, src/linalg.c:32-50).
// Reproduced bit for bit, that recurrence is a chain of 3 + 2 dependent FP64
// operations per x, which on GB300 (~70 cycles per dependent FP64 operation)
// bounds the plain step no matter how many lines run side by side. This
// form solves the same lines by the partition method with warp-shuffle
// parallel cyclic reduction (PCR): a warp per part (real, imaginary) of a
// mode line, one lane per segment of nx/32 rows, a 32-unknown interface
// system reduced in 5 shuffle levels. All RHS-independent factors (interior
// Thomas factors, spikes, PCR coefficients) are computed once on the host.
// Its results differ from the Thomas recurrence by rounding only, so the
// form is held to the path's tolerance (1e-12 relative L2 per field after
// the stated step counts) rather than to bit identity, and this unit is
// compiled with floating-point contraction.
//
// Layout: the spectrum is mode-major, spec[J * nx + p], with the rows of a
// mode line in the interleaved order p = (x % m) * 32 + x / m (m = nx / 32):
// lane k walks segment k, and at every step the 32 lanes touch 32
// consecutive elements, in global and in shared memory alike. The forward
// and inverse DFTs write and read that order: in 64-bit fixed point for
// 16 <= jtot <= 8192 (fft_fixed.cuh), by the Thomas form's radix-2/4 FFT
// otherwise.
//
// The Crank-Nicolson lines (src/linalg.c:9-108) are solved by the same
// partition method: one warp per row along x (k_par_cn), one thread per
// segment of a column along y (k_par_cn_cols).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fft_dev.cuh"
#include "fft_fixed.cuh"
#include "host_common.h"
#include "sns_gpu.h"
#include "smem_grant.h"
#include "sns_internal.h"
#include "chain.cuh"

namespace sns {
namespace {

constexpr int kParWarpsMax = 8;  // warps per block of the PCR kernel (two per mode line)
constexpr size_t kParSmemMax = 220 * 1024;

struct ParArgs {
  DevGrid g;
  StageScalars s;
  const double *ux, *uy;
  double2 *spec;  // [nh][nx], interleaved rows
  double *psi;
  int cols;       // adjacent x columns per block of the DFT kernels
  int m;          // rows per segment, nx / 32
};

// line position of column x (rows of a mode line interleaved by segment)
__device__ __forceinline__ int par_p(int x, int m) { return (x % m) * kPartSeg + x / m; }

// src/fluid/compute_potential.c:69-92: (div u*)/(gamma dt) and its real DFT
// along y, for the adjacent columns x0 .. x0+cols-1 (coalesced reads of the
// velocity); each column's spectrum goes to its line position
__global__ void __launch_bounds__(256) k_par_fwd(const ParArgs a) {
  chain_begin();
  extern __shared__ double2 z[];
  const int nx = a.g.nx, ny = a.g.ny, M = ny / 2, C = a.cols;
  const int x0 = blockIdx.x * C;
  double *zd = reinterpret_cast<double *>(z);
  const double rdy = a.g.rdy, rgdt = a.s.rgdt;
  for (int e = threadIdx.x; e < C * ny; e += blockDim.x) {
    const int c = e % C, y = e / C, x = x0 + c;
    double d = 0.0;
    if (x < nx) {
      const size_t r = (size_t)y * nx + x;
      const double uxm = a.ux[r];
      const double uxp = x == nx - 1 ? 0.0 : a.ux[r + 1];
      const double uym = a.uy[r];
      const double uyp = a.uy[(size_t)(y + 1 == ny ? 0 : y + 1) * nx + x];
      d = rgdt * ((uxp - uxm) * a.g.rdxf[x] + (uyp - uym) * rdy);
    }
    zd[2 * (c * M + fft::fft_slot(y >> 1, M, a.g.fft_nst, a.g.fft_first2)) + (y & 1)] = d;
  }
  __syncthreads();
  const double2 *tw = reinterpret_cast<const double2 *>(a.g.tw);
  fft::fft_stages<true>(z, C, M, ny, a.g.fft_nst, a.g.fft_first2, tw);
  const int half = M / 2 + 1;
  for (int e = threadIdx.x; e < C * half; e += blockDim.x) {
    const int c = e % C, k = e / C, x = x0 + c;
    if (x < nx) fft::rfft_post(z + c * M, a.spec + par_p(x, a.m), M, k, tw, (size_t)nx);
  }
}

// src/fluid/compute_potential.c:146-157: inverse real DFT and 1/jtot
__global__ void __launch_bounds__(256) k_par_bwd(const ParArgs a) {
  chain_begin();
  extern __shared__ double2 z[];
  const int nx = a.g.nx, ny = a.g.ny, M = ny / 2, C = a.cols;
  const int x0 = blockIdx.x * C;
  const double2 *tw = reinterpret_cast<const double2 *>(a.g.tw);
  const int half = M / 2 + 1;
  for (int e = threadIdx.x; e < C * half; e += blockDim.x) {
    const int c = e % C, k = e / C, x = x0 + c;
    double2 *zc = z + c * M;
    if (x >= nx) {
      zc[fft::fft_slot(k, M, a.g.fft_nst, a.g.fft_first2)] = make_double2(0.0, 0.0);
      if (k > 0) zc[fft::fft_slot(M - k, M, a.g.fft_nst, a.g.fft_first2)] = make_double2(0.0, 0.0);
      continue;
    }
    fft::rfft_pre(a.spec + par_p(x, a.m), zc, M, k, tw, a.g.fft_nst, a.g.fft_first2, (size_t)nx);
  }
  __syncthreads();
  fft::fft_stages<false>(z, C, M, ny, a.g.fft_nst, a.g.fft_first2, tw);
  const double *zd = reinterpret_cast<const double *>(z);
  for (int e = threadIdx.x; e < C * ny; e += blockDim.x) {
    const int c = e % C, y = e / C, x = x0 + c;
    if (x >= nx) continue;
    a.psi[(size_t)y * nx + x] = zd[2 * (c * M + (y >> 1)) + (y & 1)] * a.s.rny;
  }
}

// ---- the same two transforms in 64-bit fixed point (fft_fixed.cuh), for
// 16 <= jtot <= 8192: 3 FP64 instructions per value forward and 2 inverse, the
// rest integer, where the FP64 transforms took about 20 each. The solve is
// linear, so this pair moves two constant
// factors to the inverse's final scale: the forward transforms div u* without
// the factor 1/(gamma dt) and leaves the real FFT's split step unhalved
// (2 X), and the inverse multiplies by 1/(gamma dt) / (2 jtot).

struct FixArgs {
  DevGrid g;
  const double *ux, *uy;
  double2 *spec;  // [nh][nx], interleaved rows
  double *psi;
  double scale;   // of the inverse
  int lgC;        // 2^lgC adjacent x columns per block
  int m;          // rows per segment, nx / 32
};

// src/fluid/compute_potential.c:69-92: div u* along two rows per complex
// element (z[m] = d[2m] + i d[2m+1]) and 2 X[k] of its real transform at the
// columns' line positions. On uniform grids whose spacings are powers of two
// (DevGrid::p2u) the divergence is formed without the factor 1/dx, which joins the exponent:
// the same bits in 3 FP64 instructions per value instead of 4.
template <int V>
__global__ void __launch_bounds__(512, 1) k_par_fwd_fx(const FixArgs a) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char fx_sm[];
  __shared__ fx::Slots slots;
  const int nx = a.g.nx, ny = a.g.ny, x0 = blockIdx.x << a.lgC;
  const double rdy = a.g.rdy;
  const bool p2 = a.g.p2u;
  const int eoff = p2 ? ((__double2hiint(a.g.rdxf[0]) >> 20) & 0x7ff) - 1023 : 0;
  const double ratio = p2 ? rdy * a.g.dxf[0] : 0.0;
  auto in = [&](int c, int mm, double *d) {
    const int x = x0 + c;
    d[0] = d[1] = 0.0;
    if (x >= nx) return;
    const size_t r0 = (size_t)(2 * mm) * nx + x, r1 = r0 + nx;
    const size_t r2 = (size_t)(2 * mm + 2 == ny ? 0 : 2 * mm + 2) * nx + x;
    const bool right = x == nx - 1;
    const double u0m = a.ux[r0], u0p = right ? 0.0 : a.ux[r0 + 1];
    const double u1m = a.ux[r1], u1p = right ? 0.0 : a.ux[r1 + 1];
    const double v0 = a.uy[r0], v1 = a.uy[r1], v2 = a.uy[r2];
    if (p2) {
      d[0] = fma(v1 - v0, ratio, u0p - u0m);
      d[1] = fma(v2 - v1, ratio, u1p - u1m);
    } else {
      const double rdx = a.g.rdxf[x];
      d[0] = (u0p - u0m) * rdx + (v1 - v0) * rdy;
      d[1] = (u1p - u1m) * rdx + (v2 - v1) * rdy;
    }
  };
  auto out = [&](int c, int k, double2 X) {
    const int x = x0 + c;
    if (x < nx) a.spec[(size_t)k * nx + par_p(x, a.m)] = X;
  };
  fx::forward<V>(reinterpret_cast<fx::C64 *>(fx_sm), &slots, a.lgC, ny / 2, reinterpret_cast<const fx::Tw *>(a.g.twx),
              eoff, fx::doubles(in), out);
}

// src/fluid/compute_potential.c:146-157: the inverse into psi
template <int V>
__global__ void __launch_bounds__(512, 1) k_par_bwd_fx(const FixArgs a) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char fx_sm[];
  __shared__ fx::Slots slots;
  const int nx = a.g.nx, x0 = blockIdx.x << a.lgC;
  auto in = [&](int c, int k) -> double2 {
    const int x = x0 + c;
    return x < nx ? a.spec[(size_t)k * nx + par_p(x, a.m)] : make_double2(0.0, 0.0);
  };
  auto out = [&](int c, int mm, const double *d) {
    const int x = x0 + c;
    if (x >= nx) return;
    const size_t r0 = (size_t)(2 * mm) * nx + x;
    a.psi[r0] = d[0];
    a.psi[r0 + nx] = d[1];
  };
  fx::inverse<V>(reinterpret_cast<fx::C64 *>(fx_sm), &slots, a.lgC, a.g.ny / 2,
              reinterpret_cast<const fx::Tw *>(a.g.twx), a.scale, in, out);
}

struct ParTriArgs {
  double2 *spec;       // [nh][nx], interleaved rows
  const double *fac;   // [nh][stride]: inv g up v w (interleaved rows, g = a inv), alpha, beta, rD
  const double *lo;    // [nx] sub-diagonal a_i, interleaved rows (a_0 = 0)
  const double *hi;    // [nx] super-diagonal c_i, interleaved rows (c_{nx-1} = 0)
  size_t stride;       // doubles per mode in fac
  int nx, nh, m;
  unsigned *err;       // set to 1 when a copy wait gave up (the line is then left unsolved)
  unsigned spin_limit; // polls of a copy wait before it gives up
  int stale;           // test of the bounded wait: issue no copy, so the wait runs out
};

// polls of the wait that lets a warp's copies land after its first wait gave
// up, so that no copy into the warp's shared memory outlives the warp
constexpr unsigned kParDrainSpins = 1u << 22;

__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// rows per chunk of the segment sweeps: the next chunk's factors are loaded
// while the current chunk is eliminated, off the dependent chain
constexpr int kParChunk = 8;

// src/fluid/compute_potential.c:109-136 by the partition method: two warps
// per mode line, one for its real and one for its imaginary part (both see
// the same real matrix and never mix, so each part takes the operations it
// took when one warp carried both). The first warp's lane 0 moves the line
// (16 nx bytes) into shared memory with a bulk asynchronous copy (completion
// on an mbarrier both warps wait on, bounded), STAGED: also the mode's factor
// block; otherwise the factors are read from global memory, coalesced by the
// interleaved row order, a chunk ahead. Each warp solves its part in shared
// memory and writes it back.
template <bool STAGED>
__global__ void __launch_bounds__(32 * kParWarpsMax) k_par_tri(const ParTriArgs a) {
  chain_begin();
  extern __shared__ __align__(128) unsigned char sm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int li = w >> 1, comp = w & 1;  // line of the block, part (0 real, 1 imaginary)
  const int J = blockIdx.x * (blockDim.x >> 6) + li;
  if (J >= a.nh) return;  // both warps of the line
  const int n = a.nx, m = a.m;
  const size_t per_line = 16 * (size_t)n + (STAGED ? 8 * a.stride : 0);
  double2 *line = reinterpret_cast<double2 *>(sm + 128 + (size_t)li * per_line);
  double *lc = reinterpret_cast<double *>(line) + comp;  // this part of element i at lc[2 i]
  double *fs = reinterpret_cast<double *>(line + n);
  double2 *gline = a.spec + (size_t)J * n;
  const double *gfac = a.fac + (size_t)J * a.stride;
  const unsigned bar = smem_u32(reinterpret_cast<unsigned long long *>(sm) + li);
  const unsigned line_bytes = 16u * (unsigned)n, fac_bytes = STAGED ? 8u * (unsigned)a.stride : 0u;
  if (comp == 0 && lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(line_bytes + fac_bytes)
                 : "memory");
    if (!a.stale) {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       smem_u32(line)),
                   "l"(__cvta_generic_to_global(gline)), "r"(line_bytes), "r"(bar)
                   : "memory");
      if (STAGED)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(fs)),
                     "l"(__cvta_generic_to_global(gfac)), "r"(fac_bytes), "r"(bar)
                     : "memory");
    }
  }
  // the line's two warps: the mbarrier is initialised before either waits on it
  asm volatile("bar.sync %0, 64;" ::"r"(1 + li) : "memory");
  const double *f = STAGED ? fs : gfac;
  auto ld = [&](const double *p) -> double {
    if constexpr (STAGED) {
      return *p;
    } else {
      return __ldg(p);
    }
  };
  const double *inv = f, *gg = f + n, *up = f + 2 * n, *vv = f + 3 * n, *ww = f + 4 * n;
  const double *alpha = f + 5 * n, *beta = alpha + kPartLevels * kPartSeg, *rD = beta + kPartLevels * kPartSeg;
  // global form: the first chunk's factors while the copy lands
  double ci[kParChunk], cg[kParChunk];
  const double inv0 = STAGED ? 0.0 : ld(inv + lane);
  if constexpr (!STAGED) {
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = 1 + k, i = r * kPartSeg + lane;
      ci[k] = r < m - 1 ? ld(inv + i) : 0.0;
      cg[k] = r < m - 1 ? ld(gg + i) : 0.0;
    }
  }
  bool done = false;
  for (unsigned k = 0; k < a.spin_limit && !done; ++k) done = mbar_try(bar, 0u);
  if (!done) {
    if (lane == 0) atomicOr(a.err, 1u);
    // leave the line unsolved, but only once the copies issued into this
    // line's shared memory have landed (bounded as well)
    if (!a.stale)
      for (unsigned k = 0; k < kParDrainSpins && !mbar_try(bar, 0u); ++k) {
      }
    return;
  }
  if constexpr (STAGED) {
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = 1 + k, i = r * kPartSeg + lane;
      ci[k] = r < m - 1 ? ld(inv + i) : 0.0;
      cg[k] = r < m - 1 ? ld(gg + i) : 0.0;
    }
  }
  // 1) the segment's interior rows r = 0 .. m-2 (line index r*32 + lane)
  //    with zero boundary values: forward elimination and back substitution.
  //    y_r = inv_r q_r - g_r y_{r-1} with g_r = a_r inv_r: one FMA per row on
  //    the dependent chain, the product inv_r q_r off it
  double y = lc[2 * lane];
  {
    const double i0 = STAGED ? ld(inv + lane) : inv0;
    y *= i0;
  }
  lc[2 * lane] = y;
#pragma unroll 1
  for (int b = 1; b < m - 1; b += kParChunk) {
    double ni[kParChunk], ng[kParChunk];
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b + kParChunk + k, i = r * kPartSeg + lane;
      ni[k] = r < m - 1 ? ld(inv + i) : 0.0;
      ng[k] = r < m - 1 ? ld(gg + i) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b + k, i = r * kPartSeg + lane;
      if (r < m - 1) {
        const double q = fma(-cg[k], y, ci[k] * lc[2 * i]);
        lc[2 * i] = q;
        y = q;
      }
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      ci[k] = ni[k];
      cg[k] = ng[k];
    }
  }
  const double ylast = y;  // row m-2
  double cu[kParChunk];
#pragma unroll
  for (int k = 0; k < kParChunk; ++k) {
    const int r = m - 3 - k;
    cu[k] = r >= 0 ? ld(up + r * kPartSeg + lane) : 0.0;
  }
#pragma unroll 1
  for (int b = m - 3; b >= 0; b -= kParChunk) {
    double nu[kParChunk];
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b - kParChunk - k;
      nu[k] = r >= 0 ? ld(up + r * kPartSeg + lane) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b - k, i = r * kPartSeg + lane;
      if (r >= 0) {
        const double q = fma(-cu[k], y, lc[2 * i]);
        lc[2 * i] = q;
        y = q;
      }
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) cu[k] = nu[k];
  }
  // y: the first interior value (row 0). 2) right-hand side of the interface
  // row e: r_e - a_e y_{e-1} - c_e y'_0 (y'_0 of the next segment)
  const int ie = (m - 1) * kPartSeg + lane;
  const double yn = __shfl_down_sync(0xffffffffu, y, 1);
  const double re = lc[2 * ie];
  const double ae = __ldg(a.lo + ie), ce = lane < kPartSeg - 1 ? __ldg(a.hi + ie) : 0.0;
  double R = re - ae * ylast - ce * (lane < kPartSeg - 1 ? yn : 0.0);
  if (J == 0 && lane == kPartSeg - 1) R = 0.0;  // the mean mode: last unknown pinned to 0
  // 3) parallel cyclic reduction of the 32 interface equations
#pragma unroll
  for (int lev = 0; lev < kPartLevels; ++lev) {
    const int d = 1 << lev;
    const double mv = __shfl_up_sync(0xffffffffu, R, d);
    const double pv = __shfl_down_sync(0xffffffffu, R, d);
    const double al = ld(alpha + lev * kPartSeg + lane), be = ld(beta + lev * kPartSeg + lane);
    const double lm = lane >= d ? mv : 0.0;
    const double lp = lane + d < kPartSeg ? pv : 0.0;
    R = fma(be, lp, fma(al, lm, R));
  }
  const double xe = R * ld(rD + lane);
  lc[2 * ie] = xe;
  // 4) interiors from the spikes: x_i = y_i + v_i x_{e(k-1)} + w_i x_{e(k)}
  const double xl = __shfl_up_sync(0xffffffffu, xe, 1);
  const double lx = lane > 0 ? xl : 0.0;
#pragma unroll 1
  for (int b = 0; b < m - 1; b += kParChunk) {
    double cv[kParChunk], cw[kParChunk];
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b + k, i = r * kPartSeg + lane;
      cv[k] = r < m - 1 ? ld(vv + i) : 0.0;
      cw[k] = r < m - 1 ? ld(ww + i) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b + k, i = r * kPartSeg + lane;
      if (r < m - 1) lc[2 * i] = fma(cw[k], xe, fma(cv[k], lx, lc[2 * i]));
    }
  }
  __syncwarp();
  double *gc = reinterpret_cast<double *>(gline) + comp;
  for (int i = lane; i < n; i += 32) gc[2 * i] = lc[2 * i];
}

// ------------------------------------------------------------------------
// Crank-Nicolson lines by the partition method: src/linalg.c:9-30 along x
// (rows of a field, wall-bounded: src/temperature/update.c:141-157,
// src/fluid/update_velocity.c:249-280 and :500-520) and src/linalg.c:52-108
// along y (columns, periodic: src/temperature/update.c:189-207,
// src/fluid/update_velocity.c:404-430). A line of n rows is cut into 32
// segments of m = n / 32 rows; a periodic line's interface system is
// cyclic (its PCR levels couple modulo 32). All RHS-independent factors are
// computed on the host per substage (they depend on dt). Both kernels do
// the same operations on every element, in the same order.

constexpr int kCnWarpsMax = 8;
constexpr int kCnLoad = 8;  // elements in flight per thread while gathering a row

// factor block of a field's lines: inv g up v w (rows interleaved: row r of
// segment k at r * 32 + k), alpha beta (PCR levels), rD, then the interface
// rows' sub- and super-diagonals
struct CnFac {
  const double *inv, *gg, *up, *vv, *ww, *alpha, *beta, *rD, *ae, *ce;
  __device__ __forceinline__ CnFac(const double *f, int n)
      : inv(f), gg(f + n), up(f + 2 * n), vv(f + 3 * n), ww(f + 4 * n), alpha(f + 5 * (size_t)n),
        beta(alpha + kPartLevels * kPartSeg), rD(beta + kPartLevels * kPartSeg), ae(rD + kPartSeg),
        ce(ae + kPartSeg) {}
};

__device__ __forceinline__ ParCnField cn_field(const ParCnArgs &a) {
  // a select, not an index into the parameter array (which would copy the
  // array to the stack)
  return blockIdx.y == 0 ? a.f[0] : blockIdx.y == 1 ? a.f[1] : a.f[2];
}

__device__ __forceinline__ int cn_pos(int e, int m, int s) {
  const int k = e / m;
  return k * s + (e - k * m);
}

// Rows along x (wall-bounded): one warp per row, one lane per segment; the
// row is gathered into shared memory with each segment at a stride s = m | 1
// (odd, so that the 32 lanes' accesses at one row fall on distinct bank
// pairs), solved there and written back, coalesced both ways. FP64 issue
// bounds it: three instructions a row and two more where the interface values
// reach (three fields of 2048 x 4096: 357 us with the spikes over all rows, 313
// at dt 0.035, 305 at 0.002).
__global__ void __launch_bounds__(32 * kCnWarpsMax) k_par_cn(const ParCnArgs a) {
  chain_begin();
  extern __shared__ __align__(16) double cn_sm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const ParCnField F = cn_field(a);
  const int n = a.n, m = a.m, s = a.s;
  const int line = F.first + blockIdx.x * wpb + w;
  if (line >= a.lines) return;  // the whole warp
  double *sl = cn_sm + (size_t)w * ((size_t)kPartSeg * s + 8);
  const double *src = F.q + (size_t)line * a.ls;
  for (int e0 = lane; e0 < n; e0 += 32 * kCnLoad) {
    double v[kCnLoad];
#pragma unroll
    for (int k = 0; k < kCnLoad; ++k) {
      const int e = e0 + 32 * k;
      v[k] = e < n ? src[e] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kCnLoad; ++k) {
      const int e = e0 + 32 * k;
      if (e < n) sl[cn_pos(e, m, s)] = v[k];
    }
  }
  __syncwarp();
  const CnFac f(F.fac, n);
  double *seg = sl + lane * s;
  // 1) interior rows r = 0 .. m-2 with zero interface values:
  //    y_r = inv_r q_r - g_r y_{r-1}, then y_r -= up_r y_{r+1}
  double y = seg[0] * __ldg(f.inv + lane);
  seg[0] = y;
  double ci[kParChunk], cg[kParChunk];
#pragma unroll
  for (int k = 0; k < kParChunk; ++k) {
    const int r = 1 + k, i = r * kPartSeg + lane;
    ci[k] = r < m - 1 ? __ldg(f.inv + i) : 0.0;
    cg[k] = r < m - 1 ? __ldg(f.gg + i) : 0.0;
  }
#pragma unroll 1
  for (int b = 1; b < m - 1; b += kParChunk) {
    double ni[kParChunk], ng[kParChunk];
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b + kParChunk + k, i = r * kPartSeg + lane;
      ni[k] = r < m - 1 ? __ldg(f.inv + i) : 0.0;
      ng[k] = r < m - 1 ? __ldg(f.gg + i) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b + k;
      if (r < m - 1) {
        y = fma(-cg[k], y, ci[k] * seg[r]);
        seg[r] = y;
      }
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      ci[k] = ni[k];
      cg[k] = ng[k];
    }
  }
  const double ylast = y;  // row m-2
  double cu[kParChunk];
#pragma unroll
  for (int k = 0; k < kParChunk; ++k) {
    const int r = m - 3 - k;
    cu[k] = r >= 0 ? __ldg(f.up + r * kPartSeg + lane) : 0.0;
  }
#pragma unroll 1
  for (int b = m - 3; b >= 0; b -= kParChunk) {
    double nu[kParChunk];
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b - kParChunk - k;
      nu[k] = r >= 0 ? __ldg(f.up + r * kPartSeg + lane) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) {
      const int r = b - k;
      if (r >= 0) {
        y = fma(-cu[k], y, seg[r]);
        seg[r] = y;
      }
    }
#pragma unroll
    for (int k = 0; k < kParChunk; ++k) cu[k] = nu[k];
  }
  // 2) interface row e of segment k: q_e - a_e y_{e-1} - c_e y'_0 (the next
  //    segment's first interior value; c_e = 0 for the last segment)
  const double ynext = __shfl_sync(0xffffffffu, y, (lane + 1) & 31);
  double R = fma(-__ldg(f.ce + lane), ynext, fma(-__ldg(f.ae + lane), ylast, seg[m - 1]));
  // 3) PCR of the 32 interface equations; the host zeroes the couplings
  //    past the ends of the line
#pragma unroll
  for (int lev = 0; lev < kPartLevels; ++lev) {
    const int d = 1 << lev;
    const double rm = __shfl_sync(0xffffffffu, R, (lane - d) & 31);
    const double rp = __shfl_sync(0xffffffffu, R, (lane + d) & 31);
    R = fma(__ldg(f.beta + lev * kPartSeg + lane), rp, fma(__ldg(f.alpha + lev * kPartSeg + lane), rm, R));
  }
  const double xe = R * __ldg(f.rD + lane);
  seg[m - 1] = xe;
  // 4) interiors: x_r = y_r + v_r x_{e(k-1)} + w_r x_{e(k)} (v = 0 in the
  //    first segment), where v and w reach
  const double xl = __shfl_sync(0xffffffffu, xe, (lane - 1) & 31);
  auto spike = [&](const double *factor, double x, int r0, int r1) {
#pragma unroll 1
    for (int b = r0; b < r1; b += kParChunk) {
      double cf[kParChunk];
#pragma unroll
      for (int k = 0; k < kParChunk; ++k) cf[k] = b + k < r1 ? __ldg(factor + (b + k) * kPartSeg + lane) : 0.0;
#pragma unroll
      for (int k = 0; k < kParChunk; ++k)
        if (b + k < r1) seg[b + k] = fma(cf[k], x, seg[b + k]);
    }
  };
  spike(f.vv, xl, 0, min(F.nv, m - 1));
  spike(f.ww, xe, max(m - 1 - F.nw, 0), m - 1);
  __syncwarp();
  const size_t g0 = (size_t)line * a.ls;
  if (F.add.out) {
    for (int e0 = lane; e0 < n; e0 += 32 * kCnLoad) {
      double old[kCnLoad];
#pragma unroll
      for (int k = 0; k < kCnLoad; ++k)
        if (e0 + 32 * k < n) old[k] = F.add.in[g0 + e0 + 32 * k];
#pragma unroll
      for (int k = 0; k < kCnLoad; ++k) {
        const int e = e0 + 32 * k;
        if (e < n && e >= F.low) F.add.out[g0 + e] = old[k] + sl[cn_pos(e, m, s)];
      }
    }
  } else {
    for (int e = lane; e < n; e += 32) F.q[g0 + e] = sl[cn_pos(e, m, s)];
  }
}

// Columns along y (periodic): a block takes kCnCols adjacent columns and
// all 32 segments of each, thread t column t % kCnCols and segment
// t / kCnCols, and walks its segment in place in global memory; a warp's
// access covers 4 rows of kCnCols columns (whole 64-byte pairs of sectors). The
// first interior values, the interface right-hand sides and the interface
// solutions pass between the threads of a column through shared memory;
// warp c solves column c's cyclic interface system with lane = segment.
// Same operations on every element as k_par_cn.
//
// Memory traffic bounds it at 2048 x 4096 (three fields of 67 MB, larger than
// L2 together), so a row is read and written twice: once going forward, once
// going back, where it takes its increment unless an interface value reaches it
// (ParCnField::nv, nw). Solve and increments, us: in 4 columns per block, the
// spikes over all rows and the increments in launches of their own 371 + 110,
// now 384; 1024 x 2048 111 + 33, now 95; 512 x 1024 53 + 12, now 47. (4 / 16
// columns with the rest as it is: 2048 x 4096 466 / 565, 1024 x 2048 100 / 173;
// chunks of 12 or 16 rows instead of kParChunk: 2048 x 4096 513.)
constexpr int kCnCols = 8;

__global__ void __launch_bounds__(32 * kCnCols) k_par_cn_cols(const ParCnArgs a) {
  chain_begin();
  __shared__ double ex[3][kCnCols][kPartSeg];
  const ParCnField F = cn_field(a);
  const int n = a.n, m = a.m;
  const int c = threadIdx.x % kCnCols, k = threadIdx.x / kCnCols;
  const int col = F.first + blockIdx.x * kCnCols + c;
  const bool live = col < a.lines;
  const size_t es = (size_t)a.es;
  double *q = F.q + (live ? col : 0);
  const double *in = F.add.out ? F.add.in + (live ? col : 0) : nullptr;
  double *out = F.add.out ? F.add.out + (live ? col : 0) : q;
  const int mid0 = min(F.nv, m - 1), mid1 = max(m - 1 - F.nw, mid0);  // at most m - 2 (nw >= 1)
  const CnFac f(F.fac, n);
  const size_t e0 = (size_t)k * m;  // first row of the segment
  double y = 0.0, ylast = 0.0;
  if (live) {
    // 1) interior rows r = 0 .. m-2: forward elimination, back substitution
    y = q[e0 * es] * __ldg(f.inv + k);
    q[e0 * es] = y;
#pragma unroll 1
    for (int b = 1; b < m - 1; b += kParChunk) {
      double q_[kParChunk];
#pragma unroll
      for (int j = 0; j < kParChunk; ++j) q_[j] = b + j < m - 1 ? q[(e0 + b + j) * es] : 0.0;
#pragma unroll
      for (int j = 0; j < kParChunk; ++j) {
        const int r = b + j;
        if (r >= m - 1) break;
        y = fma(-__ldg(f.gg + r * kPartSeg + k), y, __ldg(f.inv + r * kPartSeg + k) * q_[j]);
        q[(e0 + r) * es] = y;
      }
    }
    ylast = y;
    // rows that no interface value reaches are final now
#pragma unroll 1
    for (int b = m - 3; b >= 0; b -= kParChunk) {
      double y_[kParChunk], old[kParChunk];
#pragma unroll
      for (int j = 0; j < kParChunk; ++j) {
        const int r = b - j;
        y_[j] = r >= 0 ? q[(e0 + r) * es] : 0.0;
        old[j] = in && r >= mid0 && r < mid1 ? in[(e0 + r) * es] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < kParChunk; ++j) {
        const int r = b - j;
        if (r < 0) break;
        y = fma(-__ldg(f.up + r * kPartSeg + k), y, y_[j]);
        if (r >= mid0 && r < mid1) {
          out[(e0 + r) * es] = in ? old[j] + y : y;
        } else {
          q[(e0 + r) * es] = y;
        }
      }
    }
  }
  ex[0][c][k] = y;  // the segment's first interior value
  __syncthreads();
  // 2) interface row e of segment k (the next segment cyclically)
  double R = 0.0;
  if (live) {
    const double ynext = ex[0][c][(k + 1) & 31];
    R = fma(-__ldg(f.ce + k), ynext, fma(-__ldg(f.ae + k), ylast, q[(e0 + m - 1) * es]));
  }
  ex[1][c][k] = R;
  __syncthreads();
  // 3) PCR: warp w takes column w, lane = segment
  {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double Rw = ex[1][w][lane];
#pragma unroll
    for (int lev = 0; lev < kPartLevels; ++lev) {
      const int d = 1 << lev;
      const double rm = __shfl_sync(0xffffffffu, Rw, (lane - d) & 31);
      const double rp = __shfl_sync(0xffffffffu, Rw, (lane + d) & 31);
      Rw = fma(__ldg(f.beta + lev * kPartSeg + lane), rp, fma(__ldg(f.alpha + lev * kPartSeg + lane), rm, Rw));
    }
    ex[2][w][lane] = Rw * __ldg(f.rD + lane);
  }
  __syncthreads();
  if (!live) return;
  // 4) interiors from the spikes
  const double xe = ex[2][c][k], xl = ex[2][c][(k - 1) & 31];
  // the others in order, loads before the stores, which could alias them for
  // the compiler
  const int gap = max(mid1 - mid0, 0);
#pragma unroll 1
  for (int b = 0; b < m - gap; b += kParChunk) {
    double y_[kParChunk], old[kParChunk];
#pragma unroll
    for (int j = 0; j < kParChunk; ++j) {
      const int r = b + j < mid0 ? b + j : b + j + gap;
      y_[j] = r < m - 1 ? q[(e0 + r) * es] : 0.0;
      old[j] = in && r < m ? in[(e0 + r) * es] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kParChunk; ++j) {
      const int r = b + j < mid0 ? b + j : b + j + gap;
      if (r >= m) break;
      double v = xe;
      if (r < m - 1) {
        v = y_[j];
        if (r < F.nv) v = fma(__ldg(f.vv + r * kPartSeg + k), xl, v);
        if (r >= m - 1 - F.nw) v = fma(__ldg(f.ww + r * kPartSeg + k), xe, v);
      }
      out[(e0 + r) * es] = in ? old[j] + v : v;
    }
  }
}

// adjacent columns per block of the FP64 DFT kernels
constexpr int kParCols = 2;
int par_cols(const DevGrid &g) {
  int c = kParCols;
  while (c > 1 && (size_t)c * g.ny * sizeof(double) > 128 * 1024) c /= 2;
  return c;
}

int par_threads(const DevGrid &g, int cols) {
  const int b = cols * (g.ny / 2) / 4;
  return b <= 64 ? 64 : b >= 256 ? 256 : (b + 31) / 32 * 32;
}

// mode lines per block: enough blocks to spread over the SMs twice, and at
// least two blocks per SM where the lines' shared memory allows it
int par_lines(int nx, size_t per_line, int nh) {
  const size_t room = 2 * per_line + 256 <= kParSmemMax ? kParSmemMax / 2 - 128 : kParSmemMax - 128;
  const int by_smem = (int)std::min<size_t>(kParWarpsMax / 2, room / per_line);
  const int spread = (nh + 2 * 152 - 1) / (2 * 152);
  return std::max(0, std::min(by_smem, std::max(1, spread)));
}

// the factor block goes to shared memory along with the line when both fit
// twice per SM (lines up to itot 1024: the copy engine brings them in one
// go); longer lines read their factors from global memory a chunk ahead
bool par_staged(int nx, size_t stride) { return 2 * (16 * (size_t)nx + 8 * stride) + 256 <= kParSmemMax; }

}  // namespace

bool parallel_tri_supported(int nx, int ny) {
  return nx >= 2 * kPartSeg && nx % kPartSeg == 0 && ny >= 4 && 16 * (size_t)nx + 128 <= kParSmemMax;
}

namespace {
// the fixed-point pair: 16 <= jtot <= 8192 (at most 512 threads a block)
bool par_fixed(const DevGrid &g) { return g.ny >= 16 && g.ny <= 8192; }

constexpr size_t kParDftSmem = 160 * 1024, kFixSmem = 80 * 1024;

// values per thread, columns per block (log2) and threads of the fixed-point
// pair: jtot / 2V threads a column. One warp's instruction latency bounds the
// pair on small grids, the instruction count on large ones: 4 values per
// thread below kFix8Warps warps of 8. us per launch, forward (beside the
// temperature update) / inverse, 8 against 4 values:
//   128 x 256   19.9 / 14.3, 14.3 / 12.2    512 x 512   23.9 / 14.9, 18.2 / 12.9
//   512 x 1024  27.7 / 17.0, 26.2 / 18.2    1024 x 2048 64.8 / 43.2, 86.2 / 61.3
//   2048 x 4096 234 / 168, 341 / 257
// (the FP64 radix-8 pair: 22.4 / 19.9 at 128 x 256, 45 / 30 at 512 x 1024,
// 410 / 364 at 2048 x 4096). Columns per block 1, 2, 4: within 5% at 512 x 1024,
// 2 the best from 256 x 512 to 1024 x 2048.
// 2 values per thread (radix 2, more passes of half the work and half as many
// values to load and to write) for short columns on small grids, us per step
// with 4 against 2: 64 x 64 101 / 95, 128 x 256 119 / 111, 256 x 256 128 / 122,
// but 512 x 256 146 / 147, 128 x 512 127 / 133, 64 x 1024 144 / 163 (a column's
// threads meet at every pass).
constexpr long kFix8Warps = 1024;
constexpr long kFix2Warps = 512;  // of 4 values
constexpr int kFix2Rows = 256;
constexpr int kFixLg = 1;
struct FixShape {
  int v, lgC, threads;
  size_t smem;
};
FixShape fix_shape(const DevGrid &g) {
  FixShape f;
  f.v = (long)g.nx * (g.ny / 16) / 32 >= kFix8Warps || g.ny > 4096            ? 8
        : (long)g.nx * (g.ny / 8) / 32 < kFix2Warps && g.ny <= kFix2Rows ? 2
                                                                         : 4;
  f.lgC = kFixLg;
  const int n = g.ny / 2 / f.v;
  while (f.lgC < 4 && (n << f.lgC) < 32) f.lgC++;
  while (f.lgC > 0 && (n << f.lgC) > 512) f.lgC--;
  f.threads = std::max(32, n << f.lgC);
  f.smem = ((size_t)fx::column_stride(g.ny / 2, f.lgC) << f.lgC) * sizeof(fx::C64);
  return f;
}
}  // namespace

cudaError_t launch_par_fwd(const DevGrid &g, const StageScalars &s, const double *ux, const double *uy,
                           double2 *spec, cudaStream_t st) {
  if (par_fixed(g)) {
    const FixShape f = fix_shape(g);
    const FixArgs a{g, ux, uy, spec, nullptr, 0.0, f.lgC, g.nx / kPartSeg};
    const int blocks = (g.nx + (1 << f.lgC) - 1) >> f.lgC;
    const auto kernel = f.v == 8 ? k_par_fwd_fx<8> : f.v == 2 ? k_par_fwd_fx<2> : k_par_fwd_fx<4>;
    if (cudaError_t e = allow_smem(kernel, f.smem, kFixSmem)) return e;
    chain_launch(kernel, blocks, f.threads, f.smem, st, a);
  } else {
    const int C = par_cols(g);
    const ParArgs a{g, s, ux, uy, spec, nullptr, C, g.nx / kPartSeg};
    const size_t smem = (size_t)C * g.ny * sizeof(double);
    if (cudaError_t e = allow_smem(k_par_fwd, smem, kParDftSmem)) return e;
    chain_launch(k_par_fwd, (g.nx + C - 1) / C, par_threads(g, C), smem, st, a);
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_par_tri(const DevGrid &g, double2 *spec, const ParFactors &pf, cudaStream_t st) {
  const bool staged = par_staged(g.nx, pf.stride);
  const size_t per_line = 16 * (size_t)g.nx + (staged ? 8 * pf.stride : 0);
  // mode lines per block, two warps each
  const int lpb = par_lines(g.nx, per_line, g.nh);
  if (lpb < 1) return cudaErrorInvalidValue;
  const ParTriArgs a{spec,  pf.fac, pf.lo, pf.hi, pf.stride, g.nx, g.nh, g.nx / kPartSeg, pf.err, pf.spin_limit,
                     pf.stale};
  const size_t smem = 128 + (size_t)lpb * per_line;
  const auto kernel = staged ? k_par_tri<true> : k_par_tri<false>;
  if (cudaError_t e = allow_smem(kernel, smem, kParSmemMax)) return e;
  chain_launch(kernel, (g.nh + lpb - 1) / lpb, 64 * lpb, smem, st, a);
  count_launches(1);
  return cudaGetLastError();
}

size_t par_cn_stride(int n) { return 5 * (size_t)n + 2 * kPartLevels * kPartSeg + 3 * kPartSeg; }

namespace {
// doubles of shared memory per warp (one line)
size_t cn_warp_doubles(int n) { return (size_t)kPartSeg * ((n / kPartSeg) | 1) + 8; }
}  // namespace

bool parallel_cn_supported(int n) {
  return n >= 2 * kPartSeg && n % kPartSeg == 0 && cn_warp_doubles(n) * sizeof(double) <= kParSmemMax;
}

cudaError_t launch_par_cn(bool columns, ParCnArgs a, cudaStream_t st) {
  if (!parallel_cn_supported(a.n) || a.nf < 1 || a.nf > 3) return cudaErrorInvalidValue;
  a.m = a.n / kPartSeg;
  a.s = a.m | 1;
  if (columns) {
    const dim3 grid((a.lines + kCnCols - 1) / kCnCols, a.nf);
    chain_launch(k_par_cn_cols, grid, 32 * kCnCols, 0, st, a);
  } else {
    const size_t per = cn_warp_doubles(a.n) * sizeof(double);
    // warps (rows) per block: two blocks per SM where the rows fit
    int wpb = (int)std::min<size_t>(kCnWarpsMax, (kParSmemMax / 2) / per);
    if (wpb < 1) wpb = 1;
    const dim3 grid((a.lines + wpb - 1) / wpb, a.nf);
    if (cudaError_t e = allow_smem(k_par_cn, wpb * per, kParSmemMax)) return e;
    chain_launch(k_par_cn, grid, 32 * wpb, wpb * per, st, a);
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_par_bwd(const DevGrid &g, const StageScalars &s, const double2 *spec, double *psi,
                           cudaStream_t st) {
  if (par_fixed(g)) {
    const FixShape f = fix_shape(g);
    const FixArgs a{g,     nullptr, nullptr, const_cast<double2 *>(spec), psi, s.rgdt * (0.5 * s.rny),
                    f.lgC, g.nx / kPartSeg};
    const int blocks = (g.nx + (1 << f.lgC) - 1) >> f.lgC;
    const auto kernel = f.v == 8 ? k_par_bwd_fx<8> : f.v == 2 ? k_par_bwd_fx<2> : k_par_bwd_fx<4>;
    if (cudaError_t e = allow_smem(kernel, f.smem, kFixSmem)) return e;
    chain_launch(kernel, blocks, f.threads, f.smem, st, a);
  } else {
    const int C = par_cols(g);
    const ParArgs a{g, s, nullptr, nullptr, const_cast<double2 *>(spec), psi, C, g.nx / kPartSeg};
    const size_t smem = (size_t)C * g.ny * sizeof(double);
    if (cudaError_t e = allow_smem(k_par_bwd, smem, kParDftSmem)) return e;
    chain_launch(k_par_bwd, (g.nx + C - 1) / C, par_threads(g, C), smem, st, a);
  }
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace sns
