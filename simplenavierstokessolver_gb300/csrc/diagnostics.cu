// Device diagnostics of a Rayleigh-Benard state: the quantities the
// reference writes to its logs (src/logging.c:36-272 with the dissipation
// stencils of src/analyses.c:8-121): maximum and sum of the divergence,
// x/y momentum, kinetic (x, y) and thermal energy, and the Nusselt number
// from the wall heat flux, the energy injection, the kinetic and the thermal
// dissipation. All arithmetic is FP64; every sum is accumulated with
// Neumaier's compensated summation per thread, merged per block and over the
// blocks with the compensation carried along, so the result agrees with the
// reference's sequential sums to their own round-off. Fields may be FP64
// (plain path) or FP32 (batched form); FP32 values are widened exactly.
//
// FP64 issue bounds the pass (an FP64 instruction holds a sub-partition of
// GB300 for ~70-80 cycles, an integer one for 1-2), so the terms are arranged
// for few FP64 instructions per cell, about 62 instead of about 590:
//  * the cell size and the constants are factors of a thread's column and
//    multiply its sums once, at the end;
//  * the reference adds every squared difference twice, with weight 1/2 to the
//    two points it separates (weight 1 at a wall, from one side); here each
//    difference is squared once, with the full weight;
//  * divisions by spacings become products by reciprocals, except in the
//    divergence, whose maximum is the reference's bit for bit: there they
//    stay divisions unless the spacings are powers of two;
//  * compensation tests compare the operands' bits with integer instructions;
//  * the sums of a block's 64 threads are merged by 60 threads and then 10,
//    not by one thread in turn (which took 0.5 ms whatever the grid).
// sns_diagnostics, host time per call: 128 x 256 547 -> 117 us, 512 x 1024
// 745 -> 167 us, 1024 x 2048 2690 -> 505 us. What is left at 512 x 1024 is
// the FP64 issue of the 62 instructions (~137 us).
#include <cstdint>
#include <mutex>

#include "diag_internal.h"

namespace sns {
namespace {

struct Neu {
  double s, c;
  __device__ __forceinline__ void add(double v) {
    const double t = s + v;
    // |s| >= |v|, on the bits (an FP64 comparison would cost as much as an addition)
    const bool ge = ((unsigned long long)__double_as_longlong(s) & 0x7fffffffffffffffull) >=
                    ((unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull);
    const double big = ge ? s : v, small = ge ? v : s;
    c += (big - t) + small;
    s = t;
  }
  __device__ __forceinline__ void merge(double os, double oc) {
    add(os);
    c += oc;
  }
};

// |v| as an order-preserving key; NaN counts as 0, as fmax ignores it
__device__ __forceinline__ unsigned long long div_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
  return b > 0x7ff0000000000000ull ? 0ull : b;
}

__device__ __forceinline__ bool pow2(double d) {
  return __double2loint(d) == 0 && (__double2hiint(d) & 0xfffff) == 0;
}

constexpr int kDiagThreads = 64;
constexpr int kDiagParts = 6;  // threads merging one sum of a block

// One thread per ux point (column x, i = x+1 in [1, nx+1]) and kDiagRows rows.
template <typename F>
__global__ void __launch_bounds__(kDiagThreads) k_diag(DiagArgs<F> a, double *partials) {
  const int nx = a.nx, ny = a.ny;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y0 = blockIdx.y * kDiagRows, y1 = min(y0 + kDiagRows, ny);
  Neu acc[kDiagSums];
#pragma unroll
  for (int k = 0; k < kDiagSums; ++k) acc[k] = {0.0, 0.0};
  unsigned long long divmax = 0ull;
  if (x <= nx) {
    const double dy = a.dy, q = a.sqrt_pr_ra;
    const bool cell = x < nx, inner = x > 0 && cell;  // cell centre i = x+1 <= nx; ux point off the walls
    auto LD = [](const F *hi, const float *lo, size_t k) -> double {
      return lo ? (double)hi[k] + (double)lo[k] : (double)hi[k];
    };
    auto UX = [&](int xi, int y) -> double {  // ux at i = xi+1; walls i = 1 and nx+1 are zero
      return (xi <= 0 || xi >= nx) ? 0.0 : LD(a.ux, a.uxl, (size_t)y * nx + xi);
    };
    auto UY = [&](int xi, int y) -> double {  // uy at i = xi+1, zero at i = 0 and nx+1
      return (xi < 0 || xi >= nx) ? 0.0 : LD(a.uy, a.uyl, (size_t)y * nx + xi);
    };
    auto TT = [&](int xi, int y) -> double {
      return xi < 0 ? 0.5 : xi >= nx ? -0.5 : LD(a.t, a.tl, (size_t)y * nx + xi);
    };
    const double dxc = a.dxc[x];               // DXC(i), i = x+1 <= nx+1
    const double dxf = cell ? a.dxf[x] : 1.0;  // DXF(i)
    const double rdy = 1.0 / dy, rdxf = 1.0 / dxf;
    const bool p2 = pow2(dy) && pow2(dxf);  // products by the reciprocals are the divisions
    // weights of the squared differences: along x across a cell (ux) and across
    // a face (uy, T), along y at a ux point and at a cell
    const double wcx = cell ? dy * rdxf : 0.0, wfx = dy / dxc;
    const double wuy = inner ? dxc * rdy : 0.0, wcy = cell ? dxf * rdy : 0.0;
    double u = UX(x, y0), v = UY(x, y0), t = TT(x, y0);
    for (int y = y0; y < y1; ++y) {
      const int yp = y + 1 == ny ? 0 : y + 1;
      const double un = UX(x, yp), vn = UY(x, yp), tn = TT(x, yp);
      const double ur = UX(x + 1, y), vl = UY(x - 1, y), tl = TT(x - 1, y);
      const double dux = ur - u, dvy = vn - v, duy = un - u, dvx = v - vl, dtx = t - tl, dty = tn - t;
      // ux point i (src/logging.c:95-100, 139-144, 208-214)
      acc[0].add(u);
      acc[2].add(u * u);
      acc[5].add(u * (tl + t));
      // cell centre i (src/logging.c:51-57 and its momentum and energies)
      if (cell) {
        const double div = p2 ? dux * rdxf + dvy * rdy : dux / dxf + dvy / dy;
        divmax = max(divmax, div_key(div));
        acc[7].add(div);
        acc[1].add(v);
        acc[3].add(v * v);
        acc[4].add(t * t);
      }
      // dissipations (src/analyses.c:8-33, 35-72 and 74-110)
      acc[6].add(((wcx * dux) * dux + (wuy * duy) * duy) + ((wfx * dvx) * dvx + (wcy * dvy) * dvy));
      acc[8].add((wfx * dtx) * dtx + (wcy * dty) * dty);
      if (x == 0) {  // wall heat flux (src/logging.c:195-199)
        const double g0 = (t - tl) / a.dxc[0];
        const double g1 = (TT(nx, y) - TT(nx - 1, y)) / a.dxc[nx];
        acc[9].add(-(0.5 * (g0 + g1) * dy));
      }
      u = un;
      v = vn;
      t = tn;
    }
    // the column's factors
    auto scale = [&](int k, double f) {
      acc[k].s *= f;
      acc[k].c *= f;
    };
    const double cs_u = dxc * dy, cs_c = cell ? dxf * dy : 0.0;
    scale(0, cs_u);
    scale(1, cs_c);
    scale(2, 0.5 * cs_u);
    scale(3, 0.5 * cs_c);
    scale(4, 0.5 * cs_c);
    scale(5, 0.5 * q * cs_u);
    scale(6, q * a.nu);
    scale(8, q * a.kappa);
  }
  // block merge: kDiagParts threads per sum, then one
  __shared__ double sh[2][kDiagSums][kDiagThreads + 1];
  __shared__ double sh2[2][kDiagSums][kDiagParts];
  __shared__ unsigned long long shmax[kDiagThreads];
  double *out = partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (2 * kDiagSums + 1);
#pragma unroll
  for (int k = 0; k < kDiagSums; ++k) {
    sh[0][k][threadIdx.x] = acc[k].s;
    sh[1][k][threadIdx.x] = acc[k].c;
  }
  shmax[threadIdx.x] = divmax;
  __syncthreads();
  if (threadIdx.x < kDiagSums * kDiagParts) {
    const int k = threadIdx.x / kDiagParts, p = threadIdx.x % kDiagParts;
    Neu m{0.0, 0.0};
    for (int t = p; t < kDiagThreads; t += kDiagParts) m.merge(sh[0][k][t], sh[1][k][t]);
    sh2[0][k][p] = m.s;
    sh2[1][k][p] = m.c;
  } else if (threadIdx.x == kDiagThreads - 1) {
    unsigned long long m = 0ull;
    for (int t = 0; t < kDiagThreads; ++t) m = max(m, shmax[t]);
    out[2 * kDiagSums] = __longlong_as_double((long long)m);
  }
  __syncthreads();
  if (threadIdx.x < kDiagSums) {
    const int k = threadIdx.x;
    Neu m{0.0, 0.0};
    for (int p = 0; p < kDiagParts; ++p) m.merge(sh2[0][k][p], sh2[1][k][p]);
    out[2 * k] = m.s;
    out[2 * k + 1] = m.c;
  }
}

// Sums over the blocks, one block of threads per sum (the last one: the
// maximum): a strided pass per thread, then a tree over shared memory; each
// of the 11 log values depends on one sum and is written by its block.
constexpr int kFinishThreads = 256;

__global__ void __launch_bounds__(kFinishThreads) k_diag_finish(const double *partials, int nblocks, double ly,
                                                               double *out) {
  __shared__ double ss[kFinishThreads], sc[kFinishThreads];
  const int k = blockIdx.x, t = threadIdx.x;
  const size_t stride = 2 * kDiagSums + 1;
  if (k == kDiagSums) {
    unsigned long long m = 0ull;
    for (int b = t; b < nblocks; b += kFinishThreads)
      m = max(m, (unsigned long long)__double_as_longlong(partials[b * stride + 2 * kDiagSums]));
    ss[t] = __longlong_as_double((long long)m);
    __syncthreads();
    for (int w = kFinishThreads / 2; w > 0; w >>= 1) {
      if (t < w)
        ss[t] = __longlong_as_double((long long)max((unsigned long long)__double_as_longlong(ss[t]),
                                                    (unsigned long long)__double_as_longlong(ss[t + w])));
      __syncthreads();
    }
    if (t == 0) out[0] = ss[0];
    return;
  }
  Neu m{0.0, 0.0};
  for (int b = t; b < nblocks; b += kFinishThreads) m.merge(partials[b * stride + 2 * k], partials[b * stride + 2 * k + 1]);
  ss[t] = m.s;
  sc[t] = m.c;
  __syncthreads();
  for (int w = kFinishThreads / 2; w > 0; w >>= 1) {
    if (t < w) {
      m.merge(ss[t + w], sc[t + w]);
      ss[t] = m.s;
      sc[t] = m.c;
    }
    __syncthreads();
  }
  if (t == 0) {
    const double r = m.s + m.c, lx = 1.0;
    switch (k) {
      case 0: out[2] = r; break;
      case 1: out[3] = r; break;
      case 2: out[4] = r; break;
      case 3: out[5] = r; break;
      case 4: out[6] = r; break;
      case 5: out[8] = r / (lx * ly) + 1.; break;
      case 6: out[9] = r / (lx * ly) + 1.; break;
      case 7: out[1] = r; break;
      case 8: out[10] = r / (lx * ly); break;
      default: out[7] = r / ly; break;
    }
  }
}

}  // namespace

int diag_blocks(int nx, int ny) {
  return ((nx + 1 + kDiagThreads - 1) / kDiagThreads) * ((ny + kDiagRows - 1) / kDiagRows);
}

size_t diag_words(int nx, int ny) { return (size_t)diag_blocks(nx, ny) * (2 * kDiagSums + 1) + kDiagOut; }

template <typename F>
cudaError_t launch_diag(const DiagArgs<F> &a, double *scratch, double **out, cudaStream_t st) {
  const dim3 grid((a.nx + 1 + kDiagThreads - 1) / kDiagThreads, (a.ny + kDiagRows - 1) / kDiagRows);
  k_diag<F><<<grid, kDiagThreads, 0, st>>>(a, scratch + kDiagOut);
  k_diag_finish<<<kDiagSums + 1, kFinishThreads, 0, st>>>(scratch + kDiagOut, (int)(grid.x * grid.y), a.ly, scratch);
  *out = scratch;
  return cudaGetLastError();
}

template cudaError_t launch_diag<double>(const DiagArgs<double> &, double *, double **, cudaStream_t);
template cudaError_t launch_diag<float>(const DiagArgs<float> &, double *, double **, cudaStream_t);

// ---------------------------------------------------------------------------
// Allocation-free variant (sns_diagnostics_static in sns_api.cpp).
//
// Some callers cannot allocate: a monitoring thread that samples a run while
// its kernels are in flight (cudaMalloc and cudaFree may synchronise the
// device and stall the solver's stream, and the first call of the allocating
// entry point makes a cudaMalloc), and a process whose device memory is
// committed to a batch arena sized to the whole HBM (an allocation there
// fails with out-of-memory). For them the block partials live in one
// file-scope device array of fixed size and the 11 results are copied
// straight into the caller's array: no device or host memory is allocated.
//
// Scratch layout: the 11 results (kDiagOut words), then kDiagStaticBlocks
// block partials of 2*kDiagSums+1 words. Nothing in it needs to start at zero:
// k_diag writes every partial word of every block it launches and
// k_diag_finish reads only those, then writes all 11 results. There is one
// scratch per device, so two calls that overlap on one device (other host
// threads, other cases) race on it and may return each other's or mixed
// results: serialise them.
namespace {

constexpr size_t kDiagStaticWords = kDiagOut + (size_t)kDiagStaticBlocks * (2 * kDiagSums + 1);
static __device__ __align__(256) double g_diag_scratch[kDiagStaticWords];

// The scratch's device address, looked up on every call with the caller's
// device current: an address kept from an earlier call could belong to a
// context that no longer exists (after cudaDeviceReset the module is loaded
// again, possibly elsewhere). The lookup is cheap once the module is loaded;
// the first call on a device may load it, so make that call before any
// stream capture.
cudaError_t scratch_for_current_device(double **ptr) {
  void *p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_diag_scratch);
  if (e != cudaSuccess) return e;
  *ptr = static_cast<double *>(p);
  return cudaSuccess;
}

}  // namespace

cudaError_t diag_static(const DiagArgs<double> &a, cudaStream_t st, double out[11]) {
  if (diag_blocks(a.nx, a.ny) > kDiagStaticBlocks) return cudaErrorInvalidValue;
  double *scratch = nullptr, *res = nullptr;
  cudaError_t e = scratch_for_current_device(&scratch);
  if (e != cudaSuccess) return e;
  if ((e = launch_diag(a, scratch, &res, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(out, res, 11 * sizeof(double), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  return cudaStreamSynchronize(st);
}

}  // namespace sns
