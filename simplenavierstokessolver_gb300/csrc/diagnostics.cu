// Device diagnostics of a Rayleigh-Benard state: the quantities the
// reference writes to its logs (src/logging.c:36-272 with the dissipation
// stencils of src/analyses.c:8-121): maximum and sum of the divergence,
// x/y momentum, kinetic (x, y) and thermal energy, and the Nusselt number
// from the wall heat flux, the energy injection, the kinetic and the thermal
// dissipation. The terms are FP64; a thread's sums of them are 128-bit
// integers, exact but for what terms below 2^-47 of the largest one hold beneath
// 2^-99 of it, then rounded to a pair of doubles, merged per block and over the
// blocks with the compensation carried along, so the result agrees with the
// reference's sequential sums to their own round-off. Fields may be FP64
// (plain path) or FP32 (batched form); FP32 values are widened exactly.
//
// FP64 issue bounds the pass (an FP64 instruction holds a sub-partition of
// GB300 for ~65-80 cycles, an integer one for 1-2), so the terms are arranged
// for few FP64 instructions per cell, 19 instead of about 590:
//  * the sums of a thread are 128-bit integers (Sum128), ~30 integer
//    instructions a term instead of the 4 FP64 additions of a compensated one;
//  * the cell size, the constants and the weights of the squared differences
//    are factors of a thread's column and multiply its sums once, at the end;
//  * the reference adds every squared difference twice, with weight 1/2 to the
//    two points it separates (weight 1 at a wall, from one side); here each
//    difference is squared once, with the full weight;
//  * divisions by spacings become products by reciprocals, except in the
//    divergence, whose maximum is the reference's bit for bit: there they
//    stay divisions unless the spacings are powers of two;
//  * the sums of a block's 64 threads are merged by 60 threads and then 10,
//    not by one thread in turn (which took 0.5 ms whatever the grid);
//  * a small grid's threads take fewer rows (diag_rows).
// sns_diagnostics, host time per call: with compensated FP64 sums (62 FP64
// instructions a cell, 16 rows per thread on every grid) against this, 64 x 128
// 110 / 42 us, 128 x 256 stretched 127 / 50, 512 x 1024 168 / 91, 1024 x 2048
// 507 / 201, 2048 x 4096 1728 / 720. The two launches, the results' way and the
// wait were ~20 us of each; with the results stored straight into pinned host
// memory and launches prepared ahead (chain.cuh) 64 x 128 takes 34, 128 x 256
// uniform 42 (52 before), 512 x 1024 82, 1024 x 2048 196. The FP64 pipe is still the busiest (65 % of its cycles at
// 512 x 1024): the merges of a thread's and a block's sums add as much as ten
// rows.
#include <cstdint>
#include <mutex>

#include "chain.cuh"
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

// A sum of doubles as a 128-bit integer in units of 2^(e - 1142): a term's 53
// bits reach from bit 67 - s up, s >= 3 its biased exponent's distance from e, so
// that 10 bits are left above for 1023 terms (a thread adds 64 at most). A term
// too close to e moves the sum down first, to an exponent 20 above its own, so
// that few threads of a warp ever do it after their first row. The unit is then
// 2^-99 of that term: terms down to 2^-47 of the largest one enter whole, smaller
// ones and the sum are cut off (towards minus infinity) at the unit. A compensated
// FP64 sum of a thread's terms holds 2^-98 of their magnitudes in the worst case.
// Infinities and NaN make the sum NaN, as the compensated sum's (inf - inf).
__device__ __forceinline__ long long shr(long long v, int s) {  // amounts of 64 and more leave the sign
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}
__device__ __forceinline__ unsigned long long shl(long long v, int s) {  // amounts of 64 and more leave 0
  unsigned long long r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}
struct Sum128 {
  static constexpr int kNan = 8192;  // e of a sum that is NaN
  static constexpr int kMargin = 20;
  static constexpr int kRoom = 3;   // least distance of e from a term's exponent
  static constexpr int kStart = 4;  // e of an empty sum (exponent 0 counts as 1)
  unsigned long long lo;
  long long hi;
  int e;
  __device__ __forceinline__ void raise(int ev) {
    const int n = ev == 0x7ff ? kNan : ev + kMargin, d = n - e;
    lo = d < 64 ? (d ? lo >> d | (unsigned long long)hi << (64 - d) : lo) : (unsigned long long)shr(hi, d - 64);
    hi = shr(hi, d);
    e = n;
  }
  template <bool NONNEG = false>
  __device__ __forceinline__ void add(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int ev = (int)(b >> 52) & 0x7ff;
    if (ev + kRoom > e) raise(ev);
    long long m = (long long)((b & 0xfffffffffffffull) | (ev ? 1ull << 52 : 0ull));
    if (!NONNEG) {
      const long long n = (long long)b >> 63;
      m = (m ^ n) - n;
    }
    const int s = e - max(ev, 1);
    const unsigned long long l = s <= 67 ? shl(m, 67 - s) : (unsigned long long)shr(m, s - 67);
    const unsigned long long t = lo + l;
    hi += shr(m, s - kRoom) + (t < l);
    lo = t;
  }
  // times f, as a pair of doubles whose sum it is to 2^-106
  __device__ __forceinline__ Neu pair(double f) const {
    if (e >= kNan) return {__longlong_as_double(0x7ff8000000000000ll), 0.0};
    const bool neg = hi < 0;
    unsigned long long h = (unsigned long long)hi, l = lo;
    if (neg) {
      l = 0ull - l;
      h = ~h + (l == 0ull);
    }
    if ((h | l) == 0ull) return {0.0, 0.0};
    const int z = h ? __clzll((long long)h) : 64 + __clzll((long long)l);
    // to the top: 53 bits for each double
    if (z >= 64) {
      h = l << (z - 64);
      l = 0ull;
    } else if (z) {
      h = h << z | l >> (64 - z);
      l <<= z;
    }
    const int k = e - 1142 + 75 - z;  // of the first double's last bit
    const unsigned long long m0 = h >> 11, m1 = (h & 0x7ff) << 42 | l >> 22;
    // m 2^q without FP64 instructions; m's top bit is bit 52 - up
    auto value = [&](unsigned long long m, int q, int up) {
      const int ex = q - up + 52 + 1023;
      const unsigned long long b = (m << up) + ((unsigned long long)(ex - 1) << 52);
      double d = __longlong_as_double((long long)(m ? b : 0ull));
      if (m && (ex < 1 || ex > 2046)) d = scalbn((double)m, q);
      return neg ? -d : d;
    };
    const int up = min(__clzll((long long)m1) - 11, 52);
    return {value(m0, k, 0) * f, value(m1, k - 53, up) * f};
  }
};

constexpr int kDiagThreads = 64;
constexpr int kDiagWarps = 608;  // one per sub-partition
constexpr int kDiagMarch = 32;   // rows per thread, at most
constexpr int kDiagParts = 6;  // threads merging one sum of a block

// One thread per column x (ux point i = x+1 and the cell behind it; the last
// column also the wall's face) and `rows` rows.
template <typename F>
__global__ void __launch_bounds__(kDiagThreads, 8) k_diag(DiagArgs<F> a, double *partials, int rows) {
  chain_begin();
  const int nx = a.nx, ny = a.ny;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y0 = blockIdx.y * rows, y1 = min(y0 + rows, ny);
  Neu acc[kDiagSums];
#pragma unroll
  for (int k = 0; k < kDiagSums; ++k) acc[k] = {0.0, 0.0};
  unsigned long long divmax = 0ull;
  if (x < nx) {
    const double dy = a.dy, q = a.sqrt_pr_ra;
    const bool first = x == 0, last = x == nx - 1;
    auto LD = [](const F *hi, const float *lo, size_t k) -> double {
      return lo ? (double)hi[k] + (double)lo[k] : (double)hi[k];
    };
    // ux at i = x+1 (zero at the walls i = 1 and nx+1), uy and T of the cell
    const double dxc = a.dxc[x], dxf = a.dxf[x], dxw = a.dxc[nx];
    const double rdy = 1.0 / dy, rdxf = 1.0 / dxf;
    const bool p2 = pow2(dy) && pow2(dxf);  // products by the reciprocals are the divisions
    const double wall = last ? dxc / dxw : 0.0;  // the wall face's weight to the column's west face's
    Sum128 su{0, 0, Sum128::kStart}, suu = su, inj = su, div = su, sv = su, svv = su, stt = su, flux = su;
    Sum128 ux2 = su, uy2 = su, vx2 = su, vy2 = su, tx2 = su, ty2 = su;
    size_t r = (size_t)y0 * nx + x;
    double u = first ? 0.0 : LD(a.ux, a.uxl, r), v = LD(a.uy, a.uyl, r), t = LD(a.t, a.tl, r);
#pragma unroll 1
    for (int y = y0; y < y1; ++y) {
      const size_t rn = (y + 1 == ny ? 0 : (size_t)(y + 1) * nx) + x;
      const double un = first ? 0.0 : LD(a.ux, a.uxl, rn), vn = LD(a.uy, a.uyl, rn), tn = LD(a.t, a.tl, rn);
      const double ur = last ? 0.0 : LD(a.ux, a.uxl, r + 1);
      const double vl = first ? 0.0 : LD(a.uy, a.uyl, r - 1), tl = first ? 0.5 : LD(a.t, a.tl, r - 1);
      const double dux = ur - u, dvy = vn - v, duy = un - u, dvx = v - vl, dtx = t - tl, dty = tn - t;
      // ux point i (src/logging.c:95-100, 139-144, 208-214)
      su.add(u);
      suu.add<true>(u * u);
      inj.add(u * (tl + t));
      // cell centre i (src/logging.c:51-57 and its momentum and energies)
      const double dv = p2 ? dux * rdxf + dvy * rdy : dux / dxf + dvy / dy;
      divmax = max(divmax, div_key(dv));
      div.add(dv);
      sv.add(v);
      svv.add<true>(v * v);
      stt.add<true>(t * t);
      // dissipations (src/analyses.c:8-33, 35-72 and 74-110)
      ux2.add<true>(dux * dux);
      uy2.add<true>(duy * duy);
      vx2.add<true>(dvx * dvx);
      vy2.add<true>(dvy * dvy);
      tx2.add<true>(dtx * dtx);
      ty2.add<true>(dty * dty);
      // wall heat flux (src/logging.c:195-199)
      if (first) flux.add(dtx);
      if (last) {
        const double dtw = -0.5 - t;
        vx2.add<true>(v * v * wall);
        tx2.add<true>(dtw * dtw * wall);
        flux.add(first ? dtw * wall : dtw);
      }
      r = rn;
      u = un;
      v = vn;
      t = tn;
    }
    // the column's factors
    const double cs_u = dxc * dy, cs_c = dxf * dy, wfx = dy / dxc, wcy = dxf * rdy, e = q * a.nu, h = q * a.kappa;
    acc[0] = su.pair(cs_u);
    acc[1] = sv.pair(cs_c);
    acc[2] = suu.pair(0.5 * cs_u);
    acc[3] = svv.pair(0.5 * cs_c);
    acc[4] = stt.pair(0.5 * cs_c);
    acc[5] = inj.pair(0.5 * q * cs_u);
    acc[6] = ux2.pair(dy * rdxf * e);
    const Neu a1 = uy2.pair(first ? 0.0 : dxc * rdy * e), a2 = vx2.pair(wfx * e), a3 = vy2.pair(wcy * e);
    acc[6].merge(a1.s, a1.c);
    acc[6].merge(a2.s, a2.c);
    acc[6].merge(a3.s, a3.c);
    acc[7] = div.pair(1.0);
    acc[8] = tx2.pair(wfx * h);
    const Neu b1 = ty2.pair(wcy * h);
    acc[8].merge(b1.s, b1.c);
    if (first | last) acc[9] = flux.pair(-(0.5 * dy) / (first ? dxc : dxw));
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
  chain_begin();
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

namespace {
// Rows per thread: a power of two that leaves one warp per sub-partition, since
// one keeps the FP64 pipe busy and every thread ends with merges worth ten rows
// or more (two per sub-partition: 400 x 512 70 against 66 us per call); at most
// kDiagMarch (16 / 32 / 64 rows: 1024 x 2048 246 / 201 / 215, 2048 x 4096 796 /
// 727 / 699).
int diag_rows(int nx, int ny) {
  const long warps1 = (long)((nx + 31) / 32) * ny;
  int rows = 1;
  while (rows < kDiagMarch && warps1 / (2 * rows) >= kDiagWarps) rows *= 2;
  return rows;
}
dim3 diag_grid(int nx, int ny) {
  const int rows = diag_rows(nx, ny);
  return dim3((nx + kDiagThreads - 1) / kDiagThreads, (ny + rows - 1) / rows);
}
}  // namespace

int diag_blocks(int nx, int ny) {
  return ((nx + 1 + kDiagThreads - 1) / kDiagThreads) * ((ny + kDiagRows - 1) / kDiagRows);
}

size_t diag_words(int nx, int ny) {
  const dim3 g = diag_grid(nx, ny);
  return (size_t)g.x * g.y * (2 * kDiagSums + 1) + kDiagOut;
}

template <typename F>
cudaError_t launch_diag(const DiagArgs<F> &a, double *scratch, double **out, cudaStream_t st, double *host) {
  const dim3 grid = diag_grid(a.nx, a.ny);
  *out = host ? host : scratch;
  chain_launch(k_diag<F>, grid, kDiagThreads, 0, st, a, scratch + kDiagOut, diag_rows(a.nx, a.ny));
  chain_launch(k_diag_finish, kDiagSums + 1, kFinishThreads, 0, st, scratch + kDiagOut, (int)(grid.x * grid.y), a.ly,
               *out);
  return cudaGetLastError();
}

template cudaError_t launch_diag<double>(const DiagArgs<double> &, double *, double **, cudaStream_t, double *);
template cudaError_t launch_diag<float>(const DiagArgs<float> &, double *, double **, cudaStream_t, double *);

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
