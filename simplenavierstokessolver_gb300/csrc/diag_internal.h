// Device diagnostics (diagnostics.cu): arguments and launch helpers.
#pragma once

#include <cmath>
#include <cstddef>

#include <cuda_runtime.h>

namespace sns {

constexpr int kDiagSums = 10;  // compensated sums per block
// rows of a block as diag_blocks counts them, which is what the static form
// accepts grids by (launches take 1 to 32)
constexpr int kDiagRows = 16;

// dense fields (x fastest, no halos), metrics as DXF(i) = dxf[i-1], DXC(i) = dxc[i-1]
template <typename F>
struct DiagArgs {
  int nx, ny;
  double dy, ly;
  double sqrt_pr_ra;  // sqrt(Pr)*sqrt(Ra)
  double nu;          // sqrt(Pr)/sqrt(Ra)
  double kappa;       // 1./sqrt(Pr)/sqrt(Ra)
  const double *dxf, *dxc;
  const F *ux, *uy, *t;
  // low words of compensated FP32 storage (value = hi + lo), or nullptr
  const float *uxl = nullptr, *uyl = nullptr, *tl = nullptr;
};

constexpr int kDiagOut = 16;  // words kept for the 11 results at the head of the scratch
// words of device scratch for a grid
size_t diag_words(int nx, int ny);
// the block sums and their final sum; *out: the 11 results, in host (pinned, if
// given) or at the head of the device's scratch:
// divergence max, sum; x, y momentum; kinetic x, y and thermal energy;
// Nu from wall flux, injection, kinetic dissipation, thermal dissipation.
// Two launches.
template <typename F>
cudaError_t launch_diag(const DiagArgs<F> &a, double *scratch, double **out, cudaStream_t st, double *host = nullptr);

// allocation-free form: block partials in a fixed file-scope device array of
// kDiagStaticBlocks blocks (672 KiB), the final sum on the device; grids with
// more blocks (diag_blocks: of kDiagRows rows and 64 ux points) are rejected.
// Launches have no more blocks than that, or 1217. Blocks until done.
constexpr int kDiagStaticBlocks = 4096;
int diag_blocks(int nx, int ny);
cudaError_t diag_static(const DiagArgs<double> &a, cudaStream_t st, double out[11]);

}  // namespace sns
