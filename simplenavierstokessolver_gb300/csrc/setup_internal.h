// Set-up kernels (setup.cu): arguments and launches.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace sns {

// the Poisson lines of every mode (src/fluid/compute_potential.c:109-127): sub-
// and super-diagonal in the factors' row order, with zeros at the line's ends,
// whose raw couplings l_first and u_last the diagonal's ends absorb (diagonal
// -l - u + eigenvalue, Neumann closure); the modes' eigenvalues
struct PoissonLines {
  int n, nh;
  const double *lo, *hi, *eig;
  double l_first, u_last;
  double *out;       // nh blocks: inv [g = lo inv] up v w alpha beta rD
  size_t stride;     // doubles per block
  bool interleave;   // row k m + r at r kPartSeg + k
  bool with_g;
};
cudaError_t launch_partition_factors(const PoissonLines &p, cudaStream_t st);
// xc: cell centres (device), xm, xp: wall temperatures; hi + lo: the field
cudaError_t launch_seeded_temperature(int nx, int ny, unsigned long long seed, const double *xc, double xm, double xp,
                                      float *hi, float *lo, cudaStream_t st);
// doubles to pairs of floats
cudaError_t launch_split(size_t n, const double *in, float *hi, float *lo, cudaStream_t st);

}  // namespace sns
