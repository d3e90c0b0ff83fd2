// Dense coarse-level operator and its inverse on the device (coarse_inverse.cu).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace tps {

struct CoarseOperator {
  int dim, k, n;                // degree, cells per direction
  const double *cmass, *clap;   // device: reference-cell matrices, (k+1)^2
  const double *kappa;          // device: per-cell coefficient, or null
  double scale;                 // h^(dim-2)
};

// a (ni x ni, ni interior DoFs lexicographic) = the interior operator
cudaError_t launch_assemble_coarse(double *a, const CoarseOperator &q, int ni, cudaStream_t s);
// a <- a^-1 for a symmetric positive definite a (n x n), tmp of the same size;
// *bad (device, 0 on entry) is set to 1 where a pivot is not positive
cudaError_t launch_spd_inverse(double *a, double *tmp, int n, int *bad, cudaStream_t s);

}  // namespace tps
