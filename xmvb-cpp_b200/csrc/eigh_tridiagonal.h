// Tridiagonal form of the dense generalized eigensolver (eigh_tridiagonal.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace vbcore {

constexpr int kTridiagonalMin = 33;   // below: one warp of Jacobi rotations in shared memory
constexpr int kTridiagonalMax = 160;  // five columns per lane of the reduction

size_t tridiagonal_workspace_doubles(int n);

// All roots (ascending) and S-normalized vectors of H C = S C E from H (upper triangle read) and
// Ui = U^-1 of S = U^T U (upper).  Synchronizes the stream; *status != 0: not settled, solve otherwise.
cudaError_t tridiagonal_eigh(const double* H, const double* Ui, int n, double* values, double* vectors, double* work,
                             int* status, cudaStream_t s);

}  // namespace vbcore
