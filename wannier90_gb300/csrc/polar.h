// Unitary polar factors on the tensor cores (k_oz_polar.cu): Q = X (X^H X)^{-1/2} of one
// rows x cols matrix per CTA.
#pragma once
#include <cuda_runtime.h>

namespace w90g {

// d_status value of a matrix k_oz_polar has finished: the FP64 kernels skip it
constexpr int kPolarDone = 0x600D;

struct PolarArgs {
  const double2* x;      // [k] rows(k) x cols, column-major
  int ldx;
  size_t strideX;        // elements between consecutive k
  double2* q;            // [k] result (may be x)
  int ldq;
  size_t strideQ;
  int qrows;             // rows of q to write; those past rows(k) become zero
  const int* rows;       // [k] rows of X(k); null: cols
  const int* row0;       // [k] first row of X(k) in x; null: 0
  int cols;
  int n;                 // order of the square work matrices, >= rows(k) and cols
  double2* work;         // [k] kPolarMats n x n
  size_t strideW;
  int* status;           // [k] kPolarDone, or 0 where the iteration left the matrix alone
};

constexpr int kPolarMats = 4;
constexpr int kPolarMaxN = 128;

// K CTAs; n <= kPolarMaxN
cudaError_t oz_polar_launch(const PolarArgs& a, int K, cudaStream_t s);

}  // namespace w90g
