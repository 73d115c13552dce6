// Matrix steps outside the iteration on the tensor cores: unitary polar factors Q = X (X^H X)^{-1/2}
// of one rows x cols matrix per CTA (k_oz_polar.cu), rotations V(k)^H M(k,b) V(k+b) (k_oz_rotate.cu).
#pragma once
#include <cuda_runtime.h>

namespace w90g {

// d_status value of a matrix k_oz_polar has finished: the FP64 kernels skip it
constexpr int kPolarDone = 0x600D;
// ... and of one it has left alone: k_lowdin does not try its own iteration first
constexpr int kPolarLeft = 0x1EF7;

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
  int* status;           // [k] kPolarDone, or kPolarLeft where the iteration left the matrix alone
};

constexpr int kPolarMats = 4;
constexpr int kPolarMaxN = 128;

struct RotateArgs {
  const double2* m;      // [item] n x n blocks, item = k B + b
  int ldm;
  size_t strideM;
  const double2* v;      // [k] rows(k) x w
  int ldv;
  size_t strideV;
  const int* rows;       // [k] rows of V(k), order of M's blocks; null: w
  int w, n, B;           // n >= rows(k) and w: order of the work matrices
  const int* nnlist;     // [item] k + b
  double2* out;          // [item] w x w (may be m)
  double2* work;         // [ctas] 4 n x n
  int ctas;              // CTAs launched at most (at least 1)
  int* failed;           // set to 1 when a bounded wait ran out
};

constexpr int kRotateCtas = 304;   // two per SM: more are of no use

// n <= kPolarMaxN
cudaError_t oz_rotate_launch(const RotateArgs& a, int items, cudaStream_t s);

// K CTAs; n <= kPolarMaxN
cudaError_t oz_polar_launch(const PolarArgs& a, int K, cudaStream_t s);

}  // namespace w90g
