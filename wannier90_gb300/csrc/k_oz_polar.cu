// Unitary polar factor Q = X (X^H X)^{-1/2} of one matrix per CTA, by the Newton-Schulz
// iteration X <- X (3 I - X^H X) / 2 with its products on the tensor cores (oz_mm.cuh).
//
// The FP64 form (X^H X, Jacobi eigenpairs, X V L^{-1/2} V^H) costs 150 to 250 W^3 FMA on a pipe
// of 2 lanes per SM: 15.9 ms for 1000 matrices of W = 32.  The iteration is two products per
// step -- a Gram matrix, Hermitian, and an update -- and doubles its digits per step once the
// singular values are near 1; below that they grow by 1.5 per step.  A product of all 1000
// matrices takes about 45 us here.  Working on X itself, its error is that of the
// products times the condition number of X, where the eigenpairs of X^H X carry the square.
//
// Singular values start in (0, 1] (the first step's coefficients carry the scale, an upper
// bound on ||X|| from the Gram matrix, so no element of X is rounded for it).  A matrix whose
// smallest one has not reached 1 after kPolarSteps steps -- a condition number above ~1e5, or
// a rank-deficient X -- is left alone with status kPolarLeft: the FP64 kernel that runs next takes it,
// with its own verdict.  That kernel also takes everything else this one cannot finish
// (a bounded wait that ran out, NaN, infinities and scales outside what the digits carry).
#include "oz_mm.cuh"
#include "polar.h"

namespace w90g {

namespace {

constexpr int kPolarSteps = 40;

template <int WP>
struct PolarSmem {
  using E = ExpProd<WP, false>;
  static constexpr size_t BYTES = E::BYTES;
};

}  // namespace

template <int WP>
__global__ void __launch_bounds__(256, 2) k_oz_polar(PolarArgs g) {
  using E = ExpProd<WP, false>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_rowexp[WP], s_colexp[WP];
  __shared__ unsigned s_key[4][2][WP];
  __shared__ int s_bad;
  __shared__ float s_wred[8];
  __shared__ int s_res;

  const int k = blockIdx.x, tid = threadIdx.x, warp = tid >> 5;
  const int N = g.n, NN = N * N, cols = g.cols;
  const int rows = g.rows ? g.rows[k] : cols;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_slot)), "r"((uint32_t)E::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_bad = 0;
  }
  double2* mats = E::MATS_IN_SMEM ? (double2*)(base + E::REGION) : g.work + (size_t)k * g.strideW;
  double2 *X = mats, *XH = mats + NN, *Y = mats + 2 * NN, *Z = mats + 3 * NN;
  Rec rX{s_key[0][0], s_key[0][1]}, rZ{s_key[1][0], s_key[1][1]}, rY{s_key[2][0], s_key[2][0]};
  rec_clear(rX, WP);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // X as an N x N matrix, zero outside rows x cols (zero rows and columns stay zero)
  const double2* Xg = g.x + (size_t)k * g.strideX + (g.row0 ? g.row0[k] : 0);
  for (int e = tid; e < NN; e += 256) {
    const int i = e % N, j = e / N;
    const double2 v = (i < rows && j < cols) ? Xg[(size_t)j * g.ldx + i] : cmk(0.0, 0.0);
    X[e] = v;
    rec_add(rX, i, j, v);
  }
  __syncthreads();
  OzCtx cx{base, base + E::SB_OFFSET, tmem_slot, smem_u32(&mbar), 0u, s_rowexp, s_colexp, &s_bad};
  const NoAdd none;
  bool ok = !__syncthreads_or(keys_wild(rX.row, N)), done = false;
  for (int step = 0; step < kPolarSteps && ok && !done; ++step) {
    for (int e = tid; e < NN; e += 256) XH[e] = cconj(X[(size_t)(e % N) * N + e / N]);
    __syncthreads();
    // (the largest entry of row i of X^H is that of column i of X)
    ok = E::mm(cx, Y, XH, rX.col, X, rX.col, N, Epi{Y, 1, rY}, none);
    if (!ok) break;
    double ca = 1.5, cb = -0.5;
    if (step == 0) {
      // ||X||_2^2 <= ||Y||_1, from FP32 moduli; 2^-10 above their sum's error, so that the
      // scaled singular values stay below 1
      float cmax = 0.0f;
      for (int j = tid; j < N; j += 256) {
        float a = 0.0f;
        for (int i = 0; i < N; ++i) {
          const double2 y = Y[(size_t)j * N + i];
          const float yr = (float)y.x, yi = (float)y.y;
          a += sqrtf(yr * yr + yi * yi);
        }
        cmax = a > cmax || !(a == a) ? a : cmax;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float b = __shfl_xor_sync(0xffffffffu, cmax, o);
        cmax = b > cmax || !(b == b) ? b : cmax;
      }
      if ((tid & 31) == 0) s_wred[warp] = cmax;
      __syncthreads();
      float nrm = 0.0f;
      for (int w = 0; w < 8; ++w) nrm = s_wred[w] > nrm || !(s_wred[w] == s_wred[w]) ? s_wred[w] : nrm;
      if (!(nrm > 1e-30f && nrm < 1e30f)) break;   // (uniform) zero, extreme or non-finite
      const double s2 = (double)nrm * (1.0 + 0x1p-10);
      // already near unitary: no scaling (3 - s^2 > 0 for every singular value below sqrt 3)
      const double r = s2 < 1.5 ? 1.0 : 1.0 / sqrt(s2);
      ca = 1.5 * r;
      cb = -0.5 * r * r * r;
    }
    // Z = ca I + cb Y on the cols x cols block, and how far Y is from I there
    rec_clear(rZ, WP);
    if (tid == 0) s_res = 0;
    __syncthreads();
    int far = 0;
    for (int e = tid; e < NN; e += 256) {
      const int i = e % N, j = e / N;
      const double2 y = Y[e];
      const bool dg = i == j && j < cols;
      const double2 z = cmk(dg ? fma(cb, y.x, ca) : cb * y.x, cb * y.y);
      // |Y - I| against 1e-8 / N elementwise: its norm is then below 1e-8 and the update's
      // error below 1e-16
      const float dr = (float)(dg ? y.x - 1.0 : y.x), di = (float)y.y;
      if (!(fabsf(dr) + fabsf(di) < 1.0e-8f / (float)N)) far = 1;
      Z[e] = z;
      rec_add(rZ, i, j, z);
    }
    if (far) s_res = 1;
    __syncthreads();
    done = s_res == 0 && ca == 1.5;
    // X <- X Z (through Y, whose storage is free; X's digits are read before Y is written)
    ok = E::mm(cx, Y, X, rX.row, Z, rZ.col, N, Epi{Y, 0, rX}, none);
    double2* t = X;
    X = Y;
    Y = t;
  }
  const bool good = ok && done;
  if (good) {
    double2* Q = g.q + (size_t)k * g.strideQ;
    for (int e = tid; e < g.qrows * cols; e += 256) {
      const int i = e % g.qrows, j = e / g.qrows;
      Q[(size_t)j * g.ldq + i] = i < rows ? X[(size_t)j * N + i] : cmk(0.0, 0.0);
    }
  }
  if (tid == 0) g.status[k] = good ? kPolarDone : kPolarLeft;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(cx.tmem), "r"((uint32_t)E::TMEM_COLS) : "memory");
  }
}

template <int WP>
static cudaError_t polar_wp(const PolarArgs& a, int K, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(k_oz_polar<WP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PolarSmem<WP>::BYTES);
  if (e != cudaSuccess) return e;
  k_oz_polar<WP><<<K, 256, PolarSmem<WP>::BYTES, s>>>(a);
  return cudaGetLastError();
}

cudaError_t oz_polar_launch(const PolarArgs& a, int K, cudaStream_t s) {
  if (a.n <= 16) return polar_wp<16>(a, K, s);
  if (a.n <= 32) return polar_wp<32>(a, K, s);
  if (a.n <= 64) return polar_wp<64>(a, K, s);
  if (a.n <= kPolarMaxN) return polar_wp<128>(a, K, s);
  return cudaErrorInvalidValue;
}

}  // namespace w90g
