// Rotations outside the iteration on the tensor cores (oz_mm.cuh, 56-bit operands):
//   k_oz_rotate  M0(k,b) = V(k)^H M(k,b) V(k+b) -- the projection of an isolated group
//                (src/overlap.F90:909-923, V = U) and the last step of the disentanglement
//                (src/disentangle.F90:220-235, :286-370, V = U_opt U);
//   k_oz_ufinal  U = U0 R at the end of a tensor-path solve.
// In FP64 these are bound by the FP64 pipe (8000 blocks of num_wann 32: 3.6 ms, 4096 of 42 states to
// 32: 2.9 ms, U0 R of 512 x 128: 8.3 ms).  The products here are as accurate as FP64 ones; what
// bounds them is the chain of slicing, MMAs and recombining, two CTAs per SM hiding some of each other's
// latency (8000 blocks of 32: 0.79 ms, ALU 39 %, issue 40 %, tensor pipe 12 %).
// Operands whose scales the digits do not carry (exp_wild: NaN, infinities, magnitudes beyond 2^+-290)
// are multiplied in FP64 here, block by block, so that they come out as FP64 gives them.
#include <algorithm>

#include "oz_mm.cuh"
#include "polar.h"

namespace w90g {

namespace {

// tensor memory, barrier and product context of a CTA
struct RotShared {
  uint64_t mbar;
  uint32_t tmem;
  int bad;
};

template <class E>
__device__ __forceinline__ void rot_begin(RotShared& sh) {
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&sh.tmem)), "r"((uint32_t)E::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&sh.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sh.bad = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

template <class E>
__device__ __forceinline__ void rot_end(RotShared& sh) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(sh.tmem), "r"((uint32_t)E::TMEM_COLS) : "memory");
}

// C (m x n, ldc) = A B in FP64, inner dimension kk
__device__ __forceinline__ void rot_fp64(double2* C, int ldc, const double2* A, int lda, const double2* B, int ldb,
                                         int m, int n, int kk) {
  for (int e = threadIdx.x; e < m * n; e += blockDim.x) {
    const int i = e % m, j = e / m;
    double2 acc = cmk(0.0, 0.0);
    for (int l = 0; l < kk; ++l) cfma(acc, A[(size_t)l * lda + i], B[(size_t)j * ldb + l]);
    C[(size_t)j * ldc + i] = acc;
  }
}

}  // namespace

template <int WP>
__global__ void __launch_bounds__(256, 2) k_oz_rotate(RotateArgs g, int items) {
  using E = ExpProd<WP, false>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) RotShared sh;
  __shared__ int s_rowexp[WP], s_colexp[WP];
  __shared__ unsigned s_key[4][2][WP];
  const int tid = threadIdx.x, N = g.n, NN = N * N, W = g.w;
  rot_begin<E>(sh);
  double2* mats = E::MATS_IN_SMEM ? (double2*)(base + E::REGION) : g.work + (size_t)blockIdx.x * 4 * NN;
  double2 *LH = mats, *M = mats + NN, *R = mats + 2 * NN, *T = mats + 3 * NN;
  Rec rL{s_key[0][0], s_key[0][1]}, rM{s_key[1][0], s_key[1][1]}, rR{s_key[2][0], s_key[2][1]},
      rT{s_key[3][0], s_key[3][1]};
  OzCtx cx{base, base + E::SB_OFFSET, sh.tmem, smem_u32(&sh.mbar), 0u, s_rowexp, s_colexp, &sh.bad};
  const NoAdd none;
  bool ok = true;
  for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
    const int k = it / g.B, k2 = g.nnlist[it];
    const int n1 = g.rows ? g.rows[k] : W, n2 = g.rows ? g.rows[k2] : W;
    const double2 *V1 = g.v + (size_t)k * g.strideV, *V2 = g.v + (size_t)k2 * g.strideV;
    const double2* Mk = g.m + (size_t)it * g.strideM;
    rec_clear(rL, WP);
    rec_clear(rM, WP);
    rec_clear(rR, WP);
    __syncthreads();
    // V(k)^H, M and V(k+b) as N x N matrices, zero outside
    for (int e = tid; e < NN; e += 256) {
      const int i = e % N, j = e / N;
      const double2 z = cmk(0.0, 0.0);
      const double2 a = (i < n1 && j < W) ? cconj(V1[(size_t)j * g.ldv + i]) : z;   // conj V(i, j) to row j
      const double2 m = (i < n1 && j < n2) ? Mk[(size_t)j * g.ldm + i] : z;
      const double2 r = (i < n2 && j < W) ? V2[(size_t)j * g.ldv + i] : z;
      LH[(size_t)i * N + j] = a;
      M[e] = m;
      R[e] = r;
      rec_add(rL, j, i, a);
      rec_add(rM, i, j, m);
      rec_add(rR, i, j, r);
    }
    __syncthreads();
    ok = E::mm(cx, T, LH, rL.row, M, rM.col, N, Epi{T, 0, rT}, none);
    if (ok) ok = E::mm(cx, M, T, rT.row, R, rR.col, N, Epi{M, 0, Rec{nullptr, nullptr}}, none);
    double2* O = g.out + (size_t)it * W * W;
    if (__syncthreads_or(keys_wild(rL.row, N) || keys_wild(rM.col, N) || keys_wild(rR.col, N))) {
      // again from the caller's block (only the matrices' own extents: a zero of the padding times an
      // infinity is not 0)
      for (int e = tid; e < n1 * n2; e += 256)
        M[(size_t)(e / n1) * N + e % n1] = Mk[(size_t)(e / n1) * g.ldm + e % n1];
      __syncthreads();
      rot_fp64(T, N, LH, N, M, N, W, n2, n1);
      __syncthreads();
      rot_fp64(O, W, T, N, R, N, W, W, n2);
    } else if (ok) {
      for (int e = tid; e < W * W; e += 256) O[e] = M[(size_t)(e / W) * N + e % W];
    }
    // (the next block's loads come after the barrier behind its rec_clear)
  }
  if (!ok && tid == 0) *g.failed = 1;
  rot_end<E>(sh);
}

// U[cur](k) <- U0(k) U[cur](k), through dU (free on the tensor path).  One CTA per (problem, k).
template <int WP>
__global__ void __launch_bounds__(256, 2) k_oz_ufinal(const Problem* __restrict__ probs, WorkMap wm) {
  using E = ExpProd<WP, false>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) RotShared sh;
  __shared__ int s_rowexp[WP], s_colexp[WP];
  int k;
  const Problem& P = probs[locate(wm, blockIdx.x, k)];
  const int W = P.W, WW = W * W;
  double2* U = P.U[P.st->cur] + (size_t)k * WW;
  double2* C = P.dU + (size_t)k * WW;
  rot_begin<E>(sh);
  OzCtx cx{base, base + E::SB_OFFSET, sh.tmem, smem_u32(&sh.mbar), 0u, s_rowexp, s_colexp, &sh.bad};
  const double2* U0 = P.U0 + (size_t)k * WW;
  const bool ok = E::mm(cx, C, U0, nullptr, U, nullptr, W, Epi{C, 0, Rec{nullptr, nullptr}}, NoAdd());
  // the scales that the product took
  bool wild = false;
  for (int i = threadIdx.x; i < W; i += 256) wild = wild || exp_wild(s_rowexp[i]) || exp_wild(s_colexp[i]);
  if (__syncthreads_or(wild)) {
    rot_fp64(C, W, U0, W, U, W, W, W, W);
    __syncthreads();
  }
  if (ok)
    for (int e = threadIdx.x; e < WW; e += 256) U[e] = C[e];
  else if (threadIdx.x == 0) P.st->error = 2;
  rot_end<E>(sh);
}

namespace {

template <int WP>
cudaError_t rotate_wp(const RotateArgs& a, int items, cudaStream_t s) {
  constexpr int sm = (int)ExpProd<WP, false>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(k_oz_rotate<WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e != cudaSuccess) return e;
  k_oz_rotate<WP><<<std::min(items, a.ctas), 256, sm, s>>>(a, items);
  return cudaGetLastError();
}

template <int WP>
cudaError_t ufinal_wp(const Problem* probs, WorkMap wm, int grid, cudaStream_t s) {
  constexpr int sm = (int)ExpProd<WP, false>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(k_oz_ufinal<WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e != cudaSuccess) return e;
  k_oz_ufinal<WP><<<grid, 256, sm, s>>>(probs, wm);
  return cudaGetLastError();
}

}  // namespace

cudaError_t oz_rotate_launch(const RotateArgs& a, int items, cudaStream_t s) {
  if (a.n <= 16) return rotate_wp<16>(a, items, s);
  if (a.n <= 32) return rotate_wp<32>(a, items, s);
  if (a.n <= 64) return rotate_wp<64>(a, items, s);
  if (a.n <= kPolarMaxN) return rotate_wp<128>(a, items, s);
  return cudaErrorInvalidValue;
}

cudaError_t oz_ufinal_launch(int wp, const Problem* probs, WorkMap wm, int grid, cudaStream_t s) {
  switch (wp) {
    case 8:
    case 16: return ufinal_wp<16>(probs, wm, grid, s);
    case 32: return ufinal_wp<32>(probs, wm, grid, s);
    case 64: return ufinal_wp<64>(probs, wm, grid, s);
    default: return ufinal_wp<128>(probs, wm, grid, s);
  }
}

}  // namespace w90g
