// Tensor-core rotation step: U(k) <- U(k) exp(s D(k)) (internal_new_u_and_m,
// src/wannierise.F90:1655-1733) with every W x W complex product on the tcgen05 tensor cores
// through exact slicing into FP16 digits at 56-bit precision (oz_mm.cuh); norms and the
// polynomials' linear combinations are FP64 (the norms' moduli FP32).
//
// The matrix function is a Taylor polynomial of degree 4, 8 or 12 of X 2^-js, squared js times.
// What it costs is products (each: slice two operands, 28 to 36 digit-pair MMAs, recombine), so
//   * the polynomials are evaluated with 2, 3 and 4 products (powers included) instead of
//     Paterson-Stockmeyer's 3, 4 and 5:
//       T4  = I + X + X^2 (1/2 + X/6 + X^2/24)
//       T8  = I + X + y2 X^2 + (x3 X^2 + A) (x4 + x5 X + x6 X^2 + x7 A),  A = X^2 (x1 X + x2 X^2)
//             (P. Bader, S. Blanes, F. Casas, Mathematics 7 (2019) 1174)
//       T12 = I + X + c2 X^2 + c3 X^3 + (B2 + A) A,  A = a2 X^2 + a3 X^3 + B4^2, B2 and B4 cubics
//             (their form; of its one-parameter family of solutions the one without constant
//             and linear terms in A, so that nothing cancels against I);
//   * the scaling follows sqrt(||X^2||_1), which bounds the 2-norm of the anti-Hermitian X and is
//     half of ||X||_1 or less for a full W = 32 matrix: one squaring less on average;
//   * the optimal step's X is a multiple of the trial step's, so its powers are the trial's: the
//     factor f goes into the coefficients and the second exp starts after them.  (Where the trial's
//     norm says too little about the optimal step's -- see `reuse` -- the second exp forms its own.)
// Truncation: theta^(m+1) / (m+1)! <= 2^-53 at the 2-norm theta (||e^X||_2 = 1).
//
// One CTA (256 threads) per (problem, k).
#include "oz_mm.cuh"

namespace w90g {

namespace {

// T8: x1..x7, y2; T12: B2 (0..3), B4 (1..3), a2, a3, c2, c3.  T8 in closed form; T12 by Newton's
// method on the 13 coefficient equations in 40 digits.
constexpr double kT8x1 = 0.10836465678522780852, kT8x2 = 0.027091164196306952131, kT8x3 = 0.66666666666666666667,
                 kT8x4 = 0.54676145797072405251, kT8x5 = 0.16112557339541759283, kT8x6 = 0.014090917158378207731,
                 kT8x7 = 0.033792797010870504141, kT8y2 = 0.13549236135285063166;
constexpr double kT12b0 = 5.0188519759285061501, kT12b1 = 1.3093238729699402869, kT12b2 = 0.15744598937135220317,
                 kT12b3 = -0.0014710039978467423724, kT12e1 = 0.13181061013830184016,
                 kT12e2 = 0.020278555405892590793, kT12e3 = 0.0067595184686308635978,
                 kT12a2 = 0.020689394224651494005, kT12a3 = 0.012386729930502613689,
                 kT12c2 = 0.30896527326341831812, kT12c3 = 0.027832075977002841435;

// degree m and squarings js of a 2-norm: the cheapest of T4 (2 products up to 1.6e-3), T8 (3 up
// to 6.6e-2) and T12 (4 up to 0.32, one more per doubling); at most 60 squarings
__device__ __forceinline__ void exp_plan(float rho, int& m, int& js) {
  js = 0;
  if (rho <= 1.6e-3f) {
    m = 4;
  } else if (rho <= 6.6e-2f) {
    m = 8;
  } else {
    m = 12;
    while (rho > 0.32f && js < 60) {
      rho *= 0.5f;
      ++js;
    }
  }
}

// |re + i im| in FP32 to a relative 2^-20 (0 below 2^-60, +inf above 2^60 or for inf / nan)
// with no FP64 instruction: each part truncated through its bits, then fma and q rsqrt(q)
__device__ __forceinline__ float abs_est(double2 v) {
  auto f32 = [](double x) -> float {
    const unsigned long long b = abs_bits(x);
    const int e = (int)(b >> 52) - 1023;
    if (e < -60) return 0.0f;
    if (e > 60) return __int_as_float(0x7f800000);
    return __uint_as_float(((unsigned)(e + 127) << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
  };
  const float a = f32(v.x), b = f32(v.y);
  const float q = fmaf(a, a, b * b);
  return q > 0.0f ? q * rsqrtf(q) : 0.0f;
}

// c0 I + c1 X + c2 P2 + c3 P3 at element e, added by a product's epilogue
struct PolyAdd {
  static constexpr bool kActive = true;
  const double2 *X, *P2, *P3;
  double c0, c1, c2, c3;
  int W;
  __device__ double2 operator()(int e) const {
    double2 v = cmk((e % W) == (e / W) ? c0 : 0.0, 0.0);
    if (c1 != 0.0) {
      const double2 x = X[e];
      v = cmk(fma(x.x, c1, v.x), x.y * c1);
    }
    const double2 p = P2[e];
    v = cmk(fma(p.x, c2, v.x), fma(p.y, c2, v.y));
    if (c3 != 0.0) {
      const double2 r = P3[e];
      v = cmk(fma(r.x, c3, v.x), fma(r.y, c3, v.y));
    }
    return v;
  }
};

}  // namespace

// which = 0: trial step (also forms D = coefG (G or Gp) + coefD D_prev); 1: optimal step
template <int WP, bool SMEM_MATS>
__global__ void __launch_bounds__(256, 2) k_oz_exp(const Problem* __restrict__ probs, WorkMap wm, int which) {
  using E = ExpProd<WP, SMEM_MATS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_rowexp[WP], s_colexp[WP];
  __shared__ unsigned s_key[5][2][WP];
  __shared__ int s_bad;
  __shared__ float s_wmax[8];
  __shared__ double s_f;
  __shared__ float s_rho;
  __shared__ int s_reuse, s_have3;

  int k;
  const int p = locate(wm, blockIdx.x, k);
  const Problem& P = probs[p];
  CtrlState* st = P.st;
  if (st->done) return;
  if (which == 1 && !st->do_second) return;
  const int W = P.W, WW = W * W;
  const int tid = threadIdx.x, warp = tid >> 5;

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
  // the matrices: shared memory for WP <= 16 (32 on request), else the per-k workspace (6 W^2),
  // whose first three -- X and its powers -- the optimal step's launch finds there
  double2* kept = P.work + (size_t)k * 6 * WW;
  double2* mats = E::MATS_IN_SMEM ? (double2*)(base + E::REGION) : kept;
  double2 *X = mats, *P2 = mats + WW, *P3 = mats + 2 * WW, *Z = mats + 3 * WW, *A = mats + 4 * WW,
          *L = mats + 5 * WW;
  float* info = P.expinfo + (size_t)k * 2;   // sqrt(||X^2||_1) of the trial step; 1 when P3 is there
  // scale records (see Rec).  The powers are exactly Hermitian or anti-Hermitian (|re| and |im| of
  // element (i, j) are those of (j, i)), so row i and column i of their records are the same
  // maximum: one array serves both.
  Rec rX{s_key[0][0], s_key[0][0]}, rP2{s_key[0][1], s_key[0][1]}, rZ{s_key[2][0], s_key[2][1]},
      rA{s_key[3][0], s_key[3][1]}, rL{s_key[4][0], s_key[4][1]};
  const Rec norec{nullptr, nullptr};
  const NoAdd none;
  rec_clear(rX, WP);
  rec_clear(rP2, WP);
  rec_clear(rZ, WP);
  rec_clear(rL, WP);
  if (which == 1 && tid == 0) {
    // (one thread: an FP64 divide by all of them takes the FP64 pipe a microsecond)
    const double q = st->s_second / st->s_trial;
    const float r = info[0], g = (float)q;
    // The trial's powers serve the optimal step where its plan is safe: abs_est leaves out moduli of
    // X^2 below 2^-60, at most 2^-53 in a column sum.  From a norm of 2^-24 on that is 1.5 % of it,
    // within the plan's own slack of 5 %; below, as long as T4 covers the step whatever was left out
    // (steps of a thousand times the trial's are ordinary near the minimum).  A longer step, or any
    // after a trial of length 0 (the ratio is NaN or infinite), starts from its own X.
    s_reuse = (r >= 0x1p-24f && fabsf(g) <= 0x1p60f) || (r * r + 0x1p-53f) * (g * g) <= 1.6e-3f * 1.6e-3f;
    s_f = q;
    s_rho = r * fabsf(g) * 1.0001f;
    s_have3 = info[1] != 0.0f;
  }
  __syncthreads();
  OzCtx cx{base, base + E::SB_OFFSET, tmem_slot, smem_u32(&mbar), 0u, s_rowexp, s_colexp, &s_bad};
  bool ok = true;
  float rho;
  double f = 1.0;
  bool have3 = false;
  int nprod = 0;
  const bool reuse = which == 1 && s_reuse;
  if (!reuse) {
    // ---- X = s D (first D = coefG G + coefD D_prev; in the symmetry-adapted mode k_sym_dir has
    // formed D already).  Each product and the sum rounded on its own, as the oracle forms D:
    // no contraction into an FMA, whose choice of product would follow the code's shape.
    double2* Dk = P.D + (size_t)k * WW;
    const double s = which == 0 ? st->s_trial : st->s_second;
    const bool form_d = which == 0 && P.sym_nir == 0;
    const double cg = st->coefG, cd = st->coefD;
    const double2* Gk = form_d ? (st->use_gp ? P.pc_gp : P.G) + (size_t)k * WW : nullptr;
#pragma unroll 4
    for (int e = tid; e < WW; e += 256) {
      double2 d = Dk[e];
      if (form_d) {
        const double2 g = Gk[e];
        d = cmk(__dadd_rn(__dmul_rn(g.x, cg), __dmul_rn(d.x, cd)), __dadd_rn(__dmul_rn(g.y, cg), __dmul_rn(d.y, cd)));
        Dk[e] = d;
      }
      const double2 x = cscale(d, s);
      X[e] = x;
      rec_add(rX, e % W, e / W, x);
    }
    __syncthreads();
    ok = E::mm(cx, P2, X, rX.row, X, rX.col, W, Epi{P2, 1, rP2}, none);
    ++nprod;
    // ---- sqrt(||X^2||_1) from FP32 moduli (their sums are within 2^-16; 2^-10 on top)
    float* absf = (float*)base;   // the digit region is free between products
    for (int e = tid; e < WW; e += 256) absf[e] = abs_est(P2[e]);
    __syncthreads();
    float cmax = 0.0f;
    for (int j = tid; j < W; j += 256) {
      float a = 0.0f;
      for (int i = 0; i < W; ++i) a += absf[(size_t)j * W + i];
      cmax = fmaxf(cmax, a);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
    if ((tid & 31) == 0) s_wmax[warp] = cmax;
    __syncthreads();
    cmax = 0.0f;
    for (int w = 0; w < 8; ++w) cmax = fmaxf(cmax, s_wmax[w]);
    rho = sqrtf(cmax * 1.001f);
  } else {
    f = s_f;
    rho = s_rho;
    have3 = s_have3 != 0;
  }
  int m, js;
  exp_plan(rho, m, js);
  f *= ldexp(1.0, -js);
  if (reuse) {
    // the powers kept by the trial step, with the records of those that enter a product
    const bool need = m < 12 || !have3;
    if (E::MATS_IN_SMEM || need)
      for (int e = tid; e < WW; e += 256) {
        const double2 x = kept[e], q = kept[WW + e];
        if (E::MATS_IN_SMEM) {
          X[e] = x;
          P2[e] = q;
          if (have3) P3[e] = kept[2 * WW + e];
        }
        if (need) {
          rec_add(rX, e % W, e / W, x);
          rec_add(rP2, e % W, e / W, q);
        }
      }
    __syncthreads();
  }
  const double f2 = f * f, f3 = f2 * f;
  double2* Ex = Z;     // where the polynomial ends up
  Rec rE = rZ;
  if (m == 4) {
    // E = P2 [f^2 (1/2 + f X / 6 + f^2 P2 / 24)] + I + f X
    for (int e = tid; e < WW; e += 256) {
      const double2 x = X[e], q = P2[e];
      const double d = (e % W) == (e / W) ? 0.5 * f2 : 0.0;
      const double2 z = cmk(fma(q.x, f2 * f2 / 24.0, fma(x.x, f3 / 6.0, d)), fma(q.y, f2 * f2 / 24.0, x.y * (f3 / 6.0)));
      L[e] = z;
      rec_add(rL, e % W, e / W, z);
    }
    __syncthreads();
    if (ok) ok = E::mm(cx, Z, P2, rP2.row, L, rL.col, W, Epi{Z, 0, rZ}, PolyAdd{X, P2, P3, 1.0, f, 0.0, 0.0, W});
    nprod += 1;
  } else if (m == 8) {
    for (int e = tid; e < WW; e += 256) {
      const double2 x = X[e], q = P2[e];
      const double2 z = cmk(fma(q.x, kT8x2 * f2 * f2, x.x * (kT8x1 * f3)), fma(q.y, kT8x2 * f2 * f2, x.y * (kT8x1 * f3)));
      L[e] = z;
      rec_add(rL, e % W, e / W, z);
    }
    __syncthreads();
    if (ok) ok = E::mm(cx, A, P2, rP2.row, L, rL.col, W, Epi{A, 0, norec}, none);
    rec_clear(rL, WP);
    rec_clear(rA, WP);
    __syncthreads();
    // left factor into L, right factor over A
    for (int e = tid; e < WW; e += 256) {
      const double2 x = X[e], q = P2[e], a = A[e];
      const double d = (e % W) == (e / W) ? kT8x4 : 0.0;
      const double2 l = cmk(fma(q.x, kT8x3 * f2, a.x), fma(q.y, kT8x3 * f2, a.y));
      const double2 r = cmk(fma(a.x, kT8x7, fma(q.x, kT8x6 * f2, fma(x.x, kT8x5 * f, d))),
                            fma(a.y, kT8x7, fma(q.y, kT8x6 * f2, x.y * (kT8x5 * f))));
      L[e] = l;
      A[e] = r;
      rec_add(rL, e % W, e / W, l);
      rec_add(rA, e % W, e / W, r);
    }
    __syncthreads();
    if (ok) ok = E::mm(cx, Z, L, rL.row, A, rA.col, W, Epi{Z, 0, rZ}, PolyAdd{X, P2, P3, 1.0, f, kT8y2 * f2, 0.0, W});
    nprod += 2;
  } else {
    if (!have3) {
      if (ok) ok = E::mm(cx, P3, P2, rP2.row, X, rX.col, W, Epi{P3, -1, norec}, none);
      ++nprod;
      have3 = true;
    }
    for (int e = tid; e < WW; e += 256) {
      const double2 x = X[e], q = P2[e], r = P3[e];
      const double2 z = cmk(fma(r.x, kT12e3 * f3, fma(q.x, kT12e2 * f2, x.x * (kT12e1 * f))),
                            fma(r.y, kT12e3 * f3, fma(q.y, kT12e2 * f2, x.y * (kT12e1 * f))));
      Z[e] = z;
      rec_add(rZ, e % W, e / W, z);
    }
    __syncthreads();
    if (ok) ok = E::mm(cx, A, Z, rZ.row, Z, rZ.col, W, Epi{A, 0, rA}, PolyAdd{X, P2, P3, 0.0, 0.0, kT12a2 * f2, kT12a3 * f3, W});
    for (int e = tid; e < WW; e += 256) {
      const double2 x = X[e], q = P2[e], r = P3[e], a = A[e];
      const double d = (e % W) == (e / W) ? kT12b0 : 0.0;
      const double2 l = cmk(a.x + fma(r.x, kT12b3 * f3, fma(q.x, kT12b2 * f2, fma(x.x, kT12b1 * f, d))),
                            a.y + fma(r.y, kT12b3 * f3, fma(q.y, kT12b2 * f2, x.y * (kT12b1 * f))));
      L[e] = l;
      rec_add(rL, e % W, e / W, l);
    }
    __syncthreads();
    if (ok)
      ok = E::mm(cx, Z, L, rL.row, A, rA.col, W, Epi{Z, 0, rZ}, PolyAdd{X, P2, P3, 1.0, f, kT12c2 * f2, kT12c3 * f3, W});
    nprod += 2;
  }
  // ---- squarings, between Z and A
  double2* other = A;
  Rec ro = rA;
  for (int sq = 0; sq < js && ok; ++sq) {
    ok = E::mm(cx, other, Ex, rE.row, Ex, rE.col, W, Epi{other, 0, ro}, none);
    double2* t = Ex;
    Ex = other;
    other = t;
    const Rec rt = rE;
    rE = ro;
    ro = rt;
  }
  // ---- U[cur^1] = U[cur] exp(s D)
  const int cur = st->cur;
  double2* Unew = P.U[cur ^ 1] + (size_t)k * WW;
  if (ok) ok = E::mm(cx, Unew, P.U[cur] + (size_t)k * WW, nullptr, Ex, rE.col, W, Epi{Unew, 0, norec}, none);
  if (which == 0) {
    // for the optimal step
    if (E::MATS_IN_SMEM)
      for (int e = tid; e < WW; e += 256) {
        kept[e] = X[e];
        kept[WW + e] = P2[e];
        if (have3) kept[2 * WW + e] = P3[e];
      }
    if (tid == 0) {
      info[0] = rho;
      info[1] = have3 ? 1.0f : 0.0f;
    }
  }
  if (tid == 0) atomicAdd(&st->exp_products, (double)(nprod + js) + 1.0);   // and U exp(s D)
  if (!ok && tid == 0) {
    st->error = 2;
    st->done = 1;
  }
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(cx.tmem), "r"((uint32_t)E::TMEM_COLS) : "memory");
  }
}

template <int WP, bool SM>
static cudaError_t oz_exp_launch_wp(const Problem* probs, WorkMap wm, int which, int grid, cudaStream_t s) {
  k_oz_exp<WP, SM><<<grid, 256, ExpProd<WP, SM>::BYTES, s>>>(probs, wm, which);
  return cudaGetLastError();
}

// smem_mats: num_wann 17..32, keep the chain's FP64 matrices in shared memory
cudaError_t oz_exp_launch(int wp, int smem_mats, const Problem* probs, WorkMap wm, int which, int grid,
                          cudaStream_t s) {
  switch (wp) {
    case 8: return oz_exp_launch_wp<8, false>(probs, wm, which, grid, s);
    case 16: return oz_exp_launch_wp<16, false>(probs, wm, which, grid, s);
    case 32:
      return smem_mats ? oz_exp_launch_wp<32, true>(probs, wm, which, grid, s)
                       : oz_exp_launch_wp<32, false>(probs, wm, which, grid, s);
    case 64: return oz_exp_launch_wp<64, false>(probs, wm, which, grid, s);
    default: return oz_exp_launch_wp<128, false>(probs, wm, which, grid, s);
  }
}

template <int WP, bool SM>
static cudaError_t oz_exp_attr_wp() {
  return cudaFuncSetAttribute(k_oz_exp<WP, SM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)ExpProd<WP, SM>::BYTES);
}

cudaError_t oz_exp_set_attributes(int wp, int smem_mats) {
  switch (wp) {
    case 8: return oz_exp_attr_wp<8, false>();
    case 16: return oz_exp_attr_wp<16, false>();
    case 32: return smem_mats ? oz_exp_attr_wp<32, true>() : oz_exp_attr_wp<32, false>();
    case 64: return oz_exp_attr_wp<64, false>();
    default: return oz_exp_attr_wp<128, false>();
  }
}

}  // namespace w90g
