// Tensor-core rotation step: dU(k) = exp(s D(k)) and U(k) <- U(k) dU(k)
// (internal_new_u_and_m, src/wannierise.F90:1655-1733) with every W x W complex
// product on the tcgen05 tensor cores through exact slicing into BF16 / FP16 digits
// (see k_tensor.cu).
//
// The matrix function is the FP64 path's (k_exp_u in k_fp64.cu): scaling and squaring
// of a Taylor polynomial evaluated by Paterson-Stockmeyer, degree and squarings chosen
// per matrix from its 1-norm.  Scalar work (norms, the polynomial's linear combinations,
// the Hermitian symmetrisation of the even powers) stays in FP64; only the products move
// to the tensor pipe (oz_mm.cuh).  The exp chain (powers, Horner steps, up to ~10 squarings
// that double any error) needs the 56-bit operands of those products.
//
// One CTA (256 threads) per (problem, k).
#include "oz_mm.cuh"

namespace w90g {

namespace {

// x 2^-j (sc = 2^-j): an exponent subtraction where the result is a normal number (the
// product is exact there, so the bits are those of x * sc), else the FP64 multiply
__device__ __forceinline__ double scale_pow2(double x, int j, double sc) {
  const long long b = __double_as_longlong(x);
  const int be = (int)((b >> 52) & 0x7FF);
  if (be > j && be != 0x7FF) return __longlong_as_double(b - ((long long)j << 52));
  return x * sc;
}

// The number of halvings that bring v >= 0 to theta (a positive normal) or below, at most
// 60: the count of the loop "while (v > theta && j < 60) { v *= 0.5; ++j; }" (halving is
// exact), from the bits with integer ops only.  Non-negative doubles order like their bit
// patterns; with v = mv 2^ev and theta = mt 2^et (mantissas in [1, 2)), v 2^-j <= theta
// first holds at j = ev - et, or one later where mv > mt.  (0 for nan, where v > theta is
// false; 60 for inf.)
__device__ __forceinline__ int halvings(double v, double theta) {
  constexpr long long kMant = 0x000FFFFFFFFFFFFFLL;
  const long long vb = __double_as_longlong(v), tb = __double_as_longlong(theta);
  if (vb <= tb) return 0;
  if ((vb >> 52) == 0x7FF && (vb & kMant) != 0) return 0;
  const int j = (int)(vb >> 52) - (int)(tb >> 52) + ((vb & kMant) > (tb & kMant) ? 1 : 0);
  return j > 60 ? 60 : j;
}

// Degree m, block size pw and squarings js of exp(X) from its 1-norm, with the cost in
// products (powers plus Horner steps, plus js): the FP64 path's table (k_exp_u), the
// cheapest candidate after the halvings that bring the norm under its theta.
struct ExpPlan {
  int m, pw, js, cost;
};
__device__ const int kPlanM[5] = {4, 6, 8, 12, 16};
__device__ const int kPlanP[5] = {4, 3, 4, 4, 4};
__device__ const double kPlanTheta[5] = {1.6e-3, 1.68e-2, 6.6e-2, 0.32, 0.78};
__device__ const int kPlanCost[5] = {3, 3, 4, 5, 6};

__device__ __noinline__ ExpPlan exp_plan(double nrm) {
  ExpPlan pl{16, 4, 0, 1 << 30};
  for (int c = 0; c < 5; ++c) {
    const int j = halvings(nrm, kPlanTheta[c]);
    const int cost = kPlanCost[c] + j;
    if (cost < pl.cost) pl = ExpPlan{kPlanM[c], kPlanP[c], j, cost};
  }
  return pl;
}

// Whether every norm within a relative 2^-14 of nrm gets the same halvings for every
// candidate -- nrm finite and at least that far from each candidate's boundaries theta
// 2^(j-1) and theta 2^j -- so that an estimate of the norm to that accuracy picks the plan
// the exact norm picks.  (nrm < x 2^j compares the bits of nrm with those of x plus j in
// the exponent field, x 2^j being a normal number here.)
__device__ __noinline__ bool exp_plan_stable(double nrm) {
  if (!(nrm < 1e300)) return false;
  const long long nb = __double_as_longlong(nrm);
  for (int c = 0; c < 5; ++c) {
    const double th = kPlanTheta[c];
    const int j = halvings(nrm, th);
    const long long lo = __double_as_longlong(th * (1.0 - 0x1p-14)), hi = __double_as_longlong(th * (1.0 + 0x1p-14));
    if (j < 60 && !(nb < lo + ((long long)j << 52))) return false;
    if (j > 0 && !(nb > hi + ((long long)(j - 1) << 52))) return false;
  }
  return true;
}

// |re + i im| to a relative 2^-20 with no FP64 instruction: each part truncated to FP32
// through its bits (0 below 2^-60, +inf above 2^60 or for inf / nan), then FP32 fma and
// q rsqrt(q) (rsqrtf: 2 ulp).  A column sum of these (<= 128 terms, FP32) is within 2^-16
// of the FP64 one.  (An infinite estimate gives a nan norm, which is never stable.)
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

__device__ const double kOzInvFact[17] = {
    1.0, 1.0, 0.5, 1.6666666666666666e-01, 4.1666666666666664e-02, 8.3333333333333332e-03,
    1.3888888888888889e-03, 1.9841269841269841e-04, 2.4801587301587302e-05,
    2.7557319223985893e-06, 2.7557319223985888e-07, 2.5052108385441720e-08,
    2.0876756987868100e-09, 1.6059043836821613e-10, 1.1470745597729725e-11,
    7.6471637318198164e-13, 4.7794773323873853e-14};

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
  __shared__ unsigned s_key[6][2][WP];
  __shared__ int s_bad;
  __shared__ double red[256];

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
  // FP64 matrices: shared memory for WP <= 32, else the per-k workspace (6 W^2)
  double2* mats = E::MATS_IN_SMEM ? (double2*)(base + E::REGION)
                                  : (P.work + (size_t)k * 6 * WW);
  double2 *X = mats, *Y2 = mats + WW, *Y3 = mats + 2 * WW, *Y4 = mats + 3 * WW, *R = mats + 4 * WW,
          *T = mats + 5 * WW;
  double2* Dk = P.D + (size_t)k * WW;
  const double s = (which == 0) ? st->s_trial : st->s_second;
  // scale records of X, Y2, Y3, Y4, R, T (see Rec).  The powers are exactly Hermitian or
  // anti-Hermitian (|re| and |im| of element (i, j) are those of (j, i)), so row i and
  // column i of their records are the same maximum: one array serves both.
  Rec rX{s_key[0][0], s_key[0][1]}, rY2{s_key[1][0], s_key[1][0]}, rY3{s_key[2][0], s_key[2][0]},
      rY4{s_key[3][0], s_key[3][0]}, rR{s_key[4][0], s_key[4][1]}, rT{s_key[5][0], s_key[5][1]};
  rec_clear(rX, WP);
  // ---- X = s D (the trial step first forms D = coefG G + coefD D_prev; in the
  // symmetry-adapted mode k_sym_dir has formed D already) and estimates of the moduli
  // |X_ij| into shared scratch.  num_wann <= 32: X stays in registers (element tid + 256 i
  // in slot i) until it is scaled below.
  constexpr bool XREG = WP <= 32;
  constexpr int NE = XREG ? (WP * WP + 255) / 256 : 1;
  double2 xr[NE];
  // the digit region is free before the first product: |X_ij| estimates, then (where the
  // exact norm is needed, once the estimates are summed) the exact moduli in its place
  float* absf = (float*)base;
  double* absx = (double*)base;
  const bool form_d = (which == 0 && P.sym_nir == 0);
  const double cg = st->coefG, cd = st->coefD;
  const double2* Gk = form_d ? (st->use_gp ? P.pc_gp : P.G) + (size_t)k * WW : nullptr;
  // (each product and the sum rounded on its own, as the oracle forms D: no contraction
  // into an FMA, whose choice of product would follow the code's shape)
  auto form_x = [&](int e) -> double2 {
    double2 d = Dk[e];
    if (form_d) {
      const double2 g = Gk[e];
      d = cmk(__dadd_rn(__dmul_rn(g.x, cg), __dmul_rn(d.x, cd)), __dadd_rn(__dmul_rn(g.y, cg), __dmul_rn(d.y, cd)));
      Dk[e] = d;
    }
    const double2 x = cscale(d, s);
    absf[e] = abs_est(x);
    return x;
  };
  if (XREG) {
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      const int e = tid + 256 * i;
      if (e < WW) xr[i] = form_x(e);
    }
  } else {
#pragma unroll 4
    for (int e = tid; e < WW; e += 256) X[e] = form_x(e);
  }
  __syncthreads();
  OzCtx cx{base, base + E::SB_OFFSET, tmem_slot, smem_u32(&mbar), 0u, s_rowexp, s_colexp, &s_bad};

  // ---- degree / squarings from the 1-norm (the FP64 path's table and choice, exp_plan).
  // The plan depends on the norm only through which side of each theta 2^j it lies, so
  // the FP32 estimate decides wherever it is clearly inside one interval
  // (exp_plan_stable); else the exact FP64 norm is formed -- moduli, then each column
  // summed in row order -- as the FP64 path forms it.  One thread plans, all read it.
  __shared__ float s_wmax[8];
  __shared__ int s_plan[5];
  {
    float colmax = 0.0f;
    for (int j = tid; j < W; j += 256) {
      float a = 0.0f;
      for (int i = 0; i < W; ++i) a += absf[(size_t)j * W + i];
      colmax = fmaxf(colmax, a);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) colmax = fmaxf(colmax, __shfl_xor_sync(0xffffffffu, colmax, o));
    if ((tid & 31) == 0) s_wmax[warp] = colmax;
  }
  __syncthreads();
  if (tid == 0) {
    float nf = 0.0f;
    for (int w = 0; w < 8; ++w) nf = fmaxf(nf, s_wmax[w]);
    const bool stable = exp_plan_stable((double)nf);
    const ExpPlan pl = exp_plan((double)nf);
    s_plan[0] = pl.m;
    s_plan[1] = pl.pw;
    s_plan[2] = pl.js;
    s_plan[3] = stable ? 0 : 1;
    s_plan[4] = pl.cost;
  }
  __syncthreads();
  if (s_plan[3]) {
    auto exact_abs = [&](int e, double2 x) { absx[e] = sqrt(cabs2(x)); };
    if (XREG) {
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const int e = tid + 256 * i;
        if (e < WW) exact_abs(e, xr[i]);
      }
    } else {
      for (int e = tid; e < WW; e += 256) exact_abs(e, X[e]);
    }
    __syncthreads();
    double colmax = 0.0;
    for (int j = tid; j < W; j += 256) {
      double a = 0.0;
      for (int i = 0; i < W; ++i) a += absx[(size_t)j * W + i];
      colmax = fmax(colmax, a);
    }
    __syncthreads();
    const double nrm = cta_max(colmax, red);
    if (tid == 0) {
      const ExpPlan pl = exp_plan(nrm);
      s_plan[0] = pl.m;
      s_plan[1] = pl.pw;
      s_plan[2] = pl.js;
      s_plan[4] = pl.cost;
    }
    __syncthreads();
  }
  const int m = s_plan[0], pw = s_plan[1], js = s_plan[2];
  const double sc = ldexp(1.0, -js);
  auto scale_x = [&](int e, double2 x) {
    const double2 v = make_double2(scale_pow2(x.x, js, sc), scale_pow2(x.y, js, sc));
    X[e] = v;
    rec_add(rX, e % W, e / W, v);
  };
  if (XREG) {
#pragma unroll
    for (int i = 0; i < NE; ++i) {
      const int e = tid + 256 * i;
      if (e < WW) scale_x(e, xr[i]);
    }
  } else {
#pragma unroll 4
    for (int e = tid; e < WW; e += 256) scale_x(e, X[e]);
  }
  __syncthreads();
  const NoAdd none;
  // powers, exactly Hermitian (even) / anti-Hermitian (odd) as the FP64 path forms them
  bool ok = E::mm(cx, Y2, X, rX.row, X, rX.col, W, Epi{Y2, 1, rY2}, none);
  if (ok) ok = E::mm(cx, Y3, Y2, rY2.row, X, rX.col, W, Epi{Y3, -1, rY3}, none);
  if (ok && pw >= 4) ok = E::mm(cx, Y4, Y2, rY2.row, Y2, rY2.col, W, Epi{Y4, 1, rY4}, none);
  const double2* Yp = (pw == 4) ? Y4 : Y3;
  const Rec rYp = (pw == 4) ? rY4 : rY3;
  const int nblk = (m + pw) / pw;
  // block q of the polynomial, sum_r c_{pw q + r} X^r (X^0 = I), one FMA per term and part
  // (the FP64 pipe runs at 1/64 of FP32 on this chip: these elementwise terms are a large
  // part of the chain's FP64 work)
  auto blk = [&](int q, int e) -> double2 {
    const int i = e % W, j = e / W;
    double2 v = cmk(0.0, 0.0);
    for (int r = 0; r < pw; ++r) {
      const int deg = pw * q + r;
      if (deg > m) break;
      const double c = kOzInvFact[deg];
      if (r == 0) {
        if (i == j) v.x += c;
      } else {
        const double2 y = (r == 1) ? X[e] : ((r == 2) ? Y2[e] : Y3[e]);
        v = cmk(fma(y.x, c, v.x), fma(y.y, c, v.y));
      }
    }
    return v;
  };
  int q = nblk - 1;
  rec_clear(rR, WP);
  __syncthreads();
  if (pw * q == m) {
    const double cm = kOzInvFact[m];
    #pragma unroll 4
    for (int e = tid; e < WW; e += blockDim.x) {
      const double2 b = blk(q - 1, e), y = Yp[e];
      const double2 v = cmk(fma(y.x, cm, b.x), fma(y.y, cm, b.y));
      R[e] = v;
      rec_add(rR, e % W, e / W, v);
    }
    q -= 1;
  } else {
    #pragma unroll 4
    for (int e = tid; e < WW; e += blockDim.x) {
      const double2 v = blk(q, e);
      R[e] = v;
      rec_add(rR, e % W, e / W, v);
    }
  }
  __syncthreads();
  // Horner steps R <- Yp R + block q (the product's epilogue adds the block)
  for (q = q - 1; q >= 0 && ok; --q) {
    const HornerAdd<decltype(blk)> hadd{&blk, q};
    ok = E::mm(cx, T, Yp, rYp.row, R, rR.col, W, Epi{R, 0, rR}, hadd);
  }
  double2* a = R;
  double2* b = T;
  Rec ra = rR, rb = rT;
  for (int sq = 0; sq < js && ok; ++sq) {
    ok = E::mm(cx, b, a, ra.row, a, ra.col, W, Epi{b, 0, rb}, none);
    double2* tmp = a;
    a = b;
    b = tmp;
    const Rec rt = ra;
    ra = rb;
    rb = rt;
  }
  // dU = exp(s D);  U[cur^1] = U[cur] dU
  double2* dUk = P.dU + (size_t)k * WW;
  #pragma unroll 4
  for (int e = tid; e < WW; e += blockDim.x) dUk[e] = a[e];
  __syncthreads();
  const int cur = st->cur;
  double2* Unew = P.U[cur ^ 1] + (size_t)k * WW;
  if (ok) ok = E::mm(cx, Unew, P.U[cur] + (size_t)k * WW, nullptr, a, ra.col, W, Epi{Unew, 0, Rec{nullptr, nullptr}},
                     none);
  if (tid == 0) atomicAdd(&st->exp_products, (double)s_plan[4] + 1.0);   // the plan's cost, + U dU
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
