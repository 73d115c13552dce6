// CTA-wide building blocks shared by the FP64 kernels: deterministic block reductions
// and a parallel-ordered Jacobi eigensolver for small Hermitian matrices.
#pragma once
#include "w90g.cuh"

namespace w90g {

__device__ __forceinline__ double block_sum(double v, double* red) {
  // deterministic tree reduction over blockDim.x (power of two, <= 1024)
  int t = threadIdx.x;
  red[t] = v;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if (t < s) red[t] += red[t + s];
    __syncthreads();
  }
  double r = red[0];
  __syncthreads();
  return r;
}

__device__ __forceinline__ double block_max(double v, double* red) {
  int t = threadIdx.x;
  red[t] = v;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if (t < s) red[t] = fmax(red[t], red[t + s]);
    __syncthreads();
  }
  double r = red[0];
  __syncthreads();
  return r;
}

// ----------------------------------------------------------------------------
// Parallel-ordered cyclic Jacobi eigensolver for a Hermitian W x W matrix H (generic
// pointer, overwritten by its near-diagonal form); V receives the eigenvectors
// (columns).  Rotation for pair (p,q):  J = [[c, s e^{i phi}], [-s e^{-i phi}, c]],
// phi = arg(H_pq), (c, s) the real Jacobi rotation of [[H_pp, |H_pq|], [|H_pq|, H_qq]].
// Convergence: sum_{p != q} |H_pq|^2 <= 1e-30 ||H||_F^2.  With skip_rel > 0, pairs with
// |H_pq|^2 <= skip_rel ||H||_F^2 are left alone and a sweep that rotates no pair also ends
// the solve (the threshold-Jacobi rule: reachable at any size, where the plain criterion
// can sit at the roundoff floor of large matrices).
// Returns the number of FP64 sweeps used (or -1 when not converged within max_sweeps).
//
// What bounds it is the FP64 pipe (2 lanes per SM), so the work is arranged to need few
// FP64 instructions:
//   * a round's rotations touch pairs of pairs: each 2 x 2 block of H is updated once,
//     B <- J_s^H B J_t, and mirrored (6 W^3 FMA per sweep for H, not 12), and a block or
//     column pair whose rotations were skipped is left alone;
//   * given two W x W scratch matrices (s1, s2), the first sweeps run in FP32 on a scaled
//     copy kept in V's storage.  Their eigenvectors, orthonormalised to FP64 by one cubic
//     Newton-Schulz step V (15/8 - 10/8 G + 3/8 G^2), G = V^H V, turn H into V^H H V with an
//     off-diagonal part of ~1e-6, from which the FP64 sweeps -- the same rotations and the
//     same convergence test -- need two instead of seven to ten.  14 W^3 FMA for that against
//     12 W^3 per sweep.
// ----------------------------------------------------------------------------
struct JacF2 {
  float x, y;
};

template <class R, class R2>
__device__ __forceinline__ R2 jac_mk(R x, R y) {
  R2 r;
  r.x = x;
  r.y = y;
  return r;
}
// c a - conj(s) b  and  s a + c b
template <class R, class R2>
__device__ __forceinline__ R2 jac_p(R c, R2 s, R2 a, R2 b) {
  return jac_mk<R, R2>(c * a.x - (s.x * b.x + s.y * b.y), c * a.y - (s.x * b.y - s.y * b.x));
}
template <class R, class R2>
__device__ __forceinline__ R2 jac_q(R c, R2 s, R2 a, R2 b) {
  return jac_mk<R, R2>(c * b.x + (s.x * a.x - s.y * a.y), c * b.y + (s.x * a.y + s.y * a.x));
}
template <class R2>
__device__ __forceinline__ R2 jac_conj(R2 a) {
  R2 r;
  r.x = a.x;
  r.y = -a.y;
  return r;
}

// element e of the upper triangle i <= j, counted down the columns: e = j (j + 1) / 2 + i
// (consecutive threads take consecutive elements, so no warp idles on the lower triangle)
__device__ __forceinline__ void tri_index(int e, int& i, int& j) {
  j = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
  while (j * (j + 1) / 2 > e) --j;
  while ((j + 1) * (j + 2) / 2 <= e) ++j;
  i = e - j * (j + 1) / 2;
}

// 1 / sqrt(x) to FP64 for x in FP32's normal range, from FP32 and two Newton steps: 8 FP64
// operations, where the FP64 square root and divide take about 40 each
__device__ __forceinline__ double jac_rsqrt(double x) {
  double y = (double)(1.0f / sqrtf((float)x));
  y = y * (1.5 - 0.5 * x * y * y);
  return y * (1.5 - 0.5 * x * y * y);
}

// Rotation of the pair block [[a, b], [conj(b), d]], b2 = |b|^2 > 0: c, s e^{i phi} and the rotated
// block (pp, off, qq).  The angle needs no more than FP32 -- it leaves 1e-7 of b for the next sweep,
// which the sweeps' quadratic convergence hides -- but c and the phase are unitary to FP64, and the
// block is formed for the angle taken.  (Angle, c and phase in FP64 were 38 % of an m = 26 sweep.)
__device__ __forceinline__ void jac_rotation(double a, double d, double2 b, double b2, double& c, double2& se,
                                             double& pp, double& qq, double2& off) {
  double rinv;
  if (b2 > 1.0e-30 && b2 < 1.0e30) rinv = jac_rsqrt(b2);
  else rinv = 1.0 / sqrt(b2);
  const double ab = b2 * rinv, g = d - a;
  const float th = (float)(0.5 * g * rinv);
  const float ath = fabsf(th);
  // (beyond 1e15 the angle is 1 / (2 th); th^2 would overflow)
  const float tf = ath < 1.0e15f ? 1.0f / (ath + sqrtf(1.0f + th * th)) : 0.5f / ath;
  const double t = th >= 0.0f ? (double)tf : -(double)tf;
  c = jac_rsqrt(1.0 + t * t);
  const double s = t * c, cs = c * s, ss = s * s;
  const double2 ph = cmk(b.x * rinv, b.y * rinv);
  se = cmk(s * ph.x, s * ph.y);
  const double x = 2.0 * cs * ab - ss * g;     // a - x, d + x
  pp = a - x;
  qq = d + x;
  const double o = (1.0 - 2.0 * ss) * ab - cs * g;
  off = cmk(o * ph.x, o * ph.y);
}
__device__ __forceinline__ void jac_rotation(float a, float d, JacF2 b, float b2, float& c, JacF2& se, float& pp,
                                             float& qq, JacF2& off) {
  const float ab = sqrtf(b2), th = (d - a) / (2.0f * ab);
  const float tt = (th >= 0.0f ? 1.0f : -1.0f) / (fabsf(th) + sqrtf(1.0f + th * th));
  c = 1.0f / sqrtf(1.0f + tt * tt);
  const float s = tt * c / ab;
  se.x = s * b.x;
  se.y = s * b.y;
  pp = a - tt * ab;
  qq = d + tt * ab;
  off.x = off.y = 0.0f;
}

// One sweep of rotations over all pairs of H, applied to V; pairs with |H_pq|^2 <= tiny
// or <= thr are skipped.  Returns how many pairs this thread rotated.
template <class R, class R2>
__device__ __forceinline__ int jac_sweep(R2* H, R2* V, int W, R thr, R tiny, R* rc, R2* rse, int* rp, int* rq) {
  const int n = (W + 1) & ~1;     // even number of players (one dummy when W is odd)
  const int npair = n / 2;
  const int nblk = npair * (npair - 1) / 2;
  int rotated = 0;
  for (int r = 0; r < n - 1; ++r) {
    for (int t = threadIdx.x; t < npair; t += blockDim.x) {
      int p, q;
      if (t == 0) {
        p = r;
        q = n - 1;
      } else {
        p = r + t;
        if (p >= n - 1) p -= n - 1;
        q = r - t;
        if (q < 0) q += n - 1;
      }
      if (p > q) {
        const int x = p;
        p = q;
        q = x;
      }
      R c = R(1);
      R2 se = jac_mk<R, R2>(R(0), R(0));
      int live = 0;
      if (q < W) {
        const R2 b = H[q * W + p];
        const R b2 = b.x * b.x + b.y * b.y;
        if (b2 > tiny && b2 > thr) {
          live = 1;
          ++rotated;
          R pp, qq;
          R2 off;
          jac_rotation(H[p * W + p].x, H[q * W + q].x, b, b2, c, se, pp, qq, off);
          H[p * W + p] = jac_mk<R, R2>(pp, R(0));
          H[q * W + q] = jac_mk<R, R2>(qq, R(0));
          H[q * W + p] = off;
          H[p * W + q] = jac_conj(off);
        }
      }
      rp[t] = p;
      rq[t] = live ? q : (q < W ? q + 0x10000 : 0x20000);   // bit 16: no rotation; bit 17: dummy
      rc[t] = c;
      rse[t] = se;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nblk + W * npair; e += blockDim.x) {
      if (e < nblk) {
        int s, t;   // block (s, t), s < t
        tri_index(e, s, t);
        ++t;
        const int qsx = rq[s], qtx = rq[t];
        if (qsx >= 0x10000 && qtx >= 0x10000) continue;
        const bool ds = (qsx & 0x20000) != 0, dt = (qtx & 0x20000) != 0;
        const int ps = rp[s], pt = rp[t], qs = ds ? ps : (qsx & 0xFFFF), qt = dt ? pt : (qtx & 0xFFFF);
        const R cs = rc[s], ct = rc[t];
        const R2 ss = rse[s], st = rse[t];
        // (a dummy's partner repeats its own element; its rotation is the identity and its
        // results are not stored)
        const R2 b11 = H[pt * W + ps], b12 = H[qt * W + ps], b21 = H[pt * W + qs], b22 = H[qt * W + qs];
        const R2 x11 = jac_p(ct, st, b11, b12), x12 = jac_q(ct, st, b11, b12);
        const R2 x21 = jac_p(ct, st, b21, b22), x22 = jac_q(ct, st, b21, b22);
        // rows by J_s^H: c x_p - s x_q and conj(s) x_p + c x_q
        const R2 sc = jac_conj(ss);
        const R2 y11 = jac_p(cs, sc, x11, x21), y21 = jac_q(cs, sc, x11, x21);
        const R2 y12 = jac_p(cs, sc, x12, x22), y22 = jac_q(cs, sc, x12, x22);
        H[pt * W + ps] = y11;
        H[ps * W + pt] = jac_conj(y11);
        if (!dt) {
          H[qt * W + ps] = y12;
          H[ps * W + qt] = jac_conj(y12);
        }
        if (!ds) {
          H[pt * W + qs] = y21;
          H[qs * W + pt] = jac_conj(y21);
          if (!dt) {
            H[qt * W + qs] = y22;
            H[qs * W + qt] = jac_conj(y22);
          }
        }
      } else {
        // columns of V: V <- V J
        const int i = (e - nblk) % W, t = (e - nblk) / W;
        const int q = rq[t];
        if (q >= 0x10000) continue;
        const int p = rp[t];
        const R2 vp = V[p * W + i], vq = V[q * W + i];
        V[p * W + i] = jac_p(rc[t], rse[t], vp, vq);
        V[q * W + i] = jac_q(rc[t], rse[t], vp, vq);
      }
    }
    __syncthreads();
  }
  return rotated;
}

// C = op(A) B (W x W, column-major), the upper triangle only and mirrored when HERM
template <bool CA, bool HERM>
__device__ __forceinline__ void jac_mm(double2* C, const double2* A, const double2* B, int W) {
  const int items = HERM ? W * (W + 1) / 2 : W * W;
  for (int e = threadIdx.x; e < items; e += blockDim.x) {
    int i, j;
    if (HERM) tri_index(e, i, j);
    else i = e % W, j = e / W;
    double2 acc = cmk(0, 0);
#pragma unroll 4
    for (int l = 0; l < W; ++l) {
      if (CA) cfmac(acc, A[i * W + l], B[j * W + l]);
      else cfma(acc, A[l * W + i], B[j * W + l]);
    }
    if (HERM && i == j) acc.y = 0.0;
    C[j * W + i] = acc;
    if (HERM && i < j) C[i * W + j] = cconj(acc);
  }
}

// The FP32 stage: eigenvectors of H to ~1e-6, made orthonormal to FP64 in V, and H <- V^H H V.
// The copy is shifted by the mean of the diagonal and scaled by the norm of what is left, so
// that FP32 resolves the eigenvalues' spread (A^H A of a nearly unitary A is close to I).
__device__ __forceinline__ void jac_fp32_stage(double2* H, double2* V, int W, double mean, double spread, double* red,
                                               double* rc, double2* rse, int* rp, int* rq, double2* s1,
                                               double2* s2) {
  const int WW = W * W;
  JacF2* Hf = reinterpret_cast<JacF2*>(V);
  JacF2* Vf = Hf + WW;
  const double sc = 1.0 / sqrt(spread);
  for (int e = threadIdx.x; e < WW; e += blockDim.x) {
    const double2 h = H[e];
    const bool d = (e % W) == (e / W);
    Hf[e].x = (float)((d ? h.x - mean : h.x) * sc);
    Hf[e].y = d ? 0.0f : (float)(h.y * sc);
    Vf[e].x = d ? 1.0f : 0.0f;
    Vf[e].y = 0.0f;
  }
  __syncthreads();
  // until a sweep rotates no pair above 1e-7 of the norm (a dozen sweeps at most: what is
  // left is the FP64 sweeps' work)
  for (int sweep = 0; sweep < 12; ++sweep) {
    const int rot = jac_sweep<float, JacF2>(Hf, Vf, W, 1.0e-14f, 1.0e-30f, reinterpret_cast<float*>(rc),
                                            reinterpret_cast<JacF2*>(rse), rp, rq);
    if (block_sum((double)rot, red) == 0.0) break;
  }
  for (int e = threadIdx.x; e < WW; e += blockDim.x) s1[e] = cmk((double)Vf[e].x, (double)Vf[e].y);
  __syncthreads();
  jac_mm<true, true>(V, s1, s1, W);      // G
  __syncthreads();
  jac_mm<false, true>(s2, V, V, W);      // G^2
  __syncthreads();
  for (int e = threadIdx.x; e < WW; e += blockDim.x) {
    const double2 g = V[e], g2 = s2[e];
    const double d = (e % W) == (e / W) ? 1.875 : 0.0;
    V[e] = cmk(d - 1.25 * g.x + 0.375 * g2.x, 0.375 * g2.y - 1.25 * g.y);
  }
  __syncthreads();
  jac_mm<false, false>(s2, s1, V, W);
  __syncthreads();
  jac_mm<false, false>(s1, H, s2, W);
  for (int e = threadIdx.x; e < WW; e += blockDim.x) V[e] = s2[e];
  __syncthreads();
  jac_mm<true, true>(H, s2, s1, W);
  __syncthreads();
}

__device__ __noinline__ static int cta_jacobi(double2* H, double2* V, int W, int max_sweeps, double* red,
                          double* rc, double2* rse, int* rp, int* rq, double skip_rel = 0.0,
                          double2* s1 = nullptr, double2* s2 = nullptr) {
  const int WW = W * W;
  // With the FP32 stage the last sweep starts from a part that may sit anywhere below the
  // plain criterion, where a solve from H itself overshoots it by orders: it is held to
  // 1e-33 instead, and its rotations below 1e-17.5 of the norm are left out.
  const double conv = s1 != nullptr && skip_rel == 0.0 ? 1.0e-33 : 1.0e-30;
  const double skip = s1 != nullptr && skip_rel == 0.0 ? 1.0e-35 : skip_rel;
  bool started = false;
  __syncthreads();
  for (int sweep = 0; sweep <= max_sweeps; ++sweep) {
    double off = 0.0, dia = 0.0, tr = 0.0;
    for (int e = threadIdx.x; e < WW; e += blockDim.x) {
      const double a = cabs2(H[e]);
      if ((e % W) != (e / W)) {
        off += a;
      } else {
        dia += a;
        tr += H[e].x;
      }
    }
    off = block_sum(off, red);
    dia = block_sum(dia, red);
    const double fro = off + dia;
    if (!started) {
      started = true;
      const double mean = block_sum(tr, red) / (double)W;
      const double spread = off + fmax(dia - (double)W * mean * mean, 0.0);
      // (a matrix whose off-diagonal part is at 1e-5 already is where the FP32 stage ends;
      // extreme or non-finite norms keep to FP64)
      if (s1 != nullptr && W >= 6 && off > 1.0e-10 * spread && off > 1.0e-26 * fro && spread > 1.0e-200 &&
          fro < 1.0e200) {
        jac_fp32_stage(H, V, W, mean, spread, red, rc, rse, rp, rq, s1, s2);
        --sweep;
        continue;
      }
      for (int e = threadIdx.x; e < WW; e += blockDim.x) V[e] = cmk((e % W) == (e / W) ? 1.0 : 0.0, 0.0);
      __syncthreads();
    }
    if (off <= conv * fro || off == 0.0) return sweep;
    if (sweep == max_sweeps) break;
    const int rotated = jac_sweep<double, double2>(H, V, W, skip * fro, 1.0e-290, rc, rse, rp, rq);
    if (skip > 0.0 && block_sum((double)rotated, red) == 0.0) return sweep + 1;
  }
  return -1;
}

// Unitary polar factor X (X^H X)^{-1/2} of an m x w matrix by the Newton-Schulz iteration
// X <- X (3 I - X^H X) / 2 on X itself: unitary to roundoff, its error that of the products times X's
// condition number.  (The eigenpairs of X^H X carry the square of that number: above ~1e4 what they
// give is not unitary, and no first-order correction is enough.)  The first step's coefficients scale
// the mean square of the singular values to 1, or the largest below 1 where it would come near sqrt(3);
// those below 1 grow by 1.5 a step, so this takes 1.7 log10(cond) + 4 steps or so of 6 m w^2 FMA.
// X (ldx) and Y (ldy) take turns, G is w x w scratch, red one double per thread.  Returns the one that
// holds the result, or null where `steps` were not enough (120: a singular value of 0) or X is not
// finite.  All threads call.
__device__ __noinline__ static double2* cta_polar_ns(double2* X, int ldx, double2* Y, int ldy, double2* G, int m, int w,
                                                     double* red, int steps = 120) {
  __shared__ int s_far;
  // G = X^H X in the first step, (I - X^H X) / 2 after it (X + X G rounds relative to what changes), and
  // whether |X^H X - I| is below 1e-8 / w elementwise: a step then leaves less than 1e-16
  auto gram = [&](bool first) -> bool {
    if (threadIdx.x == 0) s_far = 0;
    __syncthreads();
    bool far = false;
    for (int e = threadIdx.x; e < w * (w + 1) / 2; e += blockDim.x) {
      int i, j;
      tri_index(e, i, j);
      double2 g = cmk(0, 0);
      for (int l = 0; l < m; ++l) cfmac(g, X[(size_t)i * ldx + l], X[(size_t)j * ldx + l]);
      if (i == j) g.y = 0.0;
      const double d = (i == j ? 1.0 : 0.0) - g.x;
      far = far || !(fabs(d) + fabs(g.y) < 1.0e-8 / w);
      if (!first) g = cmk(0.5 * d, -0.5 * g.y);
      G[(size_t)j * w + i] = g;
      if (i < j) G[(size_t)i * w + j] = cconj(g);
    }
    if (far) s_far = 1;
    __syncthreads();
    return s_far == 0;
  };
  auto mean = [&]() {
    double t = 0.0;
    for (int j = 0; j < w; ++j) t += G[(size_t)j * w + j].x;
    return t / w;
  };
  for (int step = 0; step < steps; ++step) {
    bool done = gram(step == 0);
    double ca = 1.0, cb = 1.0;
    if (step == 0) {
      double mu = mean();
      if (!(mu > 0.0) || !isfinite(mu)) return nullptr;
      if (!(mu > 1.0e-60 && mu < 1.0e60)) {
        // far from 1: an exact scaling first
        int half;
        frexp(mu, &half);
        const double r = ldexp(1.0, -(half >> 1));
        __syncthreads();
        for (int e = threadIdx.x; e < m * w; e += blockDim.x) {
          double2& x = X[(size_t)(e / m) * ldx + e % m];
          x = cscale(x, r);
        }
        __syncthreads();
        gram(true);
        mu = mean();
      }
      // |X|_2^2 <= |X^H X|_1 <= the largest sum of |re| + |im| down a column
      double b = 0.0;
      for (int j = threadIdx.x; j < w; j += blockDim.x) {
        double t = 0.0;
        for (int i = 0; i < w; ++i) t += fabs(G[(size_t)j * w + i].x) + fabs(G[(size_t)j * w + i].y);
        b = fmax(b, t);
      }
      b = block_max(b, red);
      const double r = 1.0 / sqrt(b < 2.8 * mu ? mu : b);
      ca = 1.5 * r;
      cb = -0.5 * r * r * r;
      done = false;
    }
    for (int e = threadIdx.x; e < m * w; e += blockDim.x) {
      const int i = e % m, j = e / m;
      double2 y = cmk(0, 0);
      for (int l = 0; l < w; ++l) cfma(y, X[(size_t)l * ldx + i], G[(size_t)j * w + l]);
      const double2 x = X[(size_t)j * ldx + i];
      Y[(size_t)j * ldy + i] = cmk(fma(cb, y.x, ca * x.x), fma(cb, y.y, ca * x.y));
    }
    __syncthreads();
    double2* t = X;
    X = Y;
    Y = t;
    const int ld = ldx;
    ldx = ldy;
    ldy = ld;
    if (done) return X;
  }
  return nullptr;
}

}  // namespace w90g
