// Tensor-core M update for num_wann 33..128, pipelined: M(k,b) = U(k)^H M0(k,b) U(k+b).
//
// The two steps of k_tensor.cu -- Z(k,b) = U(k)^H M0(k,b) grouped by k, M(k,b) = Z(k,b) U(k')
// grouped by k' = k + b -- with one persistent CTA per SM and warp-specialised roles around a
// ring of K-step stages.  A stage holds one MMA K-step (16 real K: the real parts of 8 complex
// indices, then their imaginary parts) of 128 rows of A and of one chunk of B, all 7 digit
// planes of both: 28 KB + at most 14 KB, five stages in flight.
//
//   A           one bulk copy per stage from a digit image (k_oz_preslice3): step 1's of conj(M0),
//               sliced once per solve (the conjugate, so that both steps multiply by the same U:
//               conj(Z)^T = conj(M0)^T U), step 2's of Z, sliced between the steps.  (Eight warps of
//               the kernel slicing Z's rows for every column chunk took 3.1 ms a step at num_wann
//               128 on 512 k and 182 us at 48 on 216, against 1.5 ms and 95 us of step 1.)
//   B           one bulk copy per stage from the digit image of U(k), sliced once per update
//               (k_oz_slice_u) instead of once per 128-row tile, column chunk and K chunk;
//   MMA         one thread: 7 to 11 MMAs a stage (plane t of A against as many planes of B as
//               fit N = 256), committed to the stage's empty barrier;
//   epilogue    16 warps: exact recombination of the 7 diagonals in int64, FP64 stores, and in
//               step 2 the diagonal statistics and off-diagonal sums of the spread.
//
// What bounds it: the 448 accumulator columns of a chunk leave no room for a second set, so the
// epilogue and the next chunk's MMAs alternate -- a 128 x 64 x 16 stage is 28 digit-pair MMAs, and at
// num_wann 128 the tensor pipe is active 40 and 38 % of the two passes (L2 19 %, DRAM 23 %; the
// copies run at 5.5 TB/s and are not the limit).  Shapes follow num_wann itself, not a padded width: rows of consecutive blocks share
// a tile (B W / 128 tiles), K stops at the next multiple of 8 complex indices and the columns are
// cut into equal chunks of at most 32, so num_wann 48 costs 3/4 x 3/4 of 64 and not the same.
//
// Digits: 8 signed bits for num_wann <= 64, where 7 pairs of products up to 2^14 over K <= 128
// real terms stay below 2^24 in FP32: about 2^-53 of (row scale x column scale).  K = 256 keeps
// 8-bit digits from being exact, so wider problems use 7-bit ones (2^-49).
//
// Waits are bounded as in k_mupdate2.cu: a role that runs out records error 2 for its problem,
// the others stop, and the CTA drains its copies and MMAs before it leaves.
#include <algorithm>

#include "oz_mm.cuh"
#include "oz_pipe.cuh"

namespace w90g {

namespace {

constexpr int kPlaneA = kTileRows * 16 * 2;       // one digit plane of a stage's A
constexpr int kStageA = kS * kPlaneA;             // 28 KB
constexpr int kMaxN = 64;                         // real columns of a chunk
constexpr int kStage = kStageA + kS * kMaxN * 32; // with the largest B chunk
constexpr int kStages = (kDynBudget - 1024) / kStage;
static_assert(kStages >= 3, "shared memory for at least three stages");
constexpr size_t kSmem3 = (size_t)kStages * kStage + 1024;

// warps: 16 of the epilogue, the one whose first thread issues the copies, the one that issues MMAs
constexpr int kEpi3 = 16, kCopy3 = 16, kMma3 = 17, kThreads3 = 18 * 32, kEpiThreads3 = kEpi3 * 32;

// geometry of one problem
struct Geo3 {
  int ksteps;   // MMA K-steps: 8 complex indices each
  int nch;      // column chunks
  int cw;       // complex columns per chunk (a multiple of 8)
  int ntiles;   // 128-row tiles of a group
};
__host__ __device__ __forceinline__ Geo3 geo3(int W, int B) {
  Geo3 g;
  g.ksteps = (W + 7) / 8;
  g.nch = (W + 31) / 32;
  g.cw = ((W + g.nch - 1) / g.nch + 7) / 8 * 8;
  g.ntiles = (B * W + kTileRows - 1) / kTileRows;
  return g;
}
// bytes of one stage of B, and of a k's image
__host__ __device__ __forceinline__ size_t bstage3(const Geo3& g) { return (size_t)kS * (2 * g.cw) * 32; }
__host__ __device__ __forceinline__ size_t bimage3(const Geo3& g) { return bstage3(g) * g.ksteps * g.nch; }

// Step 2's image may hold the groups of one slab at a time: group g's slot there, or -1 if it is not of
// slab `slab`.  (One slab: g.)
__device__ __forceinline__ int zslot(const Problem& P, int g, int slab) {
  const int per = (P.K + P.zs_slabs - 1) / P.zs_slabs;
  return g / per == slab ? g - slab * per : -1;
}

// the 7 digit planes of 8 values with scale exponent ex, 8- or 7-bit digits
template <bool EIGHT>
__device__ __forceinline__ void slice3(uint32_t (&w)[kS][4], const double (&v)[8], int ex) {
  if (EIGHT) slice_run8_h(w, v, ex);
  else pack_digits7(w, v, ex, false);
}

// C from the 7 diagonal accumulators and the exponents' sum e.  |D_d| < 2^24 are exact integers
// in FP32; the sums below stay within 2^63 for any operands.  8-bit digits: S = D_0..D_3 at
// 2^(41-8d) plus (D_4 2^16 + D_5 2^8 + D_6) / 2^7 rounded, C = S 2^(e-55) (the digit pairs left
// out weigh ~2^(e-53)).  7-bit digits: S = (sum D_d 2^(7(6-d))) / 2 rounded, C = S 2^(e-55).
template <bool EIGHT>
__device__ __forceinline__ double recombine3(const uint32_t* dd, int stride, int e) {
  long long d[kS];
#pragma unroll
  for (int i = 0; i < kS; ++i) d[i] = (long long)__float2int_rn(__uint_as_float(dd[i * stride]));
  long long S;
  if (EIGHT) {
    const long long hi = d[0] * (1LL << 41) + d[1] * (1LL << 33) + d[2] * (1LL << 25) + d[3] * (1LL << 17);
    const long long lo = d[4] * (1LL << 16) + d[5] * 256 + d[6];
    S = hi + ((lo + 64) >> 7);
  } else {
    const long long hi = d[0] * (1LL << 21) + d[1] * (1LL << 14) + d[2] * 128 + d[3];
    const long long lo = d[4] * (1LL << 14) + d[5] * 128 + d[6];
    S = hi * (1LL << 20) + ((lo + 1) >> 1);
  }
  return int64_scaled_to_double(S, e - 55);
}

__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void arrive_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
               :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}

}  // namespace

// Work items: (group, tile), group-major, `tmax` tiles per group (the widest problem's); a
// persistent grid walks them.  EIGHT: every problem of the launch has num_wann <= 64.
template <int STEP, bool EIGHT>
__global__ void __launch_bounds__(kThreads3, 1)
    k_oz_mupdate3(const Problem* __restrict__ probs, WorkMap wm, int which, int ngroups, int tmax, int slab) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t a_full[kStages], a_empty[kStages];
  __shared__ __align__(8) uint64_t acc_full, acc_empty, drain_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_bad;
  __shared__ int s_bad_prob, s_eflag;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == kMma3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&a_full[s], 1u);   // the issuing thread's arrival with the copies' bytes
      mbar_init(&a_empty[s], 1u);
    }
    mbar_init(&acc_full, 1u);
    mbar_init(&acc_empty, (uint32_t)kEpiThreads3);
    mbar_init(&drain_bar, 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_bad = 0;
    s_bad_prob = -1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const int nitems = ngroups * tmax;

  auto fail = [&](int p) {
    if (!s_bad) {
      s_bad_prob = p;
      s_bad = 1;
    }
  };

  if (warp == kCopy3) {
    // =========================== copies ===========================
    if (lane == 0) {
      int sseq = 0;
      uint32_t inflight = 0, par = 0;   // slots with a copy issued, and its parity
      bool ok = true;
      for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        int g;
        const int p = locate(wm, item / tmax, g), tile = item % tmax;
        const Problem& P = probs[p];
        const Geo3 G = geo3(P.W, P.B);
        if (tile >= G.ntiles || !group_active(P, which) || (STEP == 2 && zslot(P, g, slab) < 0)) continue;
        const uint32_t bst = (uint32_t)bstage3(G);
        const unsigned char* bimg = P.ub2 + (size_t)g * bimage3(G);
        const unsigned char* aimg =
            (STEP == 1 ? P.m0s : P.zs) +
            ((size_t)(STEP == 1 ? g : zslot(P, g, slab)) * G.ntiles + tile) * G.ksteps * (size_t)kStageA;
        for (int nc = 0; nc < G.nch && ok; ++nc)
          for (int ks = 0; ks < G.ksteps; ++ks) {
            const int s = sseq % kStages;
            const uint32_t use = (uint32_t)(sseq / kStages);
            // (the first use of each stage slot needs no wait)
            if (use > 0 && !mbar_wait_role(smem_u32(&a_empty[s]), (use & 1) ^ 1, &s_bad)) {
              fail(p);
              ok = false;
              break;
            }
            unsigned char* dA = base + (size_t)s * kStage;
            arrive_expect(&a_full[s], bst + (uint32_t)kStageA);
            bulk_copy(dA + kStageA, bimg + ((size_t)nc * G.ksteps + ks) * bst, bst, &a_full[s]);
            bulk_copy(dA, aimg + (size_t)ks * kStageA, kStageA, &a_full[s]);
            inflight |= 1u << s;
            par = (par & ~(1u << s)) | ((use & 1) << s);
            ++sseq;
          }
      }
      // drain: the last copy into each slot must land before the CTA frees its shared memory
      for (int s = 0; s < kStages; ++s)
        if (inflight & (1u << s)) mbar_drain(smem_u32(&a_full[s]), (par >> s) & 1);
    }
  } else if (warp == kMma3) {
    // =========================== MMA issue ===========================
    if (lane == 0) {
      int sseq = 0, useq = 0;
      bool issued = false, ok = true;
      for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        int g;
        const int p = locate(wm, item / tmax, g), tile = item % tmax;
        const Problem& P = probs[p];
        const Geo3 G = geo3(P.W, P.B);
        if (tile >= G.ntiles || !group_active(P, which) || (STEP == 2 && zslot(P, g, slab) < 0)) continue;
        const int N = 2 * G.cw, ppm = 256 / N;
        for (int nc = 0; nc < G.nch && ok; ++nc) {
          if (useq > 0 && !mbar_wait_role(smem_u32(&acc_empty), (uint32_t)(useq - 1) & 1, &s_bad)) {
            fail(p);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          for (int ks = 0; ks < G.ksteps; ++ks) {
            const int s = sseq % kStages;
            if (!mbar_wait_role(smem_u32(&a_full[s]), (uint32_t)(sseq / kStages) & 1, &s_bad)) {
              fail(p);
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a0 = smem_u32(base + (size_t)s * kStage);
            const uint64_t da = smem_desc(a0, 128, 256), db = smem_desc(a0 + kStageA, 128, 256);
#pragma unroll
            for (int t = 0; t < kS; ++t)
              for (int u0 = 0; u0 + t < kS; u0 += ppm) {
                // plane t of A against planes u0 .. u0 + n - 1 of B (consecutive row groups of
                // one K-major operand): diagonals t + u0 .., N = n planes <= 256
                const int n = min(kS - t - u0, ppm);
                const uint64_t ad = da + (uint64_t)((t * kPlaneA) >> 4);
                const uint64_t bd = db + (uint64_t)((u0 * N * 32) >> 4);
                const uint32_t accf = (ks == 0 && t == 0) ? 0u : 1u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    :: "r"(tmem + (uint32_t)((t + u0) * N)), "l"(ad), "l"(bd), "r"(idesc_f16(n * N)), "r"(accf)
                    : "memory");
              }
            issued = true;
            mma_commit(&a_empty[s]);
            ++sseq;
          }
          if (!ok) break;
          mma_commit(&acc_full);
          ++useq;
        }
      }
      if (issued) {
        mma_commit(&drain_bar);
        mbar_drain(smem_u32(&drain_bar), 0);
      }
    }
  } else {
    // =========================== epilogue ===========================
    const int wq = warp & 3, cg = warp >> 2;            // TMEM lane quarter, column group
    const int r = wq * 32 + lane;                       // tile row = TMEM lane
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    int useq = 0;
    bool ok = true;
    // one thread waits, the others at the epilogue's named barrier
    auto await = [&](uint64_t* bar, uint32_t parity, int p) -> bool {
      if (tid == 0) {
        const bool o = mbar_wait_role(smem_u32(bar), parity, &s_bad);
        if (!o) fail(p);
        s_eflag = o ? 0 : 1;
      }
      bar_named(2, kEpiThreads3);
      const bool o = s_eflag == 0;
      bar_named(2, kEpiThreads3);
      return o;
    };
    for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
      int g;
      const int p = locate(wm, item / tmax, g), tile = item % tmax;
      const Problem& P = probs[p];
      const int W = P.W, WW = W * W;
      const Geo3 G = geo3(W, P.B);
      if (tile >= G.ntiles || !group_active(P, which) || (STEP == 2 && zslot(P, g, slab) < 0)) continue;
      const int cur = P.st->cur, N = 2 * G.cw, cpg = G.cw / 4;
      const int row = tile * kTileRows + r;
      const bool valid = row < P.B * W;
      const int bi = row / W, rr = row % W;
      size_t kb = 0;
      if (STEP == 1) {
        kb = (size_t)g * P.B + bi;
      } else if (valid) {
        kb = (size_t)P.inv_nnlist[(size_t)g * P.B + bi];
      }
      const int erow = (STEP == 1 ? P.m0s_exp : P.zs_exp)[((size_t)g * G.ntiles + tile) * kTileRows + r];
      double2* dst = (STEP == 1 ? P.tbuf : P.M[cur ^ 1]) + kb * WW + rr;
      const int* ecol = P.ub2_exp + (size_t)g * W;
      double od = 0.0;   // step 2: |M_mn|^2 off the diagonal, this row and column group
      for (int nc = 0; nc < G.nch; ++nc) {
        if (!await(&acc_full, (uint32_t)useq & 1, p)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        double dre = 0.0, dim = 0.0;
        bool has_diag = false;
#pragma unroll 1
        for (int j0 = cg * cpg; j0 < (cg + 1) * cpg; j0 += 2) {
          uint32_t q[kDiag][2], s2[kDiag][2];
#pragma unroll
          for (int d = 0; d < kDiag; ++d) {
            const uint32_t ta = tmem + lane_base + (uint32_t)(d * N + j0);
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
                         : "=r"(q[d][0]), "=r"(q[d][1]) : "r"(ta));
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
                         : "=r"(s2[d][0]), "=r"(s2[d][1]) : "r"(ta + (uint32_t)G.cw));
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int c = nc * G.cw + j0 + j;   // complex output column
            if (valid && c < W) {
              const int e = erow + ecol[c];
              const double re = recombine3<EIGHT>(&q[0][j], 2, e);
              double im = recombine3<EIGHT>(&s2[0][j], 2, e);
              if (STEP == 1) im = -im;          // the product is conj(Z)
              dst[(size_t)c * W] = make_double2(re, im);
              if (STEP == 2) {
                if (c == rr) {
                  dre = re;
                  dim = im;
                  has_diag = true;
                } else {
                  od = fma(re, re, od);
                  od = fma(im, im, od);
                }
              }
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(&acc_empty);
        if (has_diag) {
          P.diag_ln[kb * W + rr] = guided_ln(P, kb * W + rr, make_double2(dre, dim));
          P.diag_abs2[kb * W + rr] = dre * dre + dim * dim;
        }
        ++useq;
      }
      if (STEP == 2 && ok) {
        // The off-diagonal sums of the warp's 32 rows, which lie in one block or two (num_wann >
        // 32): piece (row / 32 - first row of the block / 32) of the block and column group cg.
        // The warp with a block's last row clears the pieces its position leaves unused.
        const int row0 = tile * kTileRows + wq * 32, b0 = row0 / W;
        for (int b = b0; b <= b0 + 1 && b < P.B; ++b) {
          double x = valid && bi == b ? od : 0.0;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          const int first = b * W / 32, last = (b * W + W - 1) / 32;
          if (row0 + 31 < b * W) break;
          if (lane == 0) {
            double* dp = P.odpart + (size_t)P.inv_nnlist[(size_t)g * P.B + b] * P.odn + cg;
            dp[(row0 / 32 - first) * 4] = x;
            if (row0 / 32 == last)
              for (int i = last - first + 1; i < P.odn / 4; ++i) dp[i * 4] = 0.0;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMma3) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
  }
  if (tid == 0 && s_bad && s_bad_prob >= 0) {
    CtrlState* st = probs[s_bad_prob].st;
    st->error = 2;
    st->done = 1;
  }
}

// The digit image of U(k) of the update (buffer cur ^ 1) for both steps: per column chunk and
// K-step the 7 planes of the B^T stage -- rows [N re | N im], K [8 re | 8 im] of the embedding
// [[B_r, B_i], [-B_i, B_r]] -- and the column exponents.  A thread slices one part of 8 consecutive
// m of a column and writes 16-byte core rows.  One CTA (256 threads) per k.
template <bool EIGHT>
__global__ void __launch_bounds__(256) k_oz_slice_u(const Problem* __restrict__ probs, WorkMap wm, int which) {
  __shared__ int s_exp[128];
  int g;
  const int p = locate(wm, blockIdx.x, g);
  const Problem& P = probs[p];
  if (!group_active(P, which)) return;
  const int W = P.W, tid = threadIdx.x;
  const Geo3 G = geo3(W, P.B);
  const double2* U = P.U[P.st->cur ^ 1] + (size_t)g * W * W;
  unsigned char* img = P.ub2 + (size_t)g * bimage3(G);
  const size_t bst = bstage3(G);
  const int pl = 2 * G.cw * 32;
  // column scales: 8 lanes per column
  for (int c0 = tid / 8; c0 < (W + 31) / 32 * 32; c0 += 32) {
    unsigned long long mx = 0ull;
    if (c0 < W)
      for (int m = tid % 8; m < W; m += 8) {
        const double2 u = U[(size_t)c0 * W + m];
        mx = max(mx, max(abs_bits(u.x), abs_bits(u.y)));
      }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
      mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)mx, o));
    if (tid % 8 == 0 && c0 < W) {
      s_exp[c0] = exp_above_bits(mx);
      P.ub2_exp[(size_t)g * W + c0] = s_exp[c0];
    }
  }
  __syncthreads();
  // items: (column of a chunk, part, K-step, chunk), columns fastest: consecutive threads write
  // consecutive core rows
  const int items = G.cw * 2 * G.ksteps * G.nch;
  for (int it = tid; it < items; it += 256) {
    const int cl = it % G.cw, part = (it / G.cw) % 2, ks = (it / (2 * G.cw)) % G.ksteps,
              nc = it / (2 * G.cw * G.ksteps);
    const int c = nc * G.cw + cl;
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = ks * 8 + i;
      v[i] = (c < W && m < W) ? ((const double*)(U + (size_t)c * W + m))[part] : 0.0;
    }
    uint32_t w[kS][4];
    slice3<EIGHT>(w, v, c < W ? s_exp[c] : 0);
    unsigned char* st = img + ((size_t)nc * G.ksteps + ks) * bst;
    // B_r: (N re, K re) and (N im, K im);  B_i: (N im, K re), and negated (N re, K im)
    const uint32_t o1 = stage_off(part == 0 ? cl : G.cw + cl, 0);
    const uint32_t o2 = stage_off(part == 0 ? G.cw + cl : cl, 8);
#pragma unroll
    for (int t = 0; t < kS; ++t) {
      *(uint4*)(st + (size_t)t * pl + o1) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
      *(uint4*)(st + (size_t)t * pl + o2) =
          part == 0 ? make_uint4(w[t][0], w[t][1], w[t][2], w[t][3])
                    : make_uint4(f16x2_neg(w[t][0]), f16x2_neg(w[t][1]), f16x2_neg(w[t][2]), f16x2_neg(w[t][3]));
    }
  }
}

// The A operands' digit planes in the stage layout, with the row exponents: STEP 1 conj(M0)^T's rows
// (k, b, n), once per solve; STEP 2 the rows of Z(k,b) of group k' = nnlist(k,b), between the steps.
// One CTA (256 threads) per (group, tile).
template <int STEP, bool EIGHT>
__global__ void __launch_bounds__(256) k_oz_preslice3(const Problem* __restrict__ probs, WorkMap wm, int tmax,
                                                      int which, int slab) {
  __shared__ int s_rowexp[kTileRows];
  int g;
  const int p = locate(wm, blockIdx.x / tmax, g), tile = blockIdx.x % tmax;
  const Problem& P = probs[p];
  const int W = P.W, WW = W * W, tid = threadIdx.x;
  const Geo3 G = geo3(W, P.B);
  const int slot = STEP == 1 ? g : zslot(P, g, slab);
  if (tile >= G.ntiles || (STEP == 2 && (slot < 0 || !group_active(P, which)))) return;
  unsigned char* img = STEP == 1 ? P.m0s : P.zs;
  int* exps = STEP == 1 ? P.m0s_exp : P.zs_exp;
  auto row_of = [&](int row) -> const double2* {
    if (row >= P.B * W) return nullptr;
    const size_t gb = (size_t)g * P.B + row / W;
    return (STEP == 1 ? P.M0 + gb * WW : P.tbuf + (size_t)P.inv_nnlist[gb] * WW) + (size_t)(row % W) * W;
  };
  const int r = tid >> 1;
  const double2* src = row_of(tile * kTileRows + r);
  {
    unsigned long long mx = 0ull;
    if (src)
#pragma unroll 8
      for (int m = tid & 1; m < W; m += 2) mx = max(mx, max(abs_bits(src[m].x), abs_bits(src[m].y)));
    mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)mx, 1));
    if ((tid & 1) == 0) {
      s_rowexp[r] = exp_above_bits(mx);
      exps[((size_t)g * G.ntiles + tile) * kTileRows + r] = s_rowexp[r];
    }
  }
  __syncthreads();
  const int rs = tid % kTileRows, part = tid / kTileRows;
  const double2* srow = row_of(tile * kTileRows + rs);
  const double* s2 = srow ? (const double*)srow + part : nullptr;
  for (int ks = 0; ks < G.ksteps; ++ks) {
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = ks * 8 + i;
      const double x = (s2 && m < W) ? s2[2 * m] : 0.0;
      v[i] = STEP == 1 && part ? -x : x;
    }
    uint32_t w[kS][4];
    slice3<EIGHT>(w, v, s_rowexp[rs]);
    unsigned char* dst = img + (((size_t)slot * G.ntiles + tile) * G.ksteps + ks) * (size_t)kStageA;
    const uint32_t o = stage_off(rs, 8 * part);
#pragma unroll
    for (int t = 0; t < kS; ++t)
      *(uint4*)(dst + (size_t)t * kPlaneA + o) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
  }
}

// ---- host side ----------------------------------------------------------------------

// bytes of a problem's digit images and exponents: m0s (and zs), m0s_exp (and zs_exp), ub2, ub2_exp
void oz3_bytes(int W, int K, int B, size_t out[4]) {
  const Geo3 G = geo3(W, B);
  out[0] = (size_t)K * G.ntiles * G.ksteps * kStageA;
  out[1] = (size_t)K * G.ntiles * kTileRows * 4;
  out[2] = (size_t)K * bimage3(G);
  out[3] = (size_t)K * W * 4;
}

int oz3_tiles(int W, int B) { return geo3(W, B).ntiles; }

cudaError_t oz3_set_attributes(int wp) {
  const int sm = (int)kSmem3;
  cudaError_t e;
  if (wp <= 64) {
    e = cudaFuncSetAttribute(k_oz_mupdate3<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_oz_mupdate3<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  } else {
    e = cudaFuncSetAttribute(k_oz_mupdate3<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_oz_mupdate3<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  }
  return e;
}

template <bool EIGHT>
static void oz3_launch_e(const Problem* probs, WorkMap wm, int which, int ngroups, int tmax, int slabs,
                         cudaStream_t s) {
  const int grid = std::min(ngroups * tmax, sm_count());
  k_oz_slice_u<EIGHT><<<ngroups, 256, 0, s>>>(probs, wm, which);
  k_oz_mupdate3<1, EIGHT><<<grid, kThreads3, kSmem3, s>>>(probs, wm, which, ngroups, tmax, 0);
  for (int i = 0; i < slabs; ++i) {
    k_oz_preslice3<2, EIGHT><<<ngroups * tmax, 256, 0, s>>>(probs, wm, tmax, which, i);
    k_oz_mupdate3<2, EIGHT><<<grid, kThreads3, kSmem3, s>>>(probs, wm, which, ngroups, tmax, i);
  }
}

// the whole update (four launches, two more for each slab of Z's image after the first) of the ngroups work items of wm; wp: the widest problem's
// padded width, 64 or 128; tmax: the largest tile count of a group
cudaError_t oz3_launch(int wp, const Problem* probs, WorkMap wm, int which, int ngroups, int tmax, int slabs,
                       cudaStream_t s) {
  if (wp <= 64) oz3_launch_e<true>(probs, wm, which, ngroups, tmax, slabs, s);
  else oz3_launch_e<false>(probs, wm, which, ngroups, tmax, slabs, s);
  return cudaGetLastError();
}

cudaError_t oz3_preslice_launch(int wp, const Problem* probs, WorkMap wm, int ngroups, int tmax, cudaStream_t s) {
  if (wp <= 64) k_oz_preslice3<1, true><<<ngroups * tmax, 256, 0, s>>>(probs, wm, tmax, 0, 0);
  else k_oz_preslice3<1, false><<<ngroups * tmax, 256, 0, s>>>(probs, wm, tmax, 0, 0);
  return cudaGetLastError();
}

}  // namespace w90g
