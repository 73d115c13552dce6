// W x W complex products on the tcgen05 tensor cores through exact digit slicing, at 56-bit
// operand precision, as CTA-wide device functions (256 threads): C = A B from FP64 matrices in
// shared or global memory, accurate to ~2^-56 of (row scale x column scale) -- below FP64 GEMM
// roundoff.  Two product forms:
//   widths <= 64: [C_r; C_i] = [[A_r, -A_i], [A_i, A_r]] [B_r; B_i], 7 signed 8-bit digits
//     (FP16 operands), 28 digit pairs (oz_cmm2);
//   widths 65..128: [C_r C_i] = [A_r A_i] [[B_r, B_i], [-B_i, B_r]], 8 signed 7-bit digits, 36
//     digit pairs (oz_cmm; K = 256 keeps 8-bit digits from being exact).
// A product puts the rows of its A operand on the 128 TMEM lanes; when fewer rows are real,
// the digit slices of A are stored row-blocks apart in one region: the MMA reading slice t sees
// slices t+1.. in the rows beyond, which only feed accumulator rows nobody reads.
#pragma once
#include <type_traits>

#include "oz.cuh"

namespace w90g {

namespace {

constexpr int kS8 = 8;   // digits per operand in this kernel

template <int WP>
struct ExpSmem {
  using L = TileSmem<WP>;
  static constexpr int CW = L::CW, KC = L::KC, NC = L::NC, NCH = L::NCH;
  static constexpr int A_ROWS = (kS8 - 1) * WP + kTileRows;      // overlapped slices
  static constexpr int A_SLICE = WP * KC * 2;                     // bytes between slices
  static constexpr int A_BYTES = A_ROWS * KC * 2;
  static constexpr int B_BYTES = NC * KC * 2;                     // per slice
  static constexpr int TMEM_COLS = (kS8 * NC <= 128) ? 128 : ((kS8 * NC <= 256) ? 256 : 512);
  static constexpr size_t REGION = (size_t)A_BYTES + (size_t)kS8 * B_BYTES;
  static constexpr size_t BYTES = REGION + 1024;
};

// per-CTA state of the tensor product
struct OzCtx {
  unsigned char* sA;
  unsigned char* sB;
  uint32_t tmem;
  uint32_t mbar;
  uint32_t phase;
  int* rowexp;   // [WP]
  int* colexp;   // [WP]
  int* bad;
};

// Scale records of the chain's matrices: for every row and column the key of its largest
// |re| or |im| (0 for none, else the biased exponent + 1; the exponent above that value
// is key - 1023, as exp_above_bits gives it).  The epilogue that writes a matrix forms its
// record with shared-memory maxima, so that the products reading the matrix take their
// scales from shared memory instead of a pass over the operand.
__device__ __forceinline__ unsigned scale_key(double re, double im) {
  const unsigned long long ab = max(abs_bits(re), abs_bits(im));
  return ab ? (unsigned)(ab >> 52) + 1u : 0u;
}
// (two of these scales and a product's 63 digit bits stay inside FP64's exponents)
constexpr int kExpMin = -480;
__device__ __forceinline__ int key_exp(unsigned key) { return key ? max((int)key - 1023, kExpMin) : 0; }

struct Rec {
  unsigned* row;
  unsigned* col;
};

// Scales that the digits carry through two products in a row: outside of this range a scale may
// leave FP64's exponents on the way, and the keys of NaN and infinities (2048) read as 2^1025.
// k_oz_rotate, k_oz_ufinal and k_oz_polar leave such operands to FP64.
constexpr int kExpSafe = 290;
__device__ __forceinline__ bool exp_wild(int e) { return e > kExpSafe || e < -kExpSafe; }
// this thread's share of n keys
__device__ __forceinline__ bool keys_wild(const unsigned* keys, int n) {
  bool w = false;
  for (int i = threadIdx.x; i < n; i += blockDim.x) w = w || exp_wild(key_exp(keys[i]));
  return w;
}

// Power-of-two scales of a product: the exponent above the largest |re| or |im| of every
// row of A and every column of B, from the operands' records where given (arow / bcol),
// else by a pass over them.  The 2 WP rows / columns share the CTA's 256 threads (TPI
// consecutive lanes each, then a max across those lanes), so each thread reads W / TPI
// entries instead of W; the maximum does not depend on the order.
template <int WP>
__device__ __forceinline__ void ab_exponents(OzCtx& cx, const double2* A, const unsigned* arow,
                                             const double2* B, const unsigned* bcol, int W) {
  constexpr int ITEMS = 2 * WP;
  constexpr int TPI = ITEMS >= 256 ? 1 : (256 / ITEMS > 32 ? 32 : 256 / ITEMS);
  if (arow != nullptr && bcol != nullptr) {
    for (int i = threadIdx.x; i < ITEMS; i += blockDim.x)
      (i < WP ? cx.rowexp : cx.colexp)[i % WP] = key_exp(i < WP ? arow[i] : bcol[i - WP]);
    return;
  }
  for (int base = 0; base < ITEMS * TPI; base += blockDim.x) {
    const int gi = base + (int)threadIdx.x;
    const int idx = gi / TPI, sub = gi % TPI;
    const int r = idx % WP;
    const bool row_of_a = idx < WP;
    const unsigned* rec = row_of_a ? arow : bcol;
    unsigned long long mx = 0ull;
    if (idx < ITEMS && r < W && rec == nullptr) {
      // eight independent loads per round (the matrices may sit in L2), then the max
      for (int l0 = sub; l0 < W; l0 += 8 * TPI) {
        double2 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int l = l0 + i * TPI;
          v[i] = (l < W) ? (row_of_a ? A[(size_t)l * W + r] : B[(size_t)r * W + l]) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) mx = max(mx, max(abs_bits(v[i].x), abs_bits(v[i].y)));
      }
    }
#pragma unroll
    for (int o = 1; o < TPI; o <<= 1)
      mx = max(mx, (unsigned long long)__shfl_xor_sync(0xffffffffu, (long long)mx, o));
    if (idx < ITEMS && sub == 0)
      (row_of_a ? cx.rowexp : cx.colexp)[r] = rec != nullptr ? key_exp(rec[r]) : max(exp_above_bits(mx), kExpMin);
  }
}

// Where a product's result goes: `out`, made exactly Hermitian (sym = +1) or
// anti-Hermitian (sym = -1) from its upper triangle as the FP64 path's structured products
// produce it, or plain (sym = 0) with an elementwise term added (Add), and its scale
// record formed in `rec` (rec.row == nullptr: none).
struct Epi {
  double2* out;
  int sym;
  Rec rec;
};

// no elementwise term
struct NoAdd {
  static constexpr bool kActive = false;
  __device__ double2 operator()(int) const { return make_double2(0.0, 0.0); }
};

__device__ __forceinline__ void rec_clear(const Rec& r, int n) {
  if (r.row != nullptr)
    for (int i = threadIdx.x; i < 2 * n; i += blockDim.x) (i < n ? r.row : r.col)[i % n] = 0u;
}

// Adds the key of v (at row i, column j) to the record (shared-memory maxima).  (A warp
// maximum before one atomic per distinct index measured slower than these atomics.)
__device__ __forceinline__ void rec_add(const Rec& r, int i, int j, double2 v) {
  if (r.row != nullptr) {
    const unsigned key = scale_key(v.x, v.y);
    if (key) {
      atomicMax(r.row + i, key);
      atomicMax(r.col + j, key);
    }
  }
}

// Applies an Epi to a product already in C (the product forms whose epilogue does not
// apply it directly): out[e] from C[e] (its upper triangle when sym != 0) plus add(e),
// and the record.  out may be C.  All threads call.
template <int WP, class Add>
__device__ void epi_apply(const double2* C, const Epi& ep, const Add& add, int W) {
  if (ep.sym == 0 && !Add::kActive && ep.rec.row == nullptr && ep.out == C) return;
  rec_clear(ep.rec, WP);
  __syncthreads();
#pragma unroll 4
  for (int e = threadIdx.x; e < W * W; e += blockDim.x) {
    const int i = e % W, j = e / W;
    double2 v;
    bool write = ep.out != C || Add::kActive;
    if (ep.sym != 0 && i > j) {
      const double2 u = C[(size_t)i * W + j];
      v = cmk(ep.sym * u.x, -ep.sym * u.y);
      write = true;
    } else if (ep.sym != 0 && i == j) {
      const double2 d = C[e];
      v = (ep.sym > 0) ? cmk(d.x, 0.0) : cmk(0.0, d.y);
      write = true;
    } else {
      v = C[e];
    }
    if (Add::kActive) v = cadd(v, add(e));
    if (write) ep.out[e] = v;
    rec_add(ep.rec, i, j, v);
  }
  __syncthreads();
}

// Part (0 re, 1 im) of 8 values base[(m0 + i) * stride], i < 8 (zero where m0 + i >= W or
// !valid): the operand run a thread slices.
__device__ __forceinline__ void load_run8(double (&v)[8], const double2* base, size_t stride, int m0, int W,
                                          bool valid, int part) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + i;
    v[i] = 0.0;
    if (valid && m < W) v[i] = ((const double*)(base + (size_t)m * stride))[part];
  }
}

// C = A B for W x W complex column-major matrices (generic pointers; C must not alias
// A or B), then the Epi applied from C.  All threads call; returns false (uniformly) if
// an MMA wait timed out.
template <int WP, class Add>
__device__ bool oz_cmm(OzCtx& cx, double2* C, const double2* A, const unsigned* arow, const double2* B,
                       const unsigned* bcol, int W, const Epi& ep, const Add& add) {
  using E = ExpSmem<WP>;
  constexpr int CW = E::CW, KC = E::KC, NC = E::NC, NCH = E::NCH;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // ---- power-of-two scales: rows of A, columns of B (over re and im parts)
  ab_exponents<WP>(cx, A, arow, B, bcol, W);
  __syncthreads();
  bool ok = true;
  for (int nc = 0; nc < NCH && ok; ++nc) {
    for (int kc = 0; kc < NCH && ok; ++kc) {
      // ---- A chunk: rows r < WP, complex K index l < CW -> real columns l, l + CW.  A thread
      // slices one part of 8 consecutive l of a row into a 16-byte core row per digit plane.
      constexpr int LG = CW / 8;
      for (int it = tid; it < WP * LG * 2; it += 256) {
        const int r = it % WP, lg = (it / WP) % LG, part = it / (WP * LG);
        double v[8];
        load_run8(v, A + r, (size_t)W, kc * CW + lg * 8, W, r < W, part);
        uint32_t w[kS8][4];
        pack_digits8(w, v, cx.rowexp[r]);
        const uint32_t o = kmaj_off(r, part * CW + lg * 8, KC);
#pragma unroll
        for (int t = 0; t < kS8; ++t)
          *(uint4*)(cx.sA + (size_t)t * E::A_SLICE + o) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
      }
      // ---- B chunk, embedded [[B_r, B_i], [-B_i, B_r]] stored as B^T (K-major): row = real N
      // index (c | c + CW), column = real K index (l | l + CW); each part goes to two places
      for (int it = tid; it < CW * LG * 2; it += 256) {
        const int c = it % CW, lg = (it / CW) % LG, part = it / (CW * LG);
        const int cc = nc * CW + c;
        double v[8];
        load_run8(v, B + (size_t)cc * W, (size_t)1, kc * CW + lg * 8, W, cc < W, part);
        uint32_t w[kS8][4];
        pack_digits8(w, v, cx.colexp[cc < WP ? cc : 0]);
        // B_r: (K re, N re), (K im, N im);  B_i: (K re, N im), negated (K im, N re)
        const uint32_t o1 = kmaj_off(part == 0 ? c : c + CW, lg * 8, KC);
        const uint32_t o2 = kmaj_off(part == 0 ? c + CW : c, CW + lg * 8, KC);
#pragma unroll
        for (int t = 0; t < kS8; ++t) {
          unsigned char* sb = cx.sB + (size_t)t * E::B_BYTES;
          *(uint4*)(sb + o1) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
          *(uint4*)(sb + o2) = part == 0 ? make_uint4(w[t][0], w[t][1], w[t][2], w[t][3])
                                         : make_uint4(f16x2_neg(w[t][0]), f16x2_neg(w[t][1]), f16x2_neg(w[t][2]),
                                                      f16x2_neg(w[t][3]));
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // descriptors from a base plus offsets / 16 (shared-memory addresses stay below
        // 2^18); B's digit planes follow one another as row groups of one K-major operand
        // and diagonal d's accumulator columns follow d - 1's, so slice t of A against
        // planes u0 .. u0 + n - 1 of B is one MMA with N = n NC (<= 256)
        const uint64_t da = smem_desc(smem_u32(cx.sA), 128, (KC / 8) * 128);
        const uint64_t db = smem_desc(smem_u32(cx.sB), 128, (KC / 8) * 128);
        constexpr int PPM = 256 / NC;
#pragma unroll
        for (int t = 0; t < kS8; ++t) {
#pragma unroll
          for (int u0 = 0; u0 + t <= kS8 - 1; u0 += PPM) {
            const int n = (kS8 - t - u0) < PPM ? (kS8 - t - u0) : PPM;
            const uint32_t dtm = cx.tmem + (uint32_t)((t + u0) * NC);
            const bool first_pair = (kc == 0) && (t == 0);
#pragma unroll
            for (int ks = 0; ks < KC / 16; ++ks) {
              const uint64_t ad = da + (uint64_t)(((size_t)t * E::A_SLICE + ks * 256) >> 4);
              const uint64_t bd = db + (uint64_t)(((size_t)u0 * E::B_BYTES + ks * 256) >> 4);
              const uint32_t acc = (first_pair && ks == 0) ? 0u : 1u;
              asm volatile(
                  "{\n\t.reg .pred p;\n\t"
                  "setp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                  :: "r"(dtm), "l"(ad), "l"(bd), "r"(idesc_f16(n * NC)), "r"(acc)
                  : "memory");
            }
          }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                     :: "r"(cx.mbar) : "memory");
      }
      // one thread waits for the commit (the others wait at the CTA barrier, issuing nothing)
      if (tid == 0 && !mbar_wait(cx.mbar, cx.phase)) {
        // record the error; drain the MMAs before tensor memory or the operands are reused
        *cx.bad = 1;
        mbar_drain(cx.mbar, cx.phase);
      }
      cx.phase ^= 1u;
      __syncthreads();
      ok = (*cx.bad == 0);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (!ok) break;
    // C(r, c) = (sum_d D_d 2^(7(7-d))) 2^(rowexp + colexp - 63)
    auto recombine = [&](const uint32_t* dr, const uint32_t* di, int stride, int r, int c) {
      const int sc = cx.rowexp[r] + cx.colexp[c] - 63;
      C[(size_t)c * W + r] = make_double2(recombine8x7(dr, stride, sc), recombine8x7(di, stride, sc));
    };
    const int wq = warp & 3, half = warp >> 2;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    const int jbeg = half * (CW / 2), jend = jbeg + CW / 2;
    // ---- direct: TMEM lane r = row r; warps w and w+4 split the chunk's columns
    const int r = wq * 32 + lane;
    if (wq * 32 < W) {   // warp-uniform
#pragma unroll 1
      for (int j0 = jbeg; j0 < jend; j0 += 4) {
        uint32_t q[kS8][4], s4[kS8][4];
#pragma unroll
        for (int d = 0; d < kS8; ++d) {
          const uint32_t ta = cx.tmem + lane_base + (uint32_t)(d * NC + j0);
          const uint32_t tb = cx.tmem + lane_base + (uint32_t)(d * NC + CW + j0);
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(q[d][0]), "=r"(q[d][1]), "=r"(q[d][2]), "=r"(q[d][3])
                       : "r"(ta));
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(s4[d][0]), "=r"(s4[d][1]), "=r"(s4[d][2]), "=r"(s4[d][3])
                       : "r"(tb));
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (r < W) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = nc * CW + j0 + j;
            if (c < W) recombine(&q[0][j], &s4[0][j], 4, r, c);
          }
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
  }
  __syncthreads();
  if (ok) epi_apply<WP>(C, ep, add, W);
  return ok;
}

// ---------------------------------------------------------------------------
// Second product form (num_wann <= 64): C = A B through
//     [C_r; C_i] = [[A_r, -A_i], [A_i, A_r]] [B_r; B_i]
// i.e. 2W accumulator rows (real parts in rows 0..WP-1, imaginary parts in rows
// WP..2WP-1), N = W columns, K = 2W; operands split into 7 signed 8-bit digits (56 bits;
// exact FP16 values, built two at a time by a packed FP16 subtraction) and the 28 digit
// pairs with t+u <= 6 kept.  Against the first
// form this halves N and TMEM, drops 36 pairs to 28 at the same 56-bit precision, and
// (FP64 matrices in L2 instead of shared memory) lets two CTAs share an SM.  Exactness:
// a diagonal holds at most 7 pairs of products <= 2^14 over K <= 128 terms, < 2^24.
// ---------------------------------------------------------------------------
constexpr int kS2 = 7;

template <int WP, bool SMEM_MATS = false>
struct Exp2Smem {
  static constexpr int CW = WP < 32 ? WP : 32;      // complex inner indices per K chunk
  static constexpr int KC = 2 * CW;                 // real K per chunk
  static constexpr int NCHK = WP / CW;              // K chunks
  static constexpr int ROWS = 2 * WP;               // accumulator rows
  static constexpr int N = WP < 16 ? 16 : WP;       // accumulator columns (MMA N >= 16)
  static constexpr int A_SLICE = ROWS * KC * 2;     // bytes between the overlapped slices
  static constexpr int A_BYTES = (kS2 - 1) * A_SLICE + kTileRows * KC * 2;
  static constexpr int B_BYTES = N * KC * 2;        // per slice
  static constexpr int TMEM_COLS = (kS2 * N <= 128) ? 128 : ((kS2 * N <= 256) ? 256 : 512);
  static constexpr bool STAGED = ROWS <= 64;        // rows in TMEM subpartitions 0-1 only
  static constexpr int STAGE_LD = N + 1;
  static constexpr size_t STAGE_BYTES = STAGED ? (size_t)kS2 * ROWS * STAGE_LD * 4 : 0;
  static constexpr size_t DIGIT_BYTES = (size_t)A_BYTES + (size_t)kS2 * B_BYTES;
  static constexpr size_t REGION = DIGIT_BYTES > STAGE_BYTES ? DIGIT_BYTES : STAGE_BYTES;
  // the six FP64 matrices of the exp chain in shared memory: always for WP <= 16; for
  // WP = 32 on request (one CTA per SM then, shared-memory latency for every operand read)
  static constexpr bool MATS_IN_SMEM = WP <= 16 || SMEM_MATS;
  static constexpr size_t MAT_BYTES = (size_t)WP * WP * 16;
  static constexpr size_t NEED = REGION + (MATS_IN_SMEM ? 6 * MAT_BYTES : 0) + 1024;
  // never more CTAs on an SM than its 512 TMEM columns hold: request enough shared
  // memory that (512 / TMEM_COLS + 1) CTAs cannot fit in the SM's 228 KB
  static constexpr size_t FLOOR = 233472 / (512 / TMEM_COLS + 1) - 1024 + 16;
  static constexpr size_t BYTES = NEED > FLOOR ? NEED : FLOOR;
};

// C = A B, then the Epi.  num_wann <= 32 (staged accumulators): the epilogue applies the
// Epi itself and writes ep.out only (C unused; ep.out may alias B, whose digits are in
// shared memory before the MMAs run, but not A); WP = 64: C as in oz_cmm.
template <int WP, class Add>
__device__ bool oz_cmm2(OzCtx& cx, double2* C, const double2* A, const unsigned* arow, const double2* B,
                        const unsigned* bcol, int W, const Epi& ep, const Add& add) {
  using E = Exp2Smem<WP>;
  constexpr int CW = E::CW, KC = E::KC, N = E::N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  ab_exponents<WP>(cx, A, arow, B, bcol, W);
  __syncthreads();
  bool ok = true;
  for (int kc = 0; kc < E::NCHK && ok; ++kc) {
    // ---- A_emb chunk: complex (r, l) -> rows r (re) and WP + r (im), K l (re) / CW + l (im),
    // and B_emb chunk as B^T (K-major): row = output column c, K l (re) / CW + l (im).  A
    // thread slices one part (re or im) of 8 consecutive l of a row of A and of a column of
    // B (contiguous in memory) -- a whole 16-byte core-matrix row per digit plane -- with
    // both runs' loads issued before either is sliced.  The A part goes to both places it
    // occupies (A_r: (re, K re) and (im, K im); A_i: (im, K re) and, negated, (re, K im));
    // lanes take consecutive rows / columns, so the 16-byte stores do not conflict.
    {
      constexpr int LG = CW / 8, NIA = WP * LG * 2, NIB = N * LG * 2;
      constexpr int NI = NIA > NIB ? NIA : NIB;
      for (int it = tid; it < NI; it += 256) {
        const int r = it % WP, lga = (it / WP) % LG, pa = it / (WP * LG);
        const int c = it % N, lgb = (it / N) % LG, pb = it / (N * LG);
        double va[8], vb[8];
        if (it < NIA) load_run8(va, A + r, (size_t)W, kc * CW + lga * 8, W, r < W, pa);
        if (it < NIB) load_run8(vb, B + (size_t)c * W, (size_t)1, kc * CW + lgb * 8, W, c < W, pb);
        uint32_t w[kS2][4];
        if (it < NIA) {
          slice_run8_h(w, va, cx.rowexp[r]);
          const int kq = lga * 8;
          const uint32_t o1 = pa == 0 ? kmaj_off(r, kq, KC) : kmaj_off(WP + r, kq, KC);
          const uint32_t o2 = pa == 0 ? kmaj_off(WP + r, CW + kq, KC) : kmaj_off(r, CW + kq, KC);
#pragma unroll
          for (int t = 0; t < kS2; ++t) {
            unsigned char* sa = cx.sA + (size_t)t * E::A_SLICE;
            *(uint4*)(sa + o1) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
            *(uint4*)(sa + o2) = pa == 0 ? make_uint4(w[t][0], w[t][1], w[t][2], w[t][3])
                                         : make_uint4(f16x2_neg(w[t][0]), f16x2_neg(w[t][1]),
                                                      f16x2_neg(w[t][2]), f16x2_neg(w[t][3]));
          }
        }
        if (it < NIB) {
          slice_run8_h(w, vb, cx.colexp[c < WP ? c : 0]);
          const uint32_t o = kmaj_off(c, pb * CW + lgb * 8, KC);
#pragma unroll
          for (int t = 0; t < kS2; ++t)
            *(uint4*)(cx.sB + (size_t)t * E::B_BYTES + o) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // descriptors of the slices' K-steps: the base descriptor plus the byte offset / 16 in
      // its address field (shared-memory addresses stay below 2^18, so the field holds it)
      const uint64_t da = smem_desc(smem_u32(cx.sA), 128, (KC / 8) * 128);
      const uint64_t db = smem_desc(smem_u32(cx.sB), 128, (KC / 8) * 128);
      // B's digit planes follow one another as row groups of one K-major operand and
      // diagonal d's accumulator columns follow d - 1's: slice t of A against planes
      // u0 .. u0 + n - 1 of B is one MMA with N = n N, writing diagonals t + u0 .. (N <= 256)
      constexpr int PPM = 256 / N;
#pragma unroll
      for (int t = 0; t < kS2; ++t) {
#pragma unroll
        for (int u0 = 0; u0 + t <= kS2 - 1; u0 += PPM) {
          const int n = (kS2 - t - u0) < PPM ? (kS2 - t - u0) : PPM;
          const uint32_t dtm = cx.tmem + (uint32_t)((t + u0) * N);
          const bool first_pair = (kc == 0) && (t == 0);
#pragma unroll
          for (int ks = 0; ks < KC / 16; ++ks) {
            const uint64_t ad = da + (uint64_t)(((size_t)t * E::A_SLICE + ks * 256) >> 4);
            const uint64_t bd = db + (uint64_t)(((size_t)u0 * E::B_BYTES + ks * 256) >> 4);
            const uint32_t acc = (first_pair && ks == 0) ? 0u : 1u;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                :: "r"(dtm), "l"(ad), "l"(bd), "r"(idesc_f16(n * N)), "r"(acc)
                : "memory");
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                   :: "r"(cx.mbar) : "memory");
    }
    // one thread waits for the commit (the others wait at the CTA barrier, issuing nothing)
    if (tid == 0 && !mbar_wait(cx.mbar, cx.phase)) {
      *cx.bad = 1;
      mbar_drain(cx.mbar, cx.phase);
    }
    cx.phase ^= 1u;
    __syncthreads();
    ok = (*cx.bad == 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (ok) {
    // accumulator row `row` (part = row / WP: 0 real, 1 imaginary; rr = row % WP),
    // column c: sum_d D_d 2^(8(6-d)) 2^(rowexp + colexp - 62)
    auto recombine = [&](const uint32_t* dd, int stride, int row, int c) {
      const int rr = row % WP;
      const double v = recombine7x8(dd, stride, cx.rowexp[rr] + cx.colexp[c] - 62);
      double* dst = (double*)(C + (size_t)c * W + rr);
      dst[row / WP] = v;
    };
    const int wq = warp & 3, half = warp >> 2;
    const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
    constexpr int NH = N / 2;   // columns per warp half
    if (E::STAGED) {
      rec_clear(ep.rec, WP);     // the operands' scales are in cx already
      uint32_t* stage = (uint32_t*)cx.sA;
      if (wq * 32 < E::ROWS) {
#pragma unroll 1
        for (int j0 = half * NH; j0 < (half + 1) * NH; j0 += 4) {
          uint32_t q[kS2][4];
#pragma unroll
          for (int d = 0; d < kS2; ++d)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                         : "=r"(q[d][0]), "=r"(q[d][1]), "=r"(q[d][2]), "=r"(q[d][3])
                         : "r"(cx.tmem + lane_base + (uint32_t)(d * N + j0)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const int row = wq * 32 + lane;
          if (row < E::ROWS) {
#pragma unroll
            for (int d = 0; d < kS2; ++d) {
              uint32_t* rp = stage + ((size_t)d * E::ROWS + row) * E::STAGE_LD + j0;
              rp[0] = q[d][0];
              rp[1] = q[d][1];
              rp[2] = q[d][2];
              rp[3] = q[d][3];
            }
          }
        }
      }
      __syncthreads();
      // both parts of element (rr, c) by one thread
      auto element = [&](int rr, int c) -> double2 {
        const int sc = cx.rowexp[rr] + cx.colexp[c] - 62;
        const double re = recombine7x8(stage + (size_t)rr * E::STAGE_LD + c, E::ROWS * E::STAGE_LD, sc);
        const double im = recombine7x8(stage + (size_t)(WP + rr) * E::STAGE_LD + c, E::ROWS * E::STAGE_LD, sc);
        return make_double2(re, im);
      };
      if (ep.sym == 0) {
#pragma unroll 2
        for (int e = tid; e < W * W; e += blockDim.x) {
          const int rr = e % W, c = e / W;
          double2 v = element(rr, c);
          if (Add::kActive) v = cadd(v, add(e));
          ep.out[e] = v;
          rec_add(ep.rec, rr, c, v);
        }
      } else {
        // the upper triangle rr <= c (linear index e = c (c + 1) / 2 + rr), mirrored
        const int ntri = W * (W + 1) / 2;
        for (int e = tid; e < ntri; e += blockDim.x) {
          int c = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
          while (c * (c + 1) / 2 > e) --c;
          while ((c + 1) * (c + 2) / 2 <= e) ++c;
          const int rr = e - c * (c + 1) / 2;
          double2 v = element(rr, c);
          if (rr == c) {
            v = (ep.sym > 0) ? cmk(v.x, 0.0) : cmk(0.0, v.y);
            ep.out[(size_t)c * W + c] = v;
            rec_add(ep.rec, c, c, v);
          } else {
            ep.out[(size_t)c * W + rr] = v;
            const double2 m = cmk(ep.sym * v.x, -ep.sym * v.y);
            ep.out[(size_t)rr * W + c] = m;
            rec_add(ep.rec, rr, c, v);
            // (a record whose rows and columns share one array already holds the mirror)
            if (ep.rec.row != ep.rec.col) rec_add(ep.rec, c, rr, m);
          }
        }
      }
    } else {
      const int row = wq * 32 + lane;   // all 128 lanes hold rows (ROWS = 128)
      const int rr = row % WP;
#pragma unroll 1
      for (int j0 = half * NH; j0 < (half + 1) * NH; j0 += 4) {
        uint32_t q[kS2][4];
#pragma unroll
        for (int d = 0; d < kS2; ++d)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(q[d][0]), "=r"(q[d][1]), "=r"(q[d][2]), "=r"(q[d][3])
                       : "r"(cx.tmem + lane_base + (uint32_t)(d * N + j0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (rr < W) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j0 + j < W) recombine(&q[0][j], 4, row, j0 + j);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (ok && !E::STAGED) epi_apply<WP>(C, ep, add, W);
  return ok;
}

// product policies of the exp kernel: first form for WP = 128, second for WP <= 64
template <int WP>
struct ProdV1 {
  using E = ExpSmem<WP>;
  static constexpr int TMEM_COLS = E::TMEM_COLS;
  static constexpr bool MATS_IN_SMEM = false;
  static constexpr size_t REGION = E::REGION, BYTES = E::BYTES;
  static constexpr size_t SB_OFFSET = E::A_BYTES;
  template <class Add>
  __device__ static bool mm(OzCtx& cx, double2* C, const double2* A, const unsigned* arow, const double2* B,
                            const unsigned* bcol, int W, const Epi& ep, const Add& add) {
    return oz_cmm<WP>(cx, C, A, arow, B, bcol, W, ep, add);
  }
};

template <int WP, bool SMEM_MATS = false>
struct ProdV2 {
  using E = Exp2Smem<WP, SMEM_MATS>;
  static constexpr int TMEM_COLS = E::TMEM_COLS;
  static constexpr bool MATS_IN_SMEM = E::MATS_IN_SMEM;
  static constexpr size_t REGION = E::REGION, BYTES = E::BYTES;
  static constexpr size_t SB_OFFSET = E::A_BYTES;
  template <class Add>
  __device__ static bool mm(OzCtx& cx, double2* C, const double2* A, const unsigned* arow, const double2* B,
                            const unsigned* bcol, int W, const Epi& ep, const Add& add) {
    return oz_cmm2<WP>(cx, C, A, arow, B, bcol, W, ep, add);
  }
};

template <int WP, bool SMEM_MATS = false>
using ExpProd = typename std::conditional<(WP <= 64), ProdV2<WP, SMEM_MATS>, ProdV1<WP>>::type;

}  // namespace

}  // namespace w90g
