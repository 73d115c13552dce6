// Host orchestration of the GB300 MLWF engine.
//
// Memory: one arena per batch (cudaMalloc, or stream-ordered cudaMallocAsync for the
// serving loop), sub-allocated at 256-byte alignment; every
// per-problem array of the iteration stays resident in HBM for the whole solve.
// Launch: the iteration (7 kernels for small problems, 16 for many k of num_wann > 32 on the
// tensor cores, +2 with the preconditioner; see k_fp64.cu) is captured once into a CUDA graph
// and replayed; the device controller makes replays after convergence no-ops, so the
// host only polls a single "all done" word every few replays.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <sstream>

#include "engine.h"
#include "polar.h"

namespace w90g {

// kernels (k_fp64.cu)
__global__ void k_mdiag(const Problem* probs, WorkMap wm);
__global__ void k_omega_p1(const Problem* probs, WorkMap wm, int slot);
__global__ void k_omega_p2(const Problem* probs, WorkMap wm, int slot);
__global__ void k_grad(const Problem* probs, WorkMap wm);
__global__ void k_grad_search(const Problem* probs, WorkMap wm);
__global__ void k_ctrl_search(const Problem* probs);
__global__ void k_exp_u(const Problem* probs, WorkMap wm, int which);
__global__ void k_m_update(const Problem* probs, WorkMap wm, int mode, int which);
__global__ void k_log_init(const Problem* probs);
__global__ void k_lowdin(const Problem* probs, WorkMap wm, int* status);
__global__ void k_unitarity(const Problem* probs, WorkMap wm, double* out);
__global__ void k_all_done(const Problem* probs, int nprob, int* out);
__global__ void k_fp64_peak(double* out, int iters, double seed);
__global__ void k_u_identity(const Problem* probs, WorkMap wm);
__global__ void k_precond(const Problem* probs, int dir);
__global__ void k_phases(const Problem* probs, int mode);
// kernels (k_sitesym.cu)
__global__ void k_sym_grad(const Problem* probs, WorkMap wm);
__global__ void k_sym_dir(const Problem* probs, WorkMap wm);
__global__ void k_sym_u(const Problem* probs, WorkMap wm);
cudaError_t oz_ufinal_launch(int wp, const Problem* probs, WorkMap wm, int grid, cudaStream_t s);
cudaError_t oz3_launch(int wp, const Problem* probs, WorkMap wm, int which, int ngroups, int tmax, int slabs,
                       cudaStream_t s);
cudaError_t oz3_preslice_launch(int wp, const Problem* probs, WorkMap wm, int ngroups, int tmax, cudaStream_t s);
cudaError_t oz3_set_attributes(int wp);
void oz3_bytes(int W, int K, int B, size_t out[4]);
int oz3_tiles(int W, int B);
cudaError_t oz2_launch(int wp, int step, const Problem* probs, WorkMap wm, int which, int ngroups,
                       cudaStream_t s);
cudaError_t oz2_set_attributes(int wp);
cudaError_t oz2_preslice_launch(int wp, const Problem* probs, WorkMap wm, int grid, cudaStream_t s);
void oz2_ub2_bytes(int wp, int K, size_t* data, size_t* exps);
cudaError_t oz_launch(int wp, int step, const Problem* probs, WorkMap wm, int which, int grid,
                      cudaStream_t s);
cudaError_t oz_set_attributes(int wp);
void oz_preslice_bytes(int wp, int K, int B, size_t* data, size_t* exps);
cudaError_t oz_preslice_launch(int wp, const Problem* probs, WorkMap wm, int grid, cudaStream_t s);
cudaError_t oz_exp_launch(int wp, int smem_mats, const Problem* probs, WorkMap wm, int which, int grid,
                          cudaStream_t s);
cudaError_t oz_exp_set_attributes(int wp, int smem_mats);

const char* kProfNames[kPNum] = {"k_grad", "k_ctrl_search", "k_exp_u", "k_m_update",
                                 "k_omega", "k_ctrl_step", "k_ctrl_end", "init", "k_precond"};

namespace {
constexpr size_t kAlign = 256;
size_t align_up(size_t x) { return (x + kAlign - 1) & ~(kAlign - 1); }
constexpr int kTileW = 32;
constexpr int kPolarMinW = 9;   // projection on the tensor cores from this width on (see project)

#define W90G_CHECK(call)                                                          \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess) {                                                      \
      err = std::string(#call) + ": " + cudaGetErrorString(e_);                   \
      return (e_ == cudaErrorMemoryAllocation) ? 2 : 1;                           \
    }                                                                             \
  } while (0)
}  // namespace

Engine::Engine() {}

Engine::~Engine() { release(); }

void Engine::release() {
  if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
  graph_exec_ = nullptr;
  if (arena_) {
    if (async_alloc_) cudaFreeAsync(arena_, stream());
    else cudaFree(arena_);
  }
  arena_ = nullptr;
  arena_bytes_ = 0;
  if (own_stream_) cudaStreamDestroy(own_stream_);
  own_stream_ = nullptr;
}

namespace {

// every k' has exactly B predecessors (k,b) (true on Monkhorst-Pack meshes)
bool regular_neighbours(const ProblemSpec& s) {
  std::vector<int> cnt(s.K, 0);
  for (int v : s.nnlist) cnt[v]++;
  for (int c : cnt)
    if (c != s.B) return false;
  return true;
}

// tensor-core M update: every problem asks for it, W <= 128, and has regular neighbour lists; returns
// the padded width or 0
int choose_tensor_wp(const std::vector<ProblemSpec>& specs, const std::vector<char>& regular) {
  bool ok = !specs.empty();
  int wmax = 0;
  for (size_t p = 0; p < specs.size(); ++p) {
    ok = ok && specs[p].tensor && specs[p].W <= 128 && regular[p];
    wmax = std::max(wmax, specs[p].W);
  }
  if (!ok) return 0;
  return wmax <= 8 ? 8 : (wmax <= 16 ? 16 : (wmax <= 32 ? 32 : (wmax <= 64 ? 64 : 128)));
}

// [k'][i] = k B + b with nnlist(k,b) = k', in the order of k B + b
std::vector<int> inverse_neighbours(const ProblemSpec& s) {
  std::vector<int> inv((size_t)s.K * s.B), fill(s.K, 0);
  for (int kb = 0; kb < s.K * s.B; ++kb) {
    const int k2 = s.nnlist[kb];
    inv[(size_t)k2 * s.B + fill[k2]++] = kb;
  }
  return inv;
}

}  // namespace

int Engine::setup(const std::vector<ProblemSpec>& specs, std::string& err) {
  for (const auto& s : specs) {
    if (s.W < 1 || s.W > 256) {
      err = "num_wann outside the engine range 1..256";
      return 5;
    }
    if (s.B < 1 || s.B > 12 || s.K < 1) {
      err = "invalid k-mesh (num_kpts / nntot)";
      return 5;
    }
    if (s.ctl.conv_window > kMaxConvWindow) {
      err = "conv_window larger than the engine maximum (64)";
      return 5;
    }
    if (s.guiding && (s.nnh < 3 || s.rguide0.size() != (size_t)3 * s.W || s.bka.size() != (size_t)3 * s.nnh ||
                      s.neigh.size() != (size_t)s.K * s.nnh)) {
      err = "guiding_centres: centres or b-direction tables missing";
      return 5;
    }
    if (s.slwf_num < 0 || s.slwf_num >= s.W ||
        (s.slwf_num > 0 && !s.slwf_c.empty() && s.slwf_c.size() != (size_t)3 * s.W)) {
      err = "slwf: slwf_num outside 1..num_wann-1 or constrained centres not num_wann x 3";
      return 5;
    }
    if (s.sym_nir > 0) {
      const size_t nir = s.sym_nir, WW2 = (size_t)2 * s.W * s.W;
      if (s.sym_ik.size() != nir || s.sym_moff.size() != nir + 1 || s.sym_goff.size() != nir + 1 ||
          s.sym_mem.size() != (size_t)2 * s.sym_moff[nir] || s.sym_grp.size() != (size_t)2 * s.sym_goff[nir] ||
          s.sym_d.empty() || s.sym_d.size() % WW2 != 0 || s.sym_db.size() != s.sym_d.size()) {
        err = "site symmetry: tables missing or inconsistent";
        return 5;
      }
    }
    if (s.precond && (s.nrpts < 1 || s.pc_kr.size() != (size_t)2 * s.K * s.nrpts ||
                      s.pc_r2.size() != (size_t)s.nrpts || s.pc_ndeg.size() != (size_t)s.nrpts)) {
      err = "precond: Wigner-Seitz tables missing or inconsistent";
      return 5;
    }
  }
  // layout key: reuse the arena when the problem shapes are unchanged, and with them all that alloc()
  // derives from the neighbour lists (choose_tensor_wp) and the options (which kernels run)
  // (neighbour lists equal to those on the device are neither examined nor uploaded again)
  std::vector<char> same(specs.size()), regular(specs.size());
  for (size_t p = 0; p < specs.size(); ++p) {
    same[p] = arena_ && p < specs_.size() && p < regular_.size() && specs[p].K == specs_[p].K &&
              specs[p].B == specs_[p].B && specs[p].nnlist == specs_[p].nnlist;
    regular[p] = same[p] ? regular_[p] : regular_neighbours(specs[p]);
  }
  regular_ = regular;
  std::ostringstream key;
  key << choose_tensor_wp(specs, regular_) << ';';
  for (const auto& s : specs)
    key << s.W << ',' << s.K << ',' << s.B << ',' << s.ctl.num_iter << ',' << s.tensor << ',' << s.tensor_exp << ','
        << s.mupdate_pipe << ',' << s.exp_smem << ',' << s.precond << ',' << s.nrpts << ',' << s.guiding << ',' << s.nnh << ',' << (s.slwf_num > 0) << ',' << s.sym_nir << ','
        << s.sym_mem.size() << ',' << s.sym_grp.size() << ',' << s.sym_d.size() << ',' << s.lean << ';';
  specs_ = specs;
  if (arena_ && key.str() == layout_key_) {
    // refresh the read-only tables (they may differ at equal shapes); the key again when that is done
    layout_key_.clear();
    for (size_t p = 0; p < specs_.size(); ++p) {
      const auto& s = specs_[p];
      Problem& P = hprobs_[p];
      if (!same[p]) {
        W90G_CHECK(cudaMemcpyAsync((void*)P.nnlist, s.nnlist.data(), s.nnlist.size() * sizeof(int), cudaMemcpyHostToDevice, stream()));
        if (P.inv_nnlist) {
          const std::vector<int> inv = inverse_neighbours(s);
          W90G_CHECK(cudaMemcpyAsync((void*)P.inv_nnlist, inv.data(), inv.size() * sizeof(int), cudaMemcpyHostToDevice, stream()));
        }
      }
      P.no_guide_iter = s.no_guide_iter;
      P.guide_cycles = s.guide_cycles;
      W90G_CHECK(cudaMemcpyAsync((void*)P.bk, s.bk.data(), s.bk.size() * sizeof(double), cudaMemcpyHostToDevice, stream()));
      W90G_CHECK(cudaMemcpyAsync((void*)P.wb, s.wb.data(), s.wb.size() * sizeof(double), cudaMemcpyHostToDevice, stream()));
      if (s.guiding) {
        W90G_CHECK(cudaMemcpyAsync((void*)P.bka, s.bka.data(), s.bka.size() * 8, cudaMemcpyHostToDevice, stream()));
        W90G_CHECK(cudaMemcpyAsync((void*)P.neigh, s.neigh.data(), s.neigh.size() * 4, cudaMemcpyHostToDevice, stream()));
      }
      if (s.precond) {
        W90G_CHECK(cudaMemcpyAsync((void*)P.pc_kr, s.pc_kr.data(), s.pc_kr.size() * 8, cudaMemcpyHostToDevice, stream()));
        W90G_CHECK(cudaMemcpyAsync((void*)P.pc_r2, s.pc_r2.data(), s.pc_r2.size() * 8, cudaMemcpyHostToDevice, stream()));
        W90G_CHECK(cudaMemcpyAsync((void*)P.pc_ndeg, s.pc_ndeg.data(), s.pc_ndeg.size() * 8, cudaMemcpyHostToDevice, stream()));
      }
      P.ctl = s.ctl;
      P.wbtot = s.wbtot;
      if (int rc = set_slwf(p, err)) return rc;
      if (int rc = set_sym(p, err)) return rc;
    }
    W90G_CHECK(cudaMemcpyAsync(dprobs_, hprobs_.data(), hprobs_.size() * sizeof(Problem), cudaMemcpyHostToDevice, stream()));
    layout_key_ = key.str();
    return 0;
  }
  release();
  layout_key_.clear();
  if (int rc = alloc(err)) return rc;
  layout_key_ = key.str();
  return 0;
}

namespace {

// chunks of the spread passes: 64 blocks (k,b) each, and from 512 blocks on down to 16 while that
// gives every SM one (64 alone left 100 of the SMs idle on 3072 blocks of num_wann 128)
int omega_chunks(const ProblemSpec& s) {
  const int KB = s.K * s.B;
  const int n = (KB + 63) / 64;
  return KB < 512 ? n : std::max(n, std::min((KB + 15) / 16, 152));
}

// partial off-diagonal sums per (k,b) that the tensor M update's epilogue writes: one per column
// group, and for num_wann > 32 per 32-row piece of the block (k_mupdate3.cu)
int odn_of(int W) { return W <= 32 ? 4 : 4 * (W / 32 + 2); }

// An array that may lie inside another one that is dead while it is used: host 1 is M0 (tensor path;
// read once, to slice it, before any of these is written), host 2 is dU (dead between the exp and the
// next one; on the FP64 path the M update reads it, so only the spread's arrays may lie there).
struct Part {
  size_t n = 0, at = 0;
  int host = 0;
  size_t own() const { return host ? 0 : n; }
};

struct Sizes {
  size_t M, U, KWW, tbuf, diag, offd, gpart, cen, log, logc, nn, bk, wb, st, m0, u0, inv, fr;
  size_t m0s, m0e, zexp;
  Part work, ub2, ub2e, einfo, odp, zs, zse, op1, op2;
  int slabs;
  size_t pkr, pr2, pgr, pgp, ppart;
  size_t gbka, gneigh, grg, gsheet, gcsheet;
  size_t slwf;
  size_t symi, symd, symw;
  size_t total() const {
    return 2 * M + 2 * U + 3 * KWW + work.own() + tbuf + 2 * diag + offd + gpart + cen + log + logc + nn + bk + wb + st +
           op1.own() + op2.own() + m0 + u0 + inv + fr + m0s + m0e + zexp + ub2.own() + ub2e.own() + einfo.own() +
           odp.own() + zs.own() + zse.own() + pkr + 2 * pr2 + pgr + pgp + ppart + gbka + gneigh + grg + gsheet + gcsheet + slwf + symi + 2 * symd + symw;
  }
};

// per-problem device arrays (bytes, 256-aligned) for tensor width wp (0: FP64 path)
Sizes problem_sizes(const ProblemSpec& s, int wp, int* pc_tiles) {
  const size_t W = s.W, K = s.K, B = s.B;
  const size_t WW = W * W;
  const size_t nt = (s.W + kTileW - 1) / kTileW;
  Sizes z;
  z.M = align_up(K * B * WW * 16);
  z.U = align_up(K * WW * 16);
  z.KWW = align_up(K * WW * 16);
  // exp workspace: FP64 kernels for W > 32; the tensor exp keeps X and its powers here
  z.work.n = (s.W > 32 || wp) ? align_up(K * 6 * WW * 16) : 0;
  z.einfo.n = wp ? align_up(K * 8) : 0;
  z.tbuf = (s.W > 32 || wp) ? align_up(K * B * WW * 16) : 0;
  z.m0 = wp ? align_up(K * B * WW * 16) : 0;
  z.u0 = wp ? align_up(K * WW * 16) : 0;
  z.inv = wp ? align_up(K * B * 4) : 0;
  z.odp.n = wp ? align_up(K * B * odn_of(s.W) * 8) : 0;
  z.fr = wp ? align_up(K * B * 8) : 0;
  z.m0s = z.m0e = 0;
  z.slabs = 1;
  z.zexp = (wp && wp <= 32) ? align_up(K * B * W * 4) : 0;
  if (wp && wp <= 32) {
    size_t d = 0, e = 0;
    oz2_ub2_bytes(wp, (int)K, &d, &e);
    z.ub2.n = align_up(d);
    z.ub2e.n = align_up(e);
  }
  if (wp > 32) {
    size_t b[4];
    oz3_bytes((int)W, (int)K, (int)B, b);
    z.m0s = align_up(b[0]);
    z.m0e = z.zse.n = align_up(b[1]);
    z.ub2.n = align_up(b[2]);
    z.ub2e.n = align_up(b[3]);
    // the digit image of Z (28 B an element against M0's 16): all groups' at once, or in as many slabs
    // as it takes to fit into M0 with U's image
    auto image = [&](int slabs) { return align_up(b[0] / K * ((K + slabs - 1) / slabs)); };
    if (s.lean)
      while (z.slabs < (int)K && image(z.slabs) + z.ub2.n > z.m0) ++z.slabs;
    z.zs.n = image(z.slabs);
    z.m0 = std::max(z.m0, z.zs.n);
  } else if (wp) {
    size_t d = 0, e = 0;
    oz_preslice_bytes(wp, (int)K, (int)B, &d, &e);
    z.m0s = align_up(d);
    z.m0e = align_up(e);
  }
  z.diag = align_up(K * B * W * 8);
  z.offd = align_up(K * B * 8);
  z.gpart = align_up(K * nt * nt * 2 * 8);
  z.cen = align_up(3 * 4 * W * 8);
  z.log = align_up((size_t)(s.ctl.num_iter + 1) * kLogStride * 8);
  z.logc = align_up((size_t)(s.ctl.num_iter + 1) * 4 * W * 8);
  z.nn = align_up(K * B * 4);
  z.bk = align_up(K * B * 3 * 8);
  z.wb = align_up(B * 8);
  z.st = align_up(sizeof(CtrlState));
  const size_t nch = omega_chunks(s);
  z.op1.n = align_up(nch * (4 * W + 2) * 8);
  z.op2.n = align_up(nch * 8);
  size_t used[3] = {0, 0, 0};
  auto inside = [&](Part& q, int host) {
    const size_t room = host == 1 ? z.m0 : z.KWW;
    if (q.n == 0 || q.host || used[host] + q.n > room) return;
    q.host = host;
    q.at = used[host];
    used[host] += q.n;
  };
  inside(z.op1, 2);
  inside(z.op2, 2);
  if (wp) {
    inside(z.zs, 1);
    if (wp > 32) inside(z.ub2, 1);
    else inside(z.work, 1);
    inside(z.odp, 2);
    inside(z.einfo, 1);
    for (Part* q : {&z.odp, &z.zse, &z.op1, &z.op2}) inside(*q, 1);
    if (wp > 32) inside(z.ub2e, 2);
    inside(z.zse, 2);
  }
  z.pkr = z.pr2 = z.pgr = z.pgp = z.ppart = 0;
  if (s.precond) {
    const size_t NR = s.nrpts;
    const size_t te = (WW + 63) / 64;
    z.pkr = align_up(K * NR * 16);
    z.pr2 = align_up(NR * 8);
    z.pgr = align_up(NR * WW * 16);
    z.pgp = align_up(K * WW * 16);
    z.ppart = align_up(te * ((K + 15) / 16) * 8);
    if (pc_tiles) *pc_tiles = std::max(*pc_tiles, (int)(te * ((std::max(K, NR) + 15) / 16)));
  }
  z.slwf = s.slwf_num > 0 ? align_up(3 * W * 8) : 0;
  z.symi = z.symd = z.symw = 0;
  if (s.sym_nir > 0) {
    const size_t nint = s.sym_ik.size() + s.sym_moff.size() + s.sym_mem.size() + s.sym_goff.size() +
                        s.sym_grp.size() + (size_t)s.sym_nir;
    z.symi = align_up(nint * 4);
    z.symd = align_up(s.sym_d.size() * 8);
    z.symw = align_up((size_t)s.sym_nir * kSymWork * WW * 16);
  }
  z.gbka = z.gneigh = z.grg = z.gsheet = z.gcsheet = 0;
  if (s.guiding) {
    z.gbka = align_up((size_t)s.nnh * 3 * 8);
    z.gneigh = align_up(K * s.nnh * 4);
    z.grg = align_up(3 * W * 8);
    z.gsheet = align_up(K * B * W * 8);
    z.gcsheet = align_up(K * B * W * 16);
  }
  return z;
}

size_t header_bytes(int np, int n_k) {
  return align_up(np * sizeof(Problem)) + 5 * align_up((np + 1) * sizeof(int)) + align_up(n_k * sizeof(int)) +
         align_up(n_k * sizeof(double)) + align_up(sizeof(int));
}

}  // namespace

size_t Engine::estimate_bytes(const std::vector<ProblemSpec>& specs) {
  std::vector<char> regular;
  for (const auto& s : specs) regular.push_back(regular_neighbours(s));
  const int wp = choose_tensor_wp(specs, regular);
  size_t total = 0;
  int nk = 0;
  for (const auto& s : specs) {
    total += problem_sizes(s, wp, nullptr).total();
    nk += s.K;
  }
  return total + header_bytes((int)specs.size(), nk);
}

int Engine::alloc(std::string& err) {
  const int np = (int)specs_.size();
  tensor_wp_ = choose_tensor_wp(specs_, regular_);
  if (!own_stream_) W90G_CHECK(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking));
  std::vector<Sizes> sz(np);
  size_t total = 0;
  n_k_ = n_kb_ = n_grad_ = 0;
  pc_tiles_ = 0;
  guide_w_ = 0;
  maxW_small_ = 0;
  max_iter_ = 0;
  std::vector<int> offs_k(np + 1, 0), offs_kb(np + 1, 0), offs_grad(np + 1, 0), offs_chunk(np + 1, 0),
      offs_ir(np + 1, 0);
  for (int p = 0; p < np; ++p) {
    const auto& s = specs_[p];
    const int nt = (s.W + kTileW - 1) / kTileW;
    sz[p] = problem_sizes(s, tensor_wp_, &pc_tiles_);
    if (s.guiding) guide_w_ = std::max(guide_w_, s.W);
    total += sz[p].total();
    offs_k[p + 1] = offs_k[p] + s.K;
    offs_kb[p + 1] = offs_kb[p] + s.K * s.B;
    offs_grad[p + 1] = offs_grad[p] + s.K * nt * nt;
    offs_chunk[p + 1] = offs_chunk[p] + omega_chunks(s);
    offs_ir[p + 1] = offs_ir[p] + s.sym_nir;
    if (s.W <= 32) maxW_small_ = std::max(maxW_small_, s.W);
    max_iter_ = std::max(max_iter_, s.ctl.num_iter);
  }
  n_k_ = offs_k[np];
  n_kb_ = offs_kb[np];
  n_grad_ = offs_grad[np];
  n_chunk_ = offs_chunk[np];
  omega_two_ = false;
  for (const auto& s : specs_) omega_two_ = omega_two_ || s.K * s.B * s.W > kOmegaOneCta;
  n_ir_ = offs_ir[np];
  total += header_bytes(np, n_k_);
  // (no room: the M update's wide form again with its image of Z in slabs)
  auto grab = [&] { return async_alloc_ ? cudaMallocAsync(&arena_, total, stream()) : cudaMalloc(&arena_, total); };
  cudaError_t ea = grab();
  if (ea == cudaErrorMemoryAllocation && tensor_wp_ > 32) {
    cudaGetLastError();
    arena_ = nullptr;
    total = header_bytes(np, n_k_);
    for (int p = 0; p < np; ++p) {
      specs_[p].lean = 1;
      sz[p] = problem_sizes(specs_[p], tensor_wp_, nullptr);
      total += sz[p].total();
    }
    ea = grab();
  }
  W90G_CHECK(ea);
  slabs_ = 1;
  arena_bytes_ = total;
  char* cur = (char*)arena_;
  auto take = [&](size_t n) {
    char* r = cur;
    cur += n;
    return (void*)r;
  };
  dprobs_ = (Problem*)take(align_up(np * sizeof(Problem)));
  d_offs_k_ = (int*)take(align_up((np + 1) * sizeof(int)));
  d_offs_kb_ = (int*)take(align_up((np + 1) * sizeof(int)));
  d_offs_grad_ = (int*)take(align_up((np + 1) * sizeof(int)));
  d_offs_chunk_ = (int*)take(align_up((np + 1) * sizeof(int)));
  d_offs_ir_ = (int*)take(align_up((np + 1) * sizeof(int)));
  d_status_ = (int*)take(align_up(n_k_ * sizeof(int)));
  d_unit_ = (double*)take(align_up(n_k_ * sizeof(double)));
  int* d_alldone = (int*)take(align_up(sizeof(int)));
  (void)d_alldone;
  hprobs_.assign(np, Problem{});
  results_.assign(np, ProblemResult{});
  for (int p = 0; p < np; ++p) {
    const auto& s = specs_[p];
    const Sizes& z = sz[p];
    Problem& P = hprobs_[p];
    P.W = s.W;
    P.K = s.K;
    P.B = s.B;
    P.wbtot = s.wbtot;
    P.M[0] = (double2*)take(z.M);
    P.M[1] = (double2*)take(z.M);
    P.U[0] = (double2*)take(z.U);
    P.U[1] = (double2*)take(z.U);
    P.G = (double2*)take(z.KWW);
    P.D = (double2*)take(z.KWW);
    P.dU = (double2*)take(z.KWW);
    P.M0 = z.m0 ? (double2*)take(z.m0) : nullptr;
    auto part = [&](const Part& q) -> void* {
      if (q.n == 0) return nullptr;
      return q.host == 0 ? (void*)take(q.n) : (char*)(q.host == 1 ? P.M0 : P.dU) + q.at;
    };
    P.work = (double2*)part(z.work);
    P.expinfo = (float*)part(z.einfo);
    P.tbuf = z.tbuf ? (double2*)take(z.tbuf) : nullptr;
    P.diag_ln = (double*)take(z.diag);
    P.diag_abs2 = (double*)take(z.diag);
    P.offd = (double*)take(z.offd);
    P.gpart = (double*)take(z.gpart);
    P.centres = (double*)take(z.cen);
    P.log = (double*)take(z.log);
    P.log_centres = (double*)take(z.logc);
    int* nn = (int*)take(z.nn);
    double* bk = (double*)take(z.bk);
    double* wb = (double*)take(z.wb);
    P.st = (CtrlState*)take(z.st);
    P.U0 = z.u0 ? (double2*)take(z.u0) : nullptr;
    int* inv = z.inv ? (int*)take(z.inv) : nullptr;
    P.inv_nnlist = inv;
    P.tensor = tensor_wp_ ? 1 : 0;
    P.frob0 = z.fr ? (double*)take(z.fr) : nullptr;
    P.odpart = (double*)part(z.odp);
    P.odn = odn_of(s.W);
    P.m0s = z.m0s ? (unsigned char*)take(z.m0s) : nullptr;
    P.m0s_exp = z.m0e ? (int*)take(z.m0e) : nullptr;
    P.zs = (unsigned char*)part(z.zs);
    P.zs_exp = (int*)part(z.zse);
    P.zs_slabs = z.slabs;
    slabs_ = std::max(slabs_, z.slabs);
    P.zexp = z.zexp ? (int*)take(z.zexp) : nullptr;
    P.ub2 = (unsigned char*)part(z.ub2);
    P.ub2_exp = (int*)part(z.ub2e);
    if (inv) {
      const std::vector<int> h_inv = inverse_neighbours(s);
      W90G_CHECK(cudaMemcpyAsync(inv, h_inv.data(), h_inv.size() * sizeof(int), cudaMemcpyHostToDevice, stream()));
    }
    P.opart1 = (double*)part(z.op1);
    P.opart2 = (double*)part(z.op2);
    P.nchunk = omega_chunks(s);
    P.ctl = s.ctl;
    W90G_CHECK(cudaMemcpyAsync(nn, s.nnlist.data(), s.nnlist.size() * sizeof(int), cudaMemcpyHostToDevice, stream()));
    W90G_CHECK(cudaMemcpyAsync(bk, s.bk.data(), s.bk.size() * sizeof(double), cudaMemcpyHostToDevice, stream()));
    W90G_CHECK(cudaMemcpyAsync(wb, s.wb.data(), s.wb.size() * sizeof(double), cudaMemcpyHostToDevice, stream()));
    P.nnlist = nn;
    P.bk = bk;
    P.wb = wb;
    P.guiding = s.guiding;
    P.nnh = s.nnh;
    P.no_guide_iter = s.no_guide_iter;
    P.guide_cycles = s.guide_cycles;
    if (s.guiding) {
      double* bka = (double*)take(z.gbka);
      int* neigh = (int*)take(z.gneigh);
      W90G_CHECK(cudaMemcpyAsync(bka, s.bka.data(), s.bka.size() * 8, cudaMemcpyHostToDevice, stream()));
      W90G_CHECK(cudaMemcpyAsync(neigh, s.neigh.data(), s.neigh.size() * 4, cudaMemcpyHostToDevice, stream()));
      P.bka = bka;
      P.neigh = neigh;
      P.rguide = (double*)take(z.grg);
      P.sheet = (double*)take(z.gsheet);
      P.csheet = (double2*)take(z.gcsheet);
    }
    P.slwf_c = z.slwf ? (const double*)take(z.slwf) : nullptr;
    if (int rc = set_slwf(p, err)) return rc;
    if (z.symi) {
      P.sym_ik = (const int*)take(z.symi);
      P.sym_d = (const double2*)take(z.symd);
      P.sym_db = (const double2*)take(z.symd);
      P.sym_work = (double2*)take(z.symw);
    }
    if (int rc = set_sym(p, err)) return rc;
    P.precond = s.precond;
    P.nrpts = s.precond ? s.nrpts : 0;
    if (s.precond) {
      double* kr = (double*)take(z.pkr);
      double* r2 = (double*)take(z.pr2);
      double* nd = (double*)take(z.pr2);
      W90G_CHECK(cudaMemcpyAsync(kr, s.pc_kr.data(), s.pc_kr.size() * 8, cudaMemcpyHostToDevice, stream()));
      W90G_CHECK(cudaMemcpyAsync(r2, s.pc_r2.data(), s.pc_r2.size() * 8, cudaMemcpyHostToDevice, stream()));
      W90G_CHECK(cudaMemcpyAsync(nd, s.pc_ndeg.data(), s.pc_ndeg.size() * 8, cudaMemcpyHostToDevice, stream()));
      P.pc_kr = (const double2*)kr;
      P.pc_r2 = r2;
      P.pc_ndeg = nd;
      P.pc_gr = (double2*)take(z.pgr);
      P.pc_gp = (double2*)take(z.pgp);
      P.pc_part = (double*)take(z.ppart);
    }
  }
  W90G_CHECK(cudaMemcpyAsync(dprobs_, hprobs_.data(), np * sizeof(Problem), cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync(d_offs_k_, offs_k.data(), (np + 1) * sizeof(int), cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync(d_offs_kb_, offs_kb.data(), (np + 1) * sizeof(int), cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync(d_offs_grad_, offs_grad.data(), (np + 1) * sizeof(int), cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync(d_offs_chunk_, offs_chunk.data(), (np + 1) * sizeof(int), cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync(d_offs_ir_, offs_ir.data(), (np + 1) * sizeof(int), cudaMemcpyHostToDevice, stream()));
  // dynamic shared memory limits of the shared-memory kernels: a function attribute is
  // process wide, so every engine sets the same value, the maximum for W <= 32 (engines
  // of different widths may run concurrently in the batched form)
  constexpr int wmax = 32;
  W90G_CHECK(cudaFuncSetAttribute(k_exp_u, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * wmax * wmax * 16));
  W90G_CHECK(cudaFuncSetAttribute(k_m_update, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * wmax * wmax * 16));
  W90G_CHECK(cudaFuncSetAttribute(k_lowdin, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * wmax * wmax * 16));
  tensor_exp_ = tensor_wp_ != 0;
  for (const auto& s : specs_) tensor_exp_ = tensor_exp_ && s.tensor_exp;
  pipe_ = tensor_wp_ != 0 && tensor_wp_ <= 32;
  for (const auto& s : specs_) pipe_ = pipe_ && s.mupdate_pipe;
  tiles3_ = 0;
  if (tensor_wp_ > 32)
    for (const auto& s : specs_) tiles3_ = std::max(tiles3_, oz3_tiles(s.W, s.B));
  if (tensor_wp_)
    W90G_CHECK(tiles3_ ? oz3_set_attributes(tensor_wp_)
                       : (pipe_ ? oz2_set_attributes(tensor_wp_) : oz_set_attributes(tensor_wp_)));
  exp_smem_ = tensor_exp_ && tensor_wp_ == 32;
  for (const auto& s : specs_) exp_smem_ = exp_smem_ && s.exp_smem;
  if (tensor_exp_) W90G_CHECK(oz_exp_set_attributes(tensor_wp_, exp_smem_ ? 1 : 0));
  return 0;
}

// selective-localisation fields of problem p from its spec (the centre array is part of
// the layout when slwf_num > 0; zero when unconstrained)
int Engine::set_slwf(int p, std::string& err) {
  const auto& s = specs_[p];
  Problem& P = hprobs_[p];
  P.slwf_num = s.slwf_num;
  P.slwf_lambda = 0.0;
  P.slwf_nu0 = 0.0;
  if (s.slwf_num <= 0) return 0;
  std::vector<double> c((size_t)3 * s.W, 0.0);
  if (!s.slwf_c.empty()) {
    // lambda_loc = lambda only with constrained centres (src/wannierise.F90:445-450)
    c = s.slwf_c;
    P.slwf_lambda = s.slwf_lambda;
    double c2 = 0.0;
    for (int n = 0; n < s.slwf_num; ++n)
      for (int i = 0; i < 3; ++i) c2 += c[(size_t)i * s.W + n] * c[(size_t)i * s.W + n];
    P.slwf_nu0 = s.slwf_lambda * c2;
  }
  slwf_host_.resize(hprobs_.size());
  slwf_host_[p] = c;   // the copy below reads it asynchronously
  W90G_CHECK(cudaMemcpyAsync((void*)P.slwf_c, slwf_host_[p].data(), c.size() * 8, cudaMemcpyHostToDevice, stream()));
  return 0;
}

// symmetry tables of problem p into its arena block: one int block (sym_ik, sym_moff,
// sym_mem, sym_goff, sym_grp, sym_status) and the slot matrices
int Engine::set_sym(int p, std::string& err) {
  const auto& s = specs_[p];
  Problem& P = hprobs_[p];
  P.sym_nir = s.sym_nir;
  P.sym_eps = s.sym_eps;
  if (s.sym_nir <= 0) return 0;
  std::vector<int> ints;
  ints.insert(ints.end(), s.sym_ik.begin(), s.sym_ik.end());
  ints.insert(ints.end(), s.sym_moff.begin(), s.sym_moff.end());
  ints.insert(ints.end(), s.sym_mem.begin(), s.sym_mem.end());
  ints.insert(ints.end(), s.sym_goff.begin(), s.sym_goff.end());
  ints.insert(ints.end(), s.sym_grp.begin(), s.sym_grp.end());
  ints.insert(ints.end(), (size_t)s.sym_nir, 0);
  int* base = const_cast<int*>(P.sym_ik);
  size_t o = 0;
  P.sym_moff = base + (o += s.sym_ik.size());
  P.sym_mem = base + (o += s.sym_moff.size());
  P.sym_goff = base + (o += s.sym_mem.size());
  P.sym_grp = base + (o += s.sym_goff.size());
  P.sym_status = base + (o += s.sym_grp.size());
  sym_host_.resize(hprobs_.size());
  sym_host_[p] = std::move(ints);
  W90G_CHECK(cudaMemcpyAsync(base, sym_host_[p].data(), sym_host_[p].size() * 4, cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync((void*)P.sym_d, s.sym_d.data(), s.sym_d.size() * 8, cudaMemcpyHostToDevice, stream()));
  W90G_CHECK(cudaMemcpyAsync((void*)P.sym_db, s.sym_db.data(), s.sym_db.size() * 8, cudaMemcpyHostToDevice, stream()));
  return 0;
}

int Engine::load(int p, const void* M, const void* U, cudaMemcpyKind kind, std::string& err, int ldm) {
  const auto& s = specs_[p];
  const size_t WW = (size_t)s.W * s.W;
  cudaStream_t st = stream();
  if (M && ldm > s.W) W90G_CHECK(copy_wblocks(hprobs_[p].M[0], s.W, M, ldm, s.W, s.K * s.B, kind, st));
  else if (M) W90G_CHECK(cudaMemcpyAsync(hprobs_[p].M[0], M, (size_t)s.K * s.B * WW * 16, kind, st));
  if (U) W90G_CHECK(cudaMemcpyAsync(hprobs_[p].U[0], U, (size_t)s.K * WW * 16, kind, st));
  return 0;
}

int Engine::store(int p, void* M, void* U, cudaMemcpyKind kind, std::string& err, int ldm) {
  const auto& s = specs_[p];
  const size_t WW = (size_t)s.W * s.W;
  cudaStream_t st = stream();
  CtrlState hs;
  W90G_CHECK(cudaMemcpyAsync(&hs, hprobs_[p].st, sizeof(CtrlState), cudaMemcpyDeviceToHost, st));
  W90G_CHECK(cudaStreamSynchronize(st));
  const int cur = hs.cur;
  if (M && ldm > s.W) W90G_CHECK(copy_wblocks(M, ldm, hprobs_[p].M[cur], s.W, s.W, s.K * s.B, kind, st));
  else if (M) W90G_CHECK(cudaMemcpyAsync(M, hprobs_[p].M[cur], (size_t)s.K * s.B * WW * 16, kind, st));
  if (U) W90G_CHECK(cudaMemcpyAsync(U, hprobs_[p].U[cur], (size_t)s.K * WW * 16, kind, st));
  W90G_CHECK(cudaStreamSynchronize(st));
  return 0;
}

int Engine::init_states(std::string& err) {
  cudaStream_t st = stream();
  for (size_t p = 0; p < hprobs_.size(); ++p) {
    CtrlState h;
    std::memset(&h, 0, sizeof(h));
    h.cur = 0;
    h.first_pass = 1;
    h.lfirst = 1;
    // wann_main starts from old_spread%om_tot = 0 (src/wannierise.F90:475)
    W90G_CHECK(cudaMemcpyAsync(hprobs_[p].st, &h, sizeof(h), cudaMemcpyHostToDevice, st));
    const auto& s = specs_[p];
    W90G_CHECK(cudaMemsetAsync(hprobs_[p].D, 0, (size_t)s.K * s.W * s.W * 16, st));
    if (s.guiding) {
      // centres from the projections; sheet 0 (csheet 1) until the first wann_phases
      const size_t n = (size_t)s.K * s.B * s.W;
      guide_init_.assign(2 * n, 0.0);
      for (size_t i = 0; i < n; ++i) guide_init_[2 * i] = 1.0;
      W90G_CHECK(cudaMemcpyAsync(hprobs_[p].rguide, s.rguide0.data(), s.rguide0.size() * 8, cudaMemcpyHostToDevice, st));
      W90G_CHECK(cudaMemsetAsync(hprobs_[p].sheet, 0, n * 8, st));
      W90G_CHECK(cudaMemcpyAsync(hprobs_[p].csheet, guide_init_.data(), n * 16, cudaMemcpyHostToDevice, st));
      W90G_CHECK(cudaStreamSynchronize(st));
    }
  }
  return 0;
}

int Engine::project(std::string& err) {
  cudaStream_t st = stream();
  launches_ = 0;
  if (int rc0 = init_states(err)) return rc0;
  const int ws = std::max(maxW_small_, 1);
  const WorkMap wmk{d_offs_k_, nprob()};
  const WorkMap wmkb{d_offs_kb_, nprob()};
  // The polar factors on the tensor cores from num_wann 9 on (project of 1000 k: W = 9 and
  // above; narrower ones fill little of a 128-row tile and their FP64 form is the faster one);
  // k_lowdin takes what is left.  Work: the second M buffer, which the projection does not use.
  W90G_CHECK(cudaMemsetAsync(d_status_, 0, n_k_ * sizeof(int), st));
  if (nprob() == 1 && specs_[0].W >= kPolarMinW && specs_[0].W <= kPolarMaxN && specs_[0].B >= kPolarMats) {
    const size_t W = specs_[0].W, WW = W * W;
    PolarArgs a{};
    a.x = a.q = hprobs_[0].U[0];
    a.ldx = a.ldq = a.qrows = a.cols = a.n = (int)W;
    a.strideX = a.strideQ = WW;
    a.work = hprobs_[0].M[1];
    a.strideW = kPolarMats * WW;
    a.status = d_status_;
    W90G_CHECK(oz_polar_launch(a, n_k_, st));
    launches_ += 1;
  }
  k_lowdin<<<n_k_, 256, 4 * ws * ws * 16, st>>>(dprobs_, wmk, d_status_);
  W90G_CHECK(cudaGetLastError());
  launches_ += 1;
  // symmetry-adapted initial U (src/overlap.F90:901-905)
  if (n_ir_) {
    k_sym_u<<<n_ir_, 256, 0, st>>>(dprobs_, WorkMap{d_offs_ir_, nprob()});
    W90G_CHECK(cudaGetLastError());
    launches_ += 1;
  }
  std::vector<int> status(n_k_);
  W90G_CHECK(cudaMemcpyAsync(status.data(), d_status_, n_k_ * sizeof(int), cudaMemcpyDeviceToHost, st));
  W90G_CHECK(cudaStreamSynchronize(st));
  for (int i = 0; i < n_k_; ++i) {
    if (status[i] == 1) {
      err = "Error in overlap_project: A(k) is rank deficient at k-point " + std::to_string(i + 1);
      return 1;
    }
    if (status[i] == 2) {
      err = "Error in overlap_project: Jacobi eigensolver did not converge at k-point " + std::to_string(i + 1);
      return 1;
    }
  }
  for (size_t p = 0; p < hprobs_.size(); ++p) {
    const int nir = hprobs_[p].sym_nir;
    if (nir <= 0) continue;
    std::vector<int> ss(nir);
    W90G_CHECK(cudaMemcpy(ss.data(), hprobs_[p].sym_status, nir * sizeof(int), cudaMemcpyDeviceToHost));
    for (int ir = 0; ir < nir; ++ir) {
      if (ss[ir] == 1) {
        // set_error_unconv (src/sitesym.F90:478-486)
        err = "symmetrize_ukirr: not converged";
        return -1;
      }
      if (ss[ir] == 2) {
        err = " ERROR: IN ZGESVD IN orthogonalize_u";
        return 1;
      }
    }
  }
  // M <- U^H M U': tensor cores from num_wann 9 on where the second M buffer, which the projection does
  // not use, holds the work matrices of kRotateCtas CTAs (1216 blocks and more); smaller meshes keep
  // the FP64 kernel
  const ProblemSpec& s0 = specs_[0];
  const size_t mat = (size_t)s0.W * s0.W;
  if (nprob() == 1 && s0.W >= kPolarMinW && s0.W <= kPolarMaxN &&
      (size_t)s0.K * s0.B * mat >= (size_t)std::min(kRotateCtas, s0.K * s0.B) * 4 * mat) {
    RotateArgs r{};
    r.m = r.out = hprobs_[0].M[0];
    r.ldm = r.ldv = r.w = r.n = s0.W;
    r.strideM = r.strideV = mat;
    r.v = hprobs_[0].U[0];
    r.B = s0.B;
    r.nnlist = hprobs_[0].nnlist;
    r.work = hprobs_[0].M[1];
    r.ctas = kRotateCtas;
    r.failed = d_status_;
    W90G_CHECK(cudaMemsetAsync(d_status_, 0, sizeof(int), st));
    W90G_CHECK(oz_rotate_launch(r, s0.K * s0.B, st));
    int failed = 0;
    W90G_CHECK(cudaMemcpyAsync(&failed, d_status_, sizeof(int), cudaMemcpyDeviceToHost, st));
    W90G_CHECK(cudaStreamSynchronize(st));
    if (failed) {
      err = "overlap_project: a bounded wait of the tensor-core rotation ran out";
      return 1;
    }
  } else {
    k_m_update<<<n_kb_, 256, 4 * ws * ws * 16, st>>>(dprobs_, wmkb, 1, 0);
    W90G_CHECK(cudaGetLastError());
  }
  launches_ += 1;
  return 0;
}

void Engine::launch_omega(cudaStream_t s, int slot) {
  const int np = nprob();
  const WorkMap wmc{d_offs_chunk_, np};
  k_omega_p1<<<n_chunk_, 256, 0, s>>>(dprobs_, wmc, slot);
  if (!(slot & kOmegaFused) || omega_two_) k_omega_p2<<<n_chunk_, 256, 0, s>>>(dprobs_, wmc, slot);
}

// tensor path: keep the entry M and U, iterate on R = U0^H U starting from identity
int Engine::prepare_tensor(cudaStream_t st, std::string& err) {
  if (!tensor_wp_) return 0;
  for (int p = 0; p < nprob(); ++p) {
    const auto& s = specs_[p];
    const size_t WW = (size_t)s.W * s.W;
    W90G_CHECK(cudaMemcpyAsync(hprobs_[p].M0, hprobs_[p].M[0], (size_t)s.K * s.B * WW * 16,
                               cudaMemcpyDeviceToDevice, st));
    W90G_CHECK(cudaMemcpyAsync(hprobs_[p].U0, hprobs_[p].U[0], (size_t)s.K * WW * 16, cudaMemcpyDeviceToDevice, st));
  }
  const WorkMap wmk{d_offs_k_, nprob()};
  k_u_identity<<<n_k_, 256, 0, st>>>(dprobs_, wmk);
  W90G_CHECK(cudaGetLastError());
  // step 1's A operand (the entry overlaps) in digit planes, once per solve
  W90G_CHECK(tiles3_ ? oz3_preslice_launch(tensor_wp_, dprobs_, wmk, n_k_, tiles3_, st)
                    : (pipe_ ? oz2_preslice_launch(tensor_wp_, dprobs_, wmk, n_k_, st)
                             : oz_preslice_launch(tensor_wp_, dprobs_, wmk, n_k_, st)));
  launches_ += 2;
  return 0;
}

void Engine::launch_mupdate(cudaStream_t s, int which) {
  const int np = nprob();
  const WorkMap wmk{d_offs_k_, np};
  const WorkMap wmkb{d_offs_kb_, np};
  if (tiles3_) {
    oz3_launch(tensor_wp_, dprobs_, wmk, which, n_k_, tiles3_, slabs_, s);
  } else if (pipe_) {
    oz2_launch(tensor_wp_, 1, dprobs_, wmk, which, n_k_, s);
    oz2_launch(tensor_wp_, 2, dprobs_, wmk, which, n_k_, s);
  } else if (tensor_wp_) {
    oz_launch(tensor_wp_, 1, dprobs_, wmk, which, n_k_, s);
    oz_launch(tensor_wp_, 2, dprobs_, wmk, which, n_k_, s);
  } else {
    const int ws = std::max(maxW_small_, 1);
    k_m_update<<<n_kb_, 256, (size_t)4 * ws * ws * 16, s>>>(dprobs_, wmkb, 0, which);
  }
}

void Engine::launch_exp(cudaStream_t s, int which) {
  const WorkMap wmk{d_offs_k_, nprob()};
  if (tensor_exp_) {
    oz_exp_launch(tensor_wp_, exp_smem_ ? 1 : 0, dprobs_, wmk, which, n_k_, s);
  } else {
    const int ws = std::max(maxW_small_, 1);
    k_exp_u<<<n_k_, 256, (size_t)6 * ws * ws * 16, s>>>(dprobs_, wmk, which);
  }
}

// k_ctrl_search in the gradient's last CTA: where nothing comes between the two, and up to 512 CTAs --
// a launch saved is 5 to 9 us there; on 1000 k of num_wann 32 counting the CTAs in costs as much
// (6.59 ms against 6.54 for the solve's four iterations)
bool Engine::fuse_search() const { return !n_ir_ && !pc_tiles_ && n_grad_ <= 512; }

void Engine::launch_iteration(cudaStream_t s) {
  const int np = nprob();
  const int ws = std::max(maxW_small_, 1);
  const WorkMap wmk{d_offs_k_, np};
  const WorkMap wmkb{d_offs_kb_, np};
  const WorkMap wmg{d_offs_grad_, np};
  if (guide_w_) k_phases<<<dim3(guide_w_, np), 256, 0, s>>>(dprobs_, 1);
  if (!fuse_search()) {
    k_grad<<<n_grad_, 256, 0, s>>>(dprobs_, wmg);
    if (n_ir_) k_sym_grad<<<n_ir_, 256, 0, s>>>(dprobs_, WorkMap{d_offs_ir_, np});
    if (pc_tiles_) {
      k_precond<<<dim3(pc_tiles_, np), 256, 0, s>>>(dprobs_, 0);
      k_precond<<<dim3(pc_tiles_, np), 256, 0, s>>>(dprobs_, 1);
    }
    k_ctrl_search<<<np, 256, 0, s>>>(dprobs_);
    if (n_ir_) k_sym_dir<<<n_ir_, 256, 0, s>>>(dprobs_, WorkMap{d_offs_ir_, np});
  } else {
    k_grad_search<<<n_grad_, 256, 0, s>>>(dprobs_, wmg);
  }
  // (k_ctrl_step and k_ctrl_end run in the spread passes' last CTAs)
  launch_exp(s, 0);
  launch_mupdate(s, 0);
  launch_omega(s, kOmegaFused);
  launch_exp(s, 1);
  launch_mupdate(s, 1);
  launch_omega(s, kOmegaFused + 1);
}

int Engine::begin(std::string& err) {
  cudaStream_t st = stream();
  launches_ = 0;
  launched_iters_ = 0;
  const int np = nprob();
  if (init_states(err)) return 1;
  const WorkMap wmkb{d_offs_kb_, np};
  if (int rc0 = prepare_tensor(st, err)) return rc0;
  // guiding centres before the loop (src/wannierise.F90:435-443)
  if (guide_w_) {
    k_phases<<<dim3(guide_w_, np), 256, 0, st>>>(dprobs_, 0);
    launches_ += 1;
  }
  // initial spread (src/wannierise.F90:452-470)
  k_mdiag<<<n_kb_, 128, 0, st>>>(dprobs_, wmkb);
  launch_omega(st, 2);
  k_log_init<<<np, 128, 0, st>>>(dprobs_);
  W90G_CHECK(cudaGetLastError());
  launches_ += 4;
  // capture one iteration into a graph (once per arena layout)
  if (!graph_exec_) {
    cudaStream_t cap;
    W90G_CHECK(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    cudaGraph_t g;
    W90G_CHECK(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    launch_iteration(cap);
    W90G_CHECK(cudaStreamEndCapture(cap, &g));
    W90G_CHECK(cudaGraphInstantiate(&graph_exec_, g, 0));
    cudaGraphDestroy(g);
    cudaStreamDestroy(cap);
    graph_stream_ = st;
  }
  return 0;
}

int Engine::advance(int n, int* d_flag, std::string& err) {
  cudaStream_t st = stream();
  n = std::min(n, max_iter_ - launched_iters_);
  for (int i = 0; i < n; ++i) W90G_CHECK(cudaGraphLaunch(graph_exec_, st));
  // grad, search (or in grad's last CTA), 2 x (exp, M update, 1 or 2 spread passes); precond and
  // symmetry: 2 each
  launches_ += (1LL + 2 * (1 + (tiles3_ ? 2 + 2 * slabs_ : (tensor_wp_ ? 2 : 1)) + (omega_two_ ? 2 : 1)) + (pc_tiles_ ? 2 : 0) +
                (n_ir_ ? 2 : 0) + (fuse_search() ? 0 : 1) + (guide_w_ ? 1 : 0)) *
               std::max(n, 0);
  launched_iters_ += std::max(n, 0);
  if (d_flag) {
    // every problem done (converged or out of iterations) -> *d_flag = 1
    k_all_done<<<1, 256, 0, st>>>(dprobs_, nprob(), d_flag);
    W90G_CHECK(cudaGetLastError());
    launches_ += 1;
  }
  return 0;
}

int Engine::wannierise(std::string& err) {
  cudaStream_t st = stream();
  if (int rc0 = begin(err)) return rc0;
  int* d_alldone = (int*)((char*)d_unit_ + align_up(n_k_ * sizeof(double)));
  int any_window = 0;
  for (const auto& s : specs_) any_window |= (s.ctl.conv_window > 1);
  int chunk = 4;
  int hdone = 0;
  while (launched_iters_ < max_iter_) {
    const int n = std::min(chunk, max_iter_ - launched_iters_);
    const bool poll = any_window && (launched_iters_ + n) < max_iter_;
    if (int rc0 = advance(n, poll ? d_alldone : nullptr, err)) return rc0;
    if (poll) {
      W90G_CHECK(cudaMemcpyAsync(&hdone, d_alldone, sizeof(int), cudaMemcpyDeviceToHost, st));
      W90G_CHECK(cudaStreamSynchronize(st));
      if (hdone) break;
      chunk = std::min(chunk * 2, 32);
    }
  }
  return finish(err);
}

int Engine::finish(std::string& err) {
  cudaStream_t st = stream();
  const int np = nprob();
  const WorkMap wmk{d_offs_k_, np};
  if (tensor_wp_) {
    W90G_CHECK(oz_ufinal_launch(tensor_wp_, dprobs_, wmk, n_k_, st));
    launches_ += 1;
  }
  // final unitarity check (src/wannierise.F90:890-892)
  k_unitarity<<<n_k_, 256, 0, st>>>(dprobs_, wmk, d_unit_);
  W90G_CHECK(cudaGetLastError());
  launches_ += 1;
  std::vector<double> unit(n_k_);
  W90G_CHECK(cudaMemcpyAsync(unit.data(), d_unit_, n_k_ * sizeof(double), cudaMemcpyDeviceToHost, st));
  std::vector<CtrlState> hs(np);
  for (int p = 0; p < np; ++p)
    W90G_CHECK(cudaMemcpyAsync(&hs[p], hprobs_[p].st, sizeof(CtrlState), cudaMemcpyDeviceToHost, st));
  W90G_CHECK(cudaStreamSynchronize(st));
  std::vector<int> offs_k(np + 1, 0);
  for (int p = 0; p < np; ++p) offs_k[p + 1] = offs_k[p] + specs_[p].K;
  int rc = 0;
  for (int p = 0; p < np; ++p) {
    ProblemResult& R = results_[p];
    const auto& s = specs_[p];
    const CtrlState& S = hs[p];
    R.niter = S.iter;
    R.converged = S.lconverged;
    R.error = S.error;
    R.spread = S.wann;
    const int W = s.W;
    std::vector<double> cen(4 * W);
    W90G_CHECK(cudaMemcpyAsync(cen.data(), hprobs_[p].centres + 2 * 4 * W, 4 * W * 8, cudaMemcpyDeviceToHost, st));
    R.log.assign((size_t)(S.iter + 1) * kLogStride, 0.0);
    R.log_centres.assign((size_t)(S.iter + 1) * 4 * W, 0.0);
    W90G_CHECK(cudaMemcpyAsync(R.log.data(), hprobs_[p].log, R.log.size() * 8, cudaMemcpyDeviceToHost, st));
    W90G_CHECK(cudaMemcpyAsync(R.log_centres.data(), hprobs_[p].log_centres, R.log_centres.size() * 8,
                               cudaMemcpyDeviceToHost, st));
    W90G_CHECK(cudaStreamSynchronize(st));
    R.centres.assign(3 * W, 0.0);
    R.spreads.assign(W, 0.0);
    for (int n = 0; n < W; ++n) {
      for (int i = 0; i < 3; ++i) R.centres[n * 3 + i] = cen[i * W + n];
      R.spreads[n] = cen[3 * W + n];
    }
    double ue = 0.0;
    for (int k = offs_k[p]; k < offs_k[p + 1]; ++k) ue = std::max(ue, unit[k]);
    R.unitarity_err = ue;
  }
  // per-problem failures (non-finite spread, unitarity) are reported through result(p);
  // a non-zero return means the engine itself failed (CUDA error or allocation)
  return rc;
}

int Engine::wannierise_profiled(int max_iters, double* ms, int* cnt, std::string& err) {
  cudaStream_t st = stream();
  launches_ = 0;
  const int np = nprob();
  if (int rc0 = init_states(err)) return rc0;
  if (int rc0 = prepare_tensor(st, err)) return rc0;
  for (int i = 0; i < kPNum; ++i) {
    ms[i] = 0.0;
    cnt[i] = 0;
  }
  const int ws = std::max(maxW_small_, 1);
  const WorkMap wmk{d_offs_k_, np};
  const WorkMap wmkb{d_offs_kb_, np};
  const WorkMap wmg{d_offs_grad_, np};
  cudaEvent_t e0, e1;
  W90G_CHECK(cudaEventCreate(&e0));
  W90G_CHECK(cudaEventCreate(&e1));
  auto timed = [&](int kind, auto&& launch) -> int {
    W90G_CHECK(cudaEventRecord(e0, st));
    launch();
    W90G_CHECK(cudaGetLastError());
    W90G_CHECK(cudaEventRecord(e1, st));
    W90G_CHECK(cudaEventSynchronize(e1));
    float t = 0.f;
    W90G_CHECK(cudaEventElapsedTime(&t, e0, e1));
    ms[kind] += t;
    cnt[kind] += 1;
    ++launches_;
    return 0;
  };
  int rc = 0;
  rc |= timed(kPInit, [&] {
    if (guide_w_) k_phases<<<dim3(guide_w_, np), 256, 0, st>>>(dprobs_, 0);
    k_mdiag<<<n_kb_, 128, 0, st>>>(dprobs_, wmkb);
    launch_omega(st, 2);
    k_log_init<<<np, 128, 0, st>>>(dprobs_);
  });
  CtrlState hs;
  const int iters = std::min(max_iters, max_iter_);
  for (int it = 0; it < iters && !rc; ++it) {
    if (guide_w_) rc |= timed(kPInit, [&] { k_phases<<<dim3(guide_w_, np), 256, 0, st>>>(dprobs_, 1); });
    // the launches of launch_iteration
    if (fuse_search()) {
      rc |= timed(kPGrad, [&] { k_grad_search<<<n_grad_, 256, 0, st>>>(dprobs_, wmg); });
    } else {
      rc |= timed(kPGrad, [&] {
        k_grad<<<n_grad_, 256, 0, st>>>(dprobs_, wmg);
        if (n_ir_) k_sym_grad<<<n_ir_, 256, 0, st>>>(dprobs_, WorkMap{d_offs_ir_, np});
      });
      if (pc_tiles_) {
        rc |= timed(kPPrecond, [&] { k_precond<<<dim3(pc_tiles_, np), 256, 0, st>>>(dprobs_, 0); });
        rc |= timed(kPPrecond, [&] { k_precond<<<dim3(pc_tiles_, np), 256, 0, st>>>(dprobs_, 1); });
      }
      rc |= timed(kPCtrlSearch, [&] {
        k_ctrl_search<<<np, 256, 0, st>>>(dprobs_);
        if (n_ir_) k_sym_dir<<<n_ir_, 256, 0, st>>>(dprobs_, WorkMap{d_offs_ir_, np});
      });
    }
    rc |= timed(kPExpU, [&] { launch_exp(st, 0); });
    rc |= timed(kPMUpdate, [&] { launch_mupdate(st, 0); });
    rc |= timed(kPOmega, [&] { launch_omega(st, kOmegaFused); });
    W90G_CHECK(cudaMemcpy(&hs, hprobs_[0].st, sizeof(CtrlState), cudaMemcpyDeviceToHost));
    if (hs.do_second) {
      rc |= timed(kPExpU, [&] { launch_exp(st, 1); });
      rc |= timed(kPMUpdate, [&] { launch_mupdate(st, 1); });
      rc |= timed(kPOmega, [&] { launch_omega(st, kOmegaFused + 1); });
    } else {
      launch_omega(st, kOmegaFused + 1);   // the iteration's end alone
    }
    W90G_CHECK(cudaMemcpy(&hs, hprobs_[0].st, sizeof(CtrlState), cudaMemcpyDeviceToHost));
    if (hs.done) break;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  W90G_CHECK(cudaMemcpy(&hs, hprobs_[0].st, sizeof(CtrlState), cudaMemcpyDeviceToHost));
  last_exp_products_ = hs.exp_products;
  return rc;
}

// FP64 pipe probe: returns TFLOP/s of a dependent-chain DFMA loop over all SMs.
int measure_fp64_peak(double* tflops, std::string& err) {
  int dev = 0, sms = 0;
  W90G_CHECK(cudaGetDevice(&dev));
  W90G_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  double* d = nullptr;
  W90G_CHECK(cudaMalloc(&d, 64));
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t e0, e1;
  W90G_CHECK(cudaEventCreate(&e0));
  W90G_CHECK(cudaEventCreate(&e1));
  k_fp64_peak<<<blocks, threads>>>(d, 64, 1.0);   // warm-up
  W90G_CHECK(cudaEventRecord(e0));
  k_fp64_peak<<<blocks, threads>>>(d, iters, 1.0);
  W90G_CHECK(cudaEventRecord(e1));
  W90G_CHECK(cudaEventSynchronize(e1));
  float ms = 0.f;
  W90G_CHECK(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(d);
  const double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return 0;
}

}  // namespace w90g
