// SIMT emulation of the iteration as a solve launches it (Engine::launch_iteration on the FP64 path):
// k_grad_search, and the spread passes with the control steps in their last CTAs -- one launch for
// problems of at most kOmegaOneCta statistics, two for others -- over several problems at once, beside
// the same iteration one kernel at a time.  See emu_iter.cpp for the emulation.
#include <algorithm>
#include <memory>

#include "emu_fibers.h"

#include "k_fp64_emu.cu"

namespace {

// one problem's arrays
struct Emu {
  std::vector<double2> M[2], U[2], G, D, dU;
  std::vector<double> dln, dab, offd, gpart, cen, log, logc, op1, op2, bk, wb;
  std::vector<int> nn;
  w90g::CtrlState st{};
  w90g::Problem P{};
  Emu(int W, int K, int B, const int* nnlist, const double* bkp, const double* wbp, double wbtot, const double* Mp,
      const double* Up, int num_iter, int conv_window, double conv_tol, int per) {
    const size_t WW = (size_t)W * W, KB = (size_t)K * B;
    const int nt = (W + 31) / 32;
    for (int i = 0; i < 2; ++i) {
      M[i].resize(KB * WW);
      U[i].resize(K * WW);
      P.M[i] = M[i].data();
      P.U[i] = U[i].data();
    }
    std::memcpy(M[0].data(), Mp, KB * WW * 16);
    std::memcpy(U[0].data(), Up, K * WW * 16);
    auto set = [](auto& v, size_t n, auto*& p) {
      v.resize(n);
      p = v.data();
    };
    set(G, K * WW, P.G);
    set(D, K * WW, P.D);
    set(dU, K * WW, P.dU);
    set(dln, KB * W, P.diag_ln);
    set(dab, KB * W, P.diag_abs2);
    set(offd, KB, P.offd);
    set(gpart, (size_t)K * nt * nt * 2, P.gpart);
    set(cen, 12 * W, P.centres);
    set(log, (size_t)(num_iter + 1) * w90g::kLogStride, P.log);
    set(logc, (size_t)(num_iter + 1) * 4 * W, P.log_centres);
    P.nchunk = (int)((KB + per - 1) / per);
    set(op1, (size_t)P.nchunk * (4 * W + 2), P.opart1);
    set(op2, P.nchunk, P.opart2);
    nn.assign(nnlist, nnlist + KB);
    bk.assign(bkp, bkp + KB * 3);
    wb.assign(wbp, wbp + B);
    P.nnlist = nn.data();
    P.bk = bk.data();
    P.wb = wb.data();
    P.W = W;
    P.K = K;
    P.B = B;
    P.wbtot = wbtot;
    P.ctl.num_iter = num_iter;
    P.ctl.num_cg_steps = 5;
    P.ctl.conv_window = conv_window;
    P.ctl.conv_tol = conv_tol;
    P.ctl.trial_step = 2.0;
    P.ctl.conv_noise_amp = -1.0;
    st.first_pass = 1;
    st.lfirst = 1;
  }
};

}  // namespace

extern "C" {

// Arrays of nprob pointers and sizes; per: blocks (k,b) per spread chunk.  fused: launch_iteration's
// order, else one kernel per step.  log (nprob pointers): (num_iter + 1) x kLogStride each; rows[p].
int emu_solve(int nprob, const int* W, const int* K, const int* B, const int** nnlist, const double** bk,
              const double** wb, const double* wbtot, const double** M, const double** U, int num_iter,
              int conv_window, double conv_tol, int per, int fused, double** log, double** U_out, int* rows) {
  using namespace w90g;
  std::vector<std::unique_ptr<Emu>> e;
  std::vector<Problem> P;
  std::vector<int> ok(1, 0), okb(1, 0), og(1, 0), oc(1, 0);
  int smax = 0, two = 0;
  for (int p = 0; p < nprob; ++p) {
    e.emplace_back(new Emu(W[p], K[p], B[p], nnlist[p], bk[p], wb[p], wbtot[p], M[p], U[p], num_iter, conv_window,
                           conv_tol, per));
    e[p]->P.st = &e[p]->st;
    P.push_back(e[p]->P);
    const int nt = (W[p] + 31) / 32;
    ok.push_back(ok[p] + K[p]);
    okb.push_back(okb[p] + K[p] * B[p]);
    og.push_back(og[p] + K[p] * nt * nt);
    oc.push_back(oc[p] + P[p].nchunk);
    smax = std::max(smax, W[p]);
    two = two || K[p] * B[p] * W[p] > kOmegaOneCta;
  }
  Problem* pp = P.data();
  const WorkMap wk{ok.data(), nprob}, wkb{okb.data(), nprob}, wg{og.data(), nprob}, wc{oc.data(), nprob};
  const size_t sm4 = (size_t)4 * smax * smax * 16, sm6 = (size_t)6 * smax * smax * 16;
  auto omega = [&](int slot) {
    launch(oc.back(), 256, 0, [&] { k_omega_p1(pp, wc, slot); });
    if (!(slot & kOmegaFused) || two) launch(oc.back(), 256, 0, [&] { k_omega_p2(pp, wc, slot); });
  };
  launch(okb.back(), 128, 0, [&] { k_mdiag(pp, wkb); });
  omega(2);
  launch(nprob, 128, 0, [&] { k_log_init(pp); });
  const int f = fused ? kOmegaFused : 0;
  for (int it = 0; it < num_iter; ++it) {
    if (fused) {
      launch(og.back(), 256, 0, [&] { k_grad_search(pp, wg); });
    } else {
      launch(og.back(), 256, 0, [&] { k_grad(pp, wg); });
      launch(nprob, 256, 0, [&] { k_ctrl_search(pp); });
    }
    launch(ok.back(), 256, sm6, [&] { k_exp_u(pp, wk, 0); });
    launch(okb.back(), 256, sm4, [&] { k_m_update(pp, wkb, 0, 0); });
    omega(f);
    if (!fused) launch(1, 128, 0, [&] { k_ctrl_step(pp, nprob); });
    launch(ok.back(), 256, sm6, [&] { k_exp_u(pp, wk, 1); });
    launch(okb.back(), 256, sm4, [&] { k_m_update(pp, wkb, 0, 1); });
    omega(f + 1);
    if (!fused) launch(nprob, 128, 0, [&] { k_ctrl_end(pp); });
  }
  for (int p = 0; p < nprob; ++p) {
    const CtrlState& st = e[p]->st;
    if (st.error) return st.error;
    // the arrival counts are back to zero, whichever CTA came last
    if (st.omega_arrive[0] || st.omega_arrive[1] || st.grad_arrive) return -1;
    rows[p] = st.iter + 1;
    std::memcpy(log[p], e[p]->log.data(), (size_t)rows[p] * kLogStride * 8);
    std::memcpy(U_out[p], P[p].U[st.cur], (size_t)K[p] * W[p] * W[p] * 16);
  }
  return 0;
}

}  // extern "C"
