// SIMT emulation of the disentanglement as dis_run launches it below the width of the tensor-core
// steps: the frozen states' part of Z formed once (k_dis_zfroz), U_opt U0 formed before one rotation
// (k_dis_v), k_dis_step with its own number of threads.  emu_dis.cpp's emu_dis_plain runs the forms
// that these replace.
#include "emu_dis.cpp"

extern "C" int emu_dis_engine(int nb, int W, int K, int B, const int* nnlist, const double* wb, double wbtot,
                              const double* eig, const double* Mraw, const double* A, int num_iter, double mix,
                              double win_min, double win_max, int frozen, double froz_min, double froz_max,
                              int threads, int step_threads, double* log_out, double* U0_out, double* M0_out,
                              double* Uopt_out, int* status_out) {
  using namespace w90g;
  DisControl c;
  c.win_min = win_min;
  c.win_max = win_max;
  c.frozen_states = frozen != 0;
  c.froz_min = froz_min;
  c.froz_max = froz_max;
  std::vector<int> ndim, nfirst, nfroz, ffirst, nfidx;
  std::vector<double> eigw;
  std::string err;
  if (int rc = dis_windows(c, eig, nb, W, K, ndim, nfirst, nfroz, ffirst, nfidx, eigw, err)) return -100 - rc;
  const size_t NN = (size_t)nb * nb, WW = (size_t)W * W;
  std::vector<int> nn(nnlist, nnlist + (size_t)K * B), st(K, 0), ps(K, 0), sw(1, 0);
  std::vector<double> wbv(wb, wb + B), wk1(K), wk(K);
  std::vector<double2> mraw((size_t)K * B * NN), mw((size_t)K * B * NN), a((size_t)K * nb * W), u0b((size_t)K * nb * W),
      u1b((size_t)K * nb * W), zin((size_t)K * NN), zout((size_t)K * NN), uw((size_t)K * WW), m0((size_t)K * B * WW),
      ws((size_t)K * kWs * NN), vz((size_t)K * NN);
  std::memcpy(mraw.data(), Mraw, mraw.size() * 16);
  std::memcpy(u0b.data(), A, u0b.size() * 16);
  DisDev D{};
  D.nb = nb;
  D.W = W;
  D.K = K;
  D.B = B;
  D.wbtot = wbtot;
  D.mix = mix;
  D.nnlist = nn.data();
  D.wb = wbv.data();
  D.ndim = ndim.data();
  D.nfirst = nfirst.data();
  D.nfroz = nfroz.data();
  D.ffirst = ffirst.data();
  D.nfidx = nfidx.data();
  D.eig = eigw.data();
  D.Mraw = mraw.data();
  D.Mw = mw.data();
  D.A = a.data();
  D.U[0] = u0b.data();
  D.U[1] = u1b.data();
  D.Zin = zin.data();
  D.Zout = zout.data();
  D.U0 = uw.data();
  D.M0 = m0.data();
  D.ws = ws.data();
  D.wk1 = wk1.data();
  D.wk = wk.data();
  D.status = st.data();
  D.pstat = ps.data();
  D.Vz = vz.data();
  D.max_sweeps = sw.data();
  D.V = ws.data() + 6 * NN;
  bool any_froz = false;
  int mmax = 0;
  for (int k = 0; k < K; ++k) {
    any_froz = any_froz || nfroz[k] > 0;
    mmax = std::max(mmax, ndim[k] - nfroz[k]);
  }
  if (any_froz) D.zfroz = ws.data() + 7 * NN;
  const size_t step_smem = 3 * (size_t)mmax * mmax * 16;
  launch(K, threads, 0, [&] { k_dis_project(D); });
  if (any_froz) launch(K, threads, 0, [&] { k_dis_froz(D); });
  if (any_froz) launch(K, threads, 0, [&] { k_dis_zfroz(D); });
  int cur = 0;
  launch(K, threads, 0, [&] { k_dis_z(D, cur, 1, 0); });
  for (int it = 1; it <= num_iter; ++it) {
    launch(K, step_threads, step_smem, [&] { k_dis_step(D, cur, it); });
    launch(K, threads, 0, [&] { k_dis_z(D, cur ^ 1, 0, 1); });
    cur ^= 1;
    double w1 = 0.0, w2 = 0.0;
    for (int k = 0; k < K; ++k) {
      w1 += wk1[k];
      w2 += wk[k];
    }
    log_out[3 * (it - 1)] = it;
    log_out[3 * (it - 1) + 1] = w1 / K;
    log_out[3 * (it - 1) + 2] = w2 / K;
  }
  launch(K, threads, 0, [&] { k_dis_gauge(D, cur); });
  launch(K, threads, 0, [&] { k_dis_findu(D, cur); });
  launch(K, threads, 0, [&] { k_dis_v(D, cur); });
  launch(K * B, threads, ((size_t)W * nb + 2 * WW) * 16, [&] { k_dis_rotate(D, cur); });
  status_out[0] = 0;
  for (int k = 0; k < K && !status_out[0]; ++k) status_out[0] = st[k];
  std::memcpy(U0_out, uw.data(), uw.size() * 16);
  std::memcpy(M0_out, m0.data(), m0.size() * 16);
  std::memcpy(Uopt_out, D.U[cur], u0b.size() * 16);
  return 0;
}
