// Host execution of the complex128 Wigner2D passes on the register-blocked
// transform (csrc/wig_wigner.cuh: xpass_blk_body, ppass_blk_body, the ODM and
// Gross-Pitaevskii kernels) in the launch sequence of wig_run.  The tile macros
// WIG_BXR, WIG_BXE, WIG_BPC, WIG_BPE (and WIG_OXR, WIG_OPC, WIG_OE) come from the
// command line, with WIG_BX = WIG_BP = 1.  wigner2d_helpers.h: wigner2d_emu.cpp up to
// its main(), written by tests/test_blocked_cpu.py, which builds this.
//
//   blocked_emu W_in W_out obs_out n_prop x_amp p_amp dt gamma d_theta d_lambda odm a_gp
#include "wigner2d_helpers.h"

int main(int argc, char** argv) {
  if (argc != 13) return 2;
  constexpr int NX = WIG_NX, NP = WIG_NP, NOBS = 11;
  const long n_prop = std::atol(argv[4]);
  const double xa = std::atof(argv[5]), pa = std::atof(argv[6]), gamma = std::atof(argv[8]), a_gp = std::atof(argv[12]);
  const int odm = std::atoi(argv[11]);
  dt = std::atof(argv[7]);
  D_Theta = std::atof(argv[9]);
  D_Lambda = std::atof(argv[10]);
  mass = hBar = 1.;
  dx = 2. * xa / NX;
  dp = 2. * pa / NP;
  dtheta = 2. * M_PI / (2. * pa);
  dlambda = 2. * M_PI / (2. * xa);
  const size_t npts = (size_t)NX * NP;
  std::vector<double2> W(npts);
  if (!read_all(argv[1], W.data(), npts * sizeof(double2))) return 4;
  const auto pad = [](int n, int e) { return n + n / std::min(e, 8); };
  const int gx = NP / WIG_BXR, xnt = WIG_BXR * (NX / WIG_BXE), gp = NX / WIG_BPC, pnt = WIG_BPC * (NP / WIG_BPE);
  const size_t smx = (size_t)WIG_BXR * (pad(NX, WIG_BXE) + wig::blk_pre_slots(NX, WIG_BXE)) * sizeof(double2);
  const size_t smp = (size_t)WIG_BPC * (wig::blk_stride(pad(NP, WIG_BPE), WIG_BPC) + wig::blk_pre_slots(NP, WIG_BPE)) * sizeof(double2);
  const int n_cta_r = clampi(NX * NP / (4 * WIG_RNT), 1, 296);
  wig::WigArgs a{};
  a.dt = dt; a.dx = dx; a.dp = dp; a.dtheta = dtheta; a.dlambda = dlambda; a.mass = mass; a.hbar = hBar;
  a.D_theta = D_Theta; a.D_lambda = D_Lambda;
  a.dX = dx; a.dP = dp; a.mass_exact = mass;
  const double g = dt * gamma, c1 = 2. / 3. * g, c2 = g, c3 = 2. * g;
  a.cl_k1 = make_double2(0., c1 + c2 != 0. ? c1 * c2 / (c1 + c2) : 0.);
  a.cl_k12 = make_double2(0., c1 + c2);
  a.cl_c3 = make_double2(0., c3);
  std::vector<double> xt = shifted_range(xa, NX), pt = shifted_range(pa, NP);
  std::vector<double> tht = shifted_range(dtheta * NP / 2., NP), ths(NP), lt = shifted_range(dlambda * NX / 2., NX);
  for (int i = 0; i < NP; ++i) ths[i] = tht[i] * (1.0 / (double)NP);
  const UserPhys ph{};
  std::vector<double> dv(NX), v0(NX), rl(NX), rt(NP), m1(NX), m2(NX), sfp(NP), rth(NP);
  for (int k = 0; k < NX; ++k) { dv[k] = ph.DPotential(0., xt[k]); v0[k] = ph.Potential(0., xt[k]); }
  std::vector<double2> twx = wighost::block_twiddles(NX, WIG_BXE), twp = wighost::block_twiddles(NP, WIG_BPE);
  std::vector<double> partials((size_t)std::max(std::max(gp, NX), n_cta_r) * wig::NACC), part_im((size_t)NX * wig::NIM);
  std::vector<double> obs((size_t)(n_prop + 1) * NOBS, 0.);
  a.x_tab = xt.data(); a.p_tab = pt.data(); a.dV_tab = dv.data(); a.V0_tab = v0.data(); a.theta_s = ths.data();
  a.r_lambda = rl.data(); a.r_theta = rt.data(); a.mask1 = m1.data(); a.mask2s = m2.data(); a.sfp = sfp.data();
  a.btw_x = twx.data(); a.btw_p = twp.data(); a.partials = partials.data();
  a.partials_im = odm ? part_im.data() : nullptr;
  a.lambda_tab = lt.data(); a.hbar_exact = hBar; a.L_material = 1.; a.r_theta_half = rth.data(); a.gp_coef = a_gp;
  std::vector<double2> colsum(NX);
  if (a_gp != 0. && !odm) a.colsum = colsum.data();
  emu_launch(1, 64, [&] { wig_setup(a, rl.data(), rt.data(), m1.data(), m2.data(), sfp.data(), rth.data()); });
  double2* Wp = W.data();
  emu_launch(n_cta_r, WIG_RNT, [&] { wig_reduce(a, Wp); });
  a.n_partials = n_cta_r;
#if WIG_ODM == 2
  std::vector<double2> c2x(NX), cth(NP), R(2 * npts);
  for (int k = 0; k < NX; ++k) c2x[k] = make_double2(cos(2. * xt[k]), sin(2. * xt[k]));
  for (int k = 0; k < NP; ++k) cth[k] = make_double2(cos(hBar * ths[k] * NP), sin(hBar * ths[k] * NP));
  a.cs2x = c2x.data();
  a.csth = cth.data();
  std::vector<double2> twox = wighost::block_twiddles(NX, WIG_OE), twop = wighost::block_twiddles(NP, WIG_OE);
  const int gox = NP / WIG_OXR, oxnt = WIG_OXR * (NX / WIG_OE), gop = NX / WIG_OPC, opnt = WIG_OPC * (NP / WIG_OE);
  const size_t smox = (size_t)WIG_OXR * (pad(NX, WIG_OE) * sizeof(double2) + (NX + 1) * sizeof(double));
  const size_t smop = (size_t)WIG_OPC * wig::blk_stride(pad(NP, WIG_OE), WIG_OPC) * sizeof(double2);
#endif
  std::vector<double> phase(npts), psq(n_prop);
#if WIG_STRANG
  const int rch = NP < 64 ? NP : 64, nch = NP / rch;
  std::vector<double2> chunks((size_t)nch * NX);
  auto gp_terms = [&](int mode, double* out, bool have) {
    if (!have) emu_launch(NX / 32 * nch, 256, [&] { wig_gp_colsum_b(Wp, chunks.data()); });
    const double2* c = have ? a.colsum : chunks.data();
    emu_launch((NP / 2 + WIG_BXR) / WIG_BXR, xnt,
               [&] { wig_gp_phase_b(a, c, have ? 1 : nch, mode, phase.data(), out); }, smx + NX * sizeof(double));
  };
  const double* gph = a_gp != 0. ? phase.data() : nullptr;
#endif
  const bool damped = gamma != 0.;
  for (long n = 0; n < n_prop; ++n) {
    const int mode = n == 0 ? 1 : (damped ? 2 : 0);
    double* orow = obs.data() + (size_t)n * NOBS;
    const double t = (double)n * dt;
#if WIG_STRANG
    if (a_gp != 0.) gp_terms(mode, nullptr, n > 0 && a.colsum);
    emu_launch(gp + 1, pnt, [&] { wig_ppass_half(a, Wp, t, mode, orow, gph); }, smp);
    emu_launch(gx + 1, xnt, [&] { wig_xpass(a, Wp, 0, nullptr); }, smx);
    if (a_gp != 0.) gp_terms(0, psq.data() + n, false);
    emu_launch(gp, pnt, [&] { wig_ppass_half_final(a, Wp, t, gph); }, smp);
#else
    emu_launch(gx + 1, xnt, [&] { wig_xpass(a, Wp, mode, orow); }, smx);
    emu_launch(gp, pnt, [&] { wig_ppass(a, Wp, t); }, smp);
#endif
    a.n_partials = gp;
#if WIG_ODM == 2
    wig::WigArgs ao = a;
    ao.btw_x = twox.data();
    ao.btw_p = twop.data();
    const double weight[2] = {1., 0.5}, sign[2] = {1., -1.};   // GPU_Wigner2D_ODM2: damping, then pumping
    for (int j = 0; j < odm; ++j) {
      const double coef = dt * 2 * gamma * weight[j] * (1.0 / (double)NP);
      emu_launch(gox, oxnt, [&] { wig_odm_xpass(ao, Wp, R.data(), sign[j]); }, smox);
      emu_launch(gop, opnt, [&] { wig_odm_ppass(ao, Wp, R.data(), coef, sign[j]); }, smop);
    }
    a.n_partials = gop;
#endif
  }
  double2 scale{1., 0.};
  const int fmode = damped ? 2 : 0;
  emu_launch(1, WIG_RNT, [&] { wig_finalize(a, fmode, obs.data() + (size_t)n_prop * NOBS, &scale); });
  if (fmode) emu_launch(2, WIG_RNT, [&] { wig_scale(Wp, (long)npts, &scale); });
  if (!write_all(argv[2], W.data(), npts * sizeof(double2))) return 4;
#if WIG_STRANG
  obs.insert(obs.end(), psq.begin(), psq.end());
#endif
  return write_all(argv[3], obs.data(), obs.size() * sizeof(double)) ? 0 : 4;
}
