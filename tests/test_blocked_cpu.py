"""The complex128 Wigner2D and Dirac passes on the register-blocked transform,
executed on the host (tests/emu/blocked_emu.cpp, the Dirac drivers), against the oracle, plain, under
ThreadSanitizer (a missing barrier between two threads' uses of an exchange
region is a reported race) and under AddressSanitizer (an index past a launch's
shared memory).  Tiles: sequences within a warp, of one and of
several warps, one and several rows or columns per CTA, every radix mix of the
stage plan (4 16, 8 8, 4 4 4, 8 16, 8 2 8, 4 2 4 4), a grid of unequal axes."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import test_emu_cpu as E
from oracle.common import rel_l2
from oracle.wigner2d import WignerOracle, WignerParams
from test_emu_cpu import staged  # noqa: F401  (the module-scoped staging fixture)

# n_x, n_p, (rows, elements), (columns, elements), form, sanitizer
CASES = [
    (64, 64, (8, 16), (8, 16), 'cl', None),
    (64, 128, (4, 8), (2, 8), 'cl', 'thread'),
    (128, 64, (1, 4), (2, 4), 'none', 'address'),
    (64, 128, (8, 16), (1, 4), 'cl', 'address'),
    (128, 64, (4, 16), (4, 8), 'odm', None),
    (64, 64, (2, 4), (4, 4), 'odm', 'thread'),
    (64, 128, (2, 4), (1, 4), 'gp', 'thread'),
    (64, 64, (4, 8), (4, 8), 'gp', None),
    (32, 32, (8, 8), (4, 4), 'cl', 'thread'),
]


@pytest.mark.parametrize('n_x,n_p,x,p,form,sanitize', CASES, ids=['%dx%d-%s-%s' % (c[0], c[1], c[4], c[5] or 'plain')
                                                                    for c in CASES])
def test_blocked_passes_match_oracle(staged, n_x, n_p, x, p, form, sanitize):  # noqa: F811
    shutil.copy(os.path.join(E.EMU, 'blocked_emu.cpp'), staged)
    with open(os.path.join(E.EMU, 'wigner2d_emu.cpp')) as f, open(os.path.join(staged, 'wigner2d_helpers.h'), 'w') as g:
        g.write(f.read().split('int main(')[0])
    gamma, odm, gp = (0. if form == 'none' else 0.1), (2 if form == 'odm' else 0), (0.5 if form == 'gp' else 0.)
    macros = dict(WIG_NX=n_x, WIG_NP=n_p, WIG_XROWS=1, WIG_XNT=32, WIG_PC=8, WIG_PNT=32, WIG_RNT=64, WIG_XMINB=1,
                  WIG_PMINB=1, WIG_KIN_STRING=int(form in ('odm', 'gp')), WIG_DAMP=int(form in ('cl', 'gp')),
                  WIG_STRANG=int(form == 'gp'), WIG_ODM=2 if odm else 0, WIG_BX=1, WIG_BP=1, WIG_BXR=x[0],
                  WIG_BXE=x[1], WIG_BXMB=1, WIG_BPC=p[0], WIG_BPE=p[1], WIG_BPMB=1, WIG_OE=min(x[1], 8),
                  WIG_OXR=max(1, 32 * min(x[1], 8) // n_x), WIG_OXMB=1, WIG_OPC=max(1, 32 * min(x[1], 8) // n_p),
                  WIG_OPMB=1)
    exe = E.build(staged, 'blocked_emu.cpp', macros, sanitize)
    prm = WignerParams(n_x, n_p, E.WXA, E.WPA, E.WDT, d_theta=E.WDTH, d_lambda=E.WDLA, gamma=gamma,
                       potential=E.WPOT, dpotential=E.WDPOT, kinetic='0.5*p*p',
                       damping='ODM' if odm else 'CaldeiraLeggett', fp_damping='fabs(p)', L_material=1.,
                       odm2=bool(odm), weight1=1., weight2=0.5 if odm else 0., constants='exact')
    X = np.fft.fftshift(np.linspace(-E.WXA, E.WXA - 2 * E.WXA / n_x, n_x))[np.newaxis, :]
    P = np.fft.fftshift(np.linspace(-E.WPA, E.WPA - 2 * E.WPA / n_p, n_p))[:, np.newaxis]
    W0 = np.ascontiguousarray(np.exp(-(X - 1.5) ** 2 - (P + 0.5) ** 2 * 1.3) + 0. * 1j)
    steps = 2
    fin, fout, fobs = (os.path.join(staged, n) for n in ('bk_in.bin', 'bk_out.bin', 'bk_obs.bin'))
    W0.tofile(fin)
    r = subprocess.run([exe, fin, fout, fobs, str(steps)] +
                       [repr(v) for v in (E.WXA, E.WPA, E.WDT, gamma, E.WDTH, E.WDLA)] + [str(odm), repr(gp)],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    got = np.fromfile(fout, dtype=np.complex128).reshape(n_p, n_x)
    raw = np.fromfile(fobs)
    obs = raw[:(steps + 1) * 11].reshape(steps + 1, 11)
    if form == 'gp':
        from oracle.gpitaevskii import GPitaevskiiOracle
        ref_obs, ref, psq = GPitaevskiiOracle(prm, gp).run(W0, steps)
        assert np.max(np.abs(raw[(steps + 1) * 11:] - psq) / np.abs(psq)) < 1e-10
        obs = obs[1:]
    else:
        ref_obs, ref = WignerOracle(prm).run(W0, steps)
    # the bars of the other passes' host runs (test_emu_cpu.py)
    assert rel_l2(got, ref) < 1e-12, rel_l2(got, ref)
    scale = np.maximum(np.abs(ref_obs[:, :10]).max(axis=0), 1e-3)
    assert np.all(np.abs(obs[:, :10] - ref_obs[:, :10]) / scale < 1e-10), (obs[:, :10] - ref_obs[:, :10]) / scale
    assert np.all(np.abs(obs[:, 10] - ref_obs[:, 10]) < 1e-12), obs[:, 10] - ref_obs[:, 10]


def _driver(staged, name, edits):
    """tests/emu/<name>.cpp with the register-blocked launch shapes and tables, as <name>_blocked.cpp."""
    with open(os.path.join(E.EMU, name + '.cpp')) as f:
        src = f.read()
    for old, new in edits:
        assert old in src, old
        src = src.replace(old, new)
    with open(os.path.join(staged, name + '_blocked.cpp'), 'w') as f:
        f.write(src)
    return name + '_blocked.cpp'


DIRAC2D = (
    ('const int n_row = NY / DIR_ROWS, n_col = NX / DIR_C;', 'const int n_row = NY / DIR_BROWS, n_col = NX / DIR_BC;\n'
     '  const auto pad = [](int n, int e) { return n + n / std::min(e, 8); };'),
    ('(size_t)wig::padded_size(4 * DIR_ROWS * NX) * sizeof(double2)',
     '(size_t)DIR_BROWS * 4 * pad(NX, DIR_BRE) * sizeof(double2)'),
    ('(size_t)wig::padded_size(4 * DIR_C * NY) * sizeof(double2)',
     '(size_t)DIR_BC * wig::blk_stride(4 * pad(NY, DIR_BCE), DIR_BC) * sizeof(double2)'),
    ('emu_launch(n_row, DIR_RNT', 'emu_launch(n_row + 1, DIR_BROWS * (NX / DIR_BRE)'),
    ('emu_launch(n_col, DIR_CNT', 'emu_launch(n_col, DIR_BC * (NY / DIR_BCE)'),
    ('a.n_row_cta = n_row;', 'a.n_row_cta = n_row;\n  const std::vector<double2> bx2 = wighost::block_twiddles(NX, '
     'DIR_BRE), by2 = wighost::block_twiddles(NY, DIR_BCE);\n  a.btw_x = bx2.data(); a.btw_y = by2.data();'),
    ('#include <cstdlib>', '#include "wig_batch_host.h"\n#include <algorithm>\n#include <cstdlib>'))

DIRAC3D = (
    ('NY * NZ / D3_ROWS', 'NY * NZ / D3_BXC'), ('NX / D3_YC', 'NX / D3_BYC'), ('NX / D3_ZC', 'NX / D3_BZC'),
    ('(size_t)wig::padded_size(4 * D3_ROWS * NX)', '(size_t)D3_BXC * 4 * pad(NX, D3_BXE)'),
    ('(size_t)wig::padded_size(NY * D3_YC)', '(size_t)D3_BYC * wig::blk_stride(pad(NY, D3_BYE), D3_BYC)'),
    ('(size_t)wig::padded_size(4 * D3_ZC * NZ)', '(size_t)D3_BZC * wig::blk_stride(4 * pad(NZ, D3_BZE), D3_BZC)'),
    ('emu_launch(gx, D3_XNT', 'emu_launch(gx + 1, D3_BXC * (NX / D3_BXE)'),
    ('emu_launch(gy, D3_YNT', 'emu_launch(gy, D3_BYC * (NY / D3_BYE)'),
    ('emu_launch(gz, D3_ZNT', 'emu_launch(gz, D3_BZC * (NZ / D3_BZE)'),
    ('  // d3_plan / dirac3_create', '  const auto pad = [](int n, int e) { return n + n / std::min(e, 8); };\n  // d3_plan'),
    ('a.n_z_cta = gz;', 'a.n_z_cta = gz;\n  const std::vector<double2> bx = wighost::block_twiddles(NX, D3_BXE), by = '
     'wighost::block_twiddles(NY, D3_BYE), bz = wighost::block_twiddles(NZ, D3_BZE);\n  a.btw_x = bx.data(); '
     'a.btw_y = by.data(); a.btw_z = bz.data();'),
    ('#include "wig_jit_dirac3.cuh"', '#include "wig_jit_dirac3.cuh"\n#include "wig_batch_host.h"\n#include <algorithm>'))

ADJOINT_LAUNCHES = """
  // wiga_forward and wiga_adjoint_sweep (csrc/wig_adjoint.cu: forward_blk, adjoint_blk)
  const auto pad = [](int n, int e) { return n + n / std::min(e, 8); };
  const std::vector<double2> bx = wighost::block_twiddles(nx, WIGA_BXE), bp = wighost::block_twiddles(np, WIGA_BPE);
  a.btw_x = bx.data(); a.btw_p = bp.data();
  const int bxn = np / WIGA_BXR, bxt = WIGA_BXR * (nx / WIGA_BXE), bpn = nx / WIGA_BPC, bpt = WIGA_BPC * (np / WIGA_BPE);
  const size_t sbx = (size_t)WIGA_BXR * (pad(nx, WIGA_BXE) + wig::blk_pre_slots(nx, WIGA_BXE)) * 16;
  const size_t pre = (size_t)WIGA_BPC * wig::blk_pre_slots(np, WIGA_BPE) * 16;
  const size_t sbp = (size_t)WIGA_BPC * wig::blk_stride(pad(np, WIGA_BPE), WIGA_BPC) * 16 + pre;
  const size_t sbt = (size_t)WIGA_BPC * wig::blk_stride(2 * pad(np, WIGA_BPE), WIGA_BPC) * 16 + pre;
  std::vector<double> bpart(3 * bpn), dot(2 * bxn);
  double* part_p = bpart.data();
  const double2* cur = W.data();
  for (long n = 0; n < n_steps; ++n) {
    double2* Yn = Y.data() + (size_t)n * plane;
    double2* out = damped ? U.data() + (size_t)n * plane : W.data();
    const bool pend = damped && n > 0;
    emu_launch(bxn + 1, bxt, [&] { wiga_bx(a, cur, Yn, 1., pend ? part_p : nullptr, bpn, pend ? s.data() : nullptr,
                                           (long long)(n - 1), nullptr, nullptr, nullptr, 0, nullptr); }, sbx);
    emu_launch(bpn, bpt, [&] { wiga_bp(a, Yn, out, eps.data(), (long long)n, part_p); }, sbp);
    cur = out;
  }
  if (damped) emu_launch(4, 256, [&] { wiga_bscale(a, cur, W.data(), (long long)plane, part_p, bpn, s.data(),
                                                   (long long)(n_steps - 1)); });
  for (long n = n_steps - 1; n >= 0; --n) {
    const double2* Yn = Y.data() + (size_t)n * plane;
    if (damped && n == n_steps - 1)
      emu_launch(bxn, bxt, [&] { wiga_bdot(lam.data(), U.data() + (size_t)n * plane, dot.data()); });
    emu_launch(bpn, bpt, [&] { wiga_bpt(a, lam.data(), Yn, eps.data(), (long long)n, part_p, dot.data(), bxn, s.data()); }, sbt);
    const double2* Un = damped && n > 0 ? U.data() + (size_t)(n - 1) * plane : nullptr;
    emu_launch(bxn + 1, bxt, [&] { wiga_bx(a, lam.data(), lam.data(), -1., nullptr, 0, nullptr, (long long)n, Un,
                                           dot.data(), part_p, bpn, grad.data()); }, sbx);
  }
  if (!write_all(argv[4]"""


def _adjoint_driver(staged):
    """tests/emu/adjoint_emu.cpp with the launches of the register-blocked complex128 passes."""
    with open(os.path.join(E.EMU, 'adjoint_emu.cpp')) as f:
        head, rest = f.read().split('  // wiga_forward with the records kept')
    tail = rest.split('  if (!write_all(argv[4]')[1]
    src = head.replace('#include <cstdlib>', '#include <algorithm>\n#include <cstdlib>') + ADJOINT_LAUNCHES + tail
    with open(os.path.join(staged, 'adjoint_emu_blocked.cpp'), 'w') as f:
        f.write(src)
    return 'adjoint_emu_blocked.cpp'


@pytest.mark.parametrize('x,p,gamma,sanitize', [((1, 4), (2, 4), 0.1, 'address'), ((4, 8), (4, 8), 0.1, 'thread'),
                                                ((2, 4), (4, 8), 0., None)])
def test_blocked_adjoint_matches_twin(staged, monkeypatch, x, p, gamma, sanitize):  # noqa: F811
    """The complex128 forward and adjoint sweeps against the twin, by test_emu_cpu's test with this driver."""
    macros = dict(WIGA_B=1, WIGA_BXR=x[0], WIGA_BXE=x[1], WIGA_BXMB=1, WIGA_BPC=p[0], WIGA_BPE=p[1], WIGA_BPMB=1)
    build = E.build
    monkeypatch.setattr(E, 'build', lambda dst, source, m: build(dst, _adjoint_driver(dst), dict(m, **macros), sanitize))
    E.test_adjoint_device_code_matches_twin(staged, 1, gamma)


@pytest.mark.parametrize('n_x,n_y,row,col,sanitize', [(64, 128, (2, 4), (1, 4), 'address'), (128, 64, (4, 8), (4, 8), None),
                                                      (64, 64, (4, 8), (2, 4), 'thread')])
def test_blocked_dirac2d_passes_match_oracle(staged, n_x, n_y, row, col, sanitize):  # noqa: F811
    from oracle.dirac2d import DiracOracle, DiracParams, spinor_particle_spin_up
    exe = E.build(staged, _driver(staged, 'dirac2d_emu', DIRAC2D),
                  dict(DIR_NX=n_x, DIR_NY=n_y, DIR_ROWS=1, DIR_RNT=32, DIR_RMB=1, DIR_C=1, DIR_CNT=32, DIR_CMB=1,
                       DIR_SNT=64, DIR_B=1, DIR_BROWS=row[0], DIR_BRE=row[1], DIR_BRMB=1, DIR_BC=col[0],
                       DIR_BCE=col[1], DIR_BCMB=1), sanitize)
    prm = DiracParams(n_x, n_y, E.XA, E.YA, E.DT, mass=E.MASS, c=E.C, A0=E.A[0], A1=E.A[1], A2=E.A[2], A3=E.A[3],
                      constants='exact')
    psi0 = spinor_particle_spin_up(prm, (2., 1.), lambda x, y: np.exp(-(x * x + y * y) / 4.))
    psi0 = np.ascontiguousarray(psi0, dtype=np.complex128)
    steps = 2
    fin, fout, fobs = (os.path.join(staged, n) for n in ('bd_in.bin', 'bd_out.bin', 'bd_obs.bin'))
    psi0.tofile(fin)
    r = subprocess.run([exe, fin, fout, fobs, str(steps)] + [repr(v) for v in (E.XA, E.YA, E.DT, E.MASS, E.C)],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    ref_obs, ref = DiracOracle(prm).run(psi0, steps)
    got, obs = np.fromfile(fout, dtype=np.complex128).reshape(4, n_y, n_x), np.fromfile(fobs).reshape(steps, 10)
    assert rel_l2(got, ref) < 1e-12
    scale = np.maximum(np.abs(ref_obs).max(axis=0), 1e-3)
    assert np.all(np.abs(obs - ref_obs) / scale < 1e-10), (obs - ref_obs) / scale


@pytest.mark.parametrize('dims,x,y,z,cap,sanitize', [((32, 64, 32), (8, 8), (8, 16), (8, 8), 3, 'address'),
                                                     ((64, 32, 32), (4, 4), (4, 4), (4, 4), 5, 'thread')])
def test_blocked_dirac3d_passes_match_oracle(staged, dims, x, y, z, cap, sanitize):  # noqa: F811
    """`cap` CTAs a pass: each takes several tiles, so a tile's loads follow the previous tile's exchange."""
    from oracle.dirac3d import Dirac3DOracle, Dirac3DParams, spinor_particle_spin_up_3d
    n_x, n_y, n_z = dims
    macros = dict(D3_NX=n_x, D3_NY=n_y, D3_NZ=n_z, D3_ROWS=1, D3_XNT=32, D3_YC=2, D3_YNT=32, D3_ZC=1, D3_ZNT=32,
                  D3_SNT=64, D3_XR=8, D3_YR=8, D3_ZR=8, D3_XMB=1, D3_YMB=1, D3_ZMB=1, D3_B=1)
    for axis, (lines, e) in zip('XYZ', (x, y, z)):
        macros.update({'D3_B%sC' % axis: lines, 'D3_B%sE' % axis: e, 'D3_B%sMB' % axis: 1})
    exe = E.build(staged, _driver(staged, 'dirac3d_emu', DIRAC3D), macros, sanitize)
    prm = Dirac3DParams(n_x, n_y, n_z, *E.D3A, E.D3DT, mass=1., c=137.036, A0=E.D3POT[0], A1=E.D3POT[1],
                        A2=E.D3POT[2], A3=E.D3POT[3], constants='exact')
    psi0 = spinor_particle_spin_up_3d(prm, (2., 0.5, 1.), lambda x, y, z: np.exp(-(x * x + y * y + z * z) / 4.))
    psi0 = np.ascontiguousarray(psi0, dtype=np.complex128)
    steps = 2
    fin, fout, fobs = (os.path.join(staged, n) for n in ('b3_in.bin', 'b3_out.bin', 'b3_obs.bin'))
    psi0.tofile(fin)
    r = subprocess.run([exe, fin, fout, fobs, str(steps)] + [repr(v) for v in E.D3A + (E.D3DT, 1., 137.036)] + [str(cap)],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    ref_obs, ref = Dirac3DOracle(prm).run(psi0, steps)
    got, obs = np.fromfile(fout, dtype=np.complex128).reshape(ref.shape), np.fromfile(fobs).reshape(steps, 12)
    assert rel_l2(got, ref) < 1e-12
    scale = np.maximum(np.abs(ref_obs).max(axis=0), 1e-3)
    assert np.all(np.abs(obs - ref_obs) / scale < 1e-10), (obs - ref_obs) / scale


@pytest.mark.parametrize('warps,sanitize', [(2, 'address'), (4, 'thread')])
def test_mixed_batch_long_axes_match_oracle(staged, monkeypatch, warps, sanitize):  # noqa: F811
    """The mixed batched form's sequences of 16 elements a thread (512 points): a 64 x 512 and a
    512 x 64 instance beside an undamped 64 x 64 one, by test_emu_cpu's test with these shapes."""
    monkeypatch.setattr(E, 'BSIZES', ())
    monkeypatch.setattr(E, 'BSHAPES', ((64, 512, 10., 8.), (512, 64, 8., 10.), (64, 64, 10., 10.)))
    monkeypatch.setattr(E, 'BEXTRA', {})
    build = E.build
    monkeypatch.setattr(E, 'build', lambda dst, source, m: build(dst, source, dict(m, **{'WIGB_CASES(F)': 'F(64) F(512)'}),
                                                                 sanitize))
    E.test_batch_device_code_matches_oracle(staged, warps, 3, 1, 0)
