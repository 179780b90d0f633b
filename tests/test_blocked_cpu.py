"""The complex128 Wigner2D passes on the register-blocked transform, executed on
the host (tests/emu/blocked_emu.cpp), against the oracle, plain, under
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
