"""The register-blocked complex128 Wigner2D passes on the GPU against the oracle,
over the tiles that the planner picks: axes from 32 to 4096 points, 4, 8 and 16
elements a thread (grids below 2^17, 2^19 points and above; the last with the
Caldeira-Leggett base in tensor memory), one axis of 16 points left to the
Stockham passes.  Bars: those of the other complex128 paths (relative L2 1e-10,
observables 1e-10 of their scale)."""
import numpy as np
import pytest

from oracle.common import rel_l2
from oracle.gpitaevskii import GPitaevskiiOracle
from oracle.wigner2d import WignerOracle, WignerParams, wigner_harmonic_oscillator
from golden_cases import obs_close
from instances import gp_instance, wigner_instance, wigner_obs

pytestmark = pytest.mark.gpu
TOL = 1e-10
POT, DPOT = '0.05*pow(x,4) - pow(x,2) + 0.1*x*sin(3.*t)', '0.2*pow(x,3) - 2.*x + 0.1*sin(3.*t)'

CASES = [(32, 32, 'cl'), (32, 64, 'gp'), (64, 32, 'odm2'), (32, 4096, 'cl'), (16, 64, 'none'), (512, 16, 'odm'),
         (64, 64, 'cl'), (128, 64, 'none'), (64, 256, 'odm2'), (512, 32, 'cl'), (32, 512, 'odm'), (2048, 64, 'kvn'),
         (64, 2048, 'cl'), (4096, 64, 'cl'), (64, 4096, 'cl'), (512, 512, 'cl'), (1024, 256, 'odm'),
         (512, 1024, 'cl'), (1024, 1024, 'kvn'), (256, 2048, 'none'), (2048, 512, 'odm2'), (256, 4096, 'cl'),
         (64, 64, 'gp'), (256, 64, 'gp'), (512, 1024, 'gp'), (64, 128, 'gpodm')]


@pytest.mark.parametrize('n_x,n_p,form', CASES)
def test_blocked_passes_match_oracle(n_x, n_p, form):
    odm = 'odm' in form
    prm = WignerParams(n_x, n_p, 10., 8., 0.01, hbar=0.9, mass=1.3, d_theta=0.05, d_lambda=0.01,
                       gamma=0. if form == 'none' else 0.05, potential=POT, dpotential=DPOT,
                       damping='ODM' if odm else 'CaldeiraLeggett', fp_damping='p*p/sqrt(p*p + 0.5)', L_material=2.,
                       kvn=form == 'kvn', odm2=form == 'odm2', weight1=1., weight2=0.5 if form == 'odm2' else 0.)
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1.5, -0.5)
    if form.startswith('gp'):
        inst = gp_instance(prm, 0.5, W0, 2)
        inst.Run()
        obs, W, psq = GPitaevskiiOracle(prm, 0.5).run(W0, 3)
        assert np.max(np.abs(inst.ProbabilitySquare_average - psq) / np.abs(psq)) < TOL
    else:
        inst = wigner_instance(prm, W0, 2)
        inst.Run()
        obs, W = WignerOracle(prm).run(W0, 3)
        obs = obs[:3]
    assert rel_l2(inst.W_end_complex, W) < TOL
    got = wigner_obs(inst)
    assert obs_close(got[:, :9], obs[:3, 1:10], TOL) < TOL
    # the negative area sums the points below zero: those within rounding of zero enter one sum and not the other
    assert np.max(np.abs(got[:, 9] - obs[:3, 10])) < 1e-10


@pytest.mark.parametrize('n_x,n_y', [(32, 32), (16, 64), (64, 64), (128, 256), (64, 2048), (2048, 64), (512, 256),
                                     (1024, 512), (512, 1024)])
def test_blocked_dirac2d_passes_match_oracle(n_x, n_y):
    """4 elements a thread below 2^17 points, 8 from there; one to four columns a CTA."""
    from instances import dirac_instance, dirac_obs
    from oracle.dirac2d import DiracOracle, DiracParams, spinor_particle_spin_up
    prm = DiracParams(n_x, n_y, 12., 8., 1e-4, mass=1., c=137.036, A0='-1./sqrt(x*x+y*y+0.5) + 3.*t*x', A1='-0.5*y',
                      A2='0.5*x', A3='0.1*x')
    psi0 = spinor_particle_spin_up(prm, (3., 1.), lambda x, y: np.exp(-(x * x + y * y) / 2.))
    inst = dirac_instance(prm, psi0, 3)
    inst.Run()
    obs, psi = DiracOracle(prm).run(psi0, 3)
    assert rel_l2(inst.Psi_end, psi) < TOL
    assert obs_close(dirac_obs(inst), obs[:, :7], TOL) < TOL
    assert obs_close(np.stack([inst.Px_average, inst.Py_average, inst.NormKept_average], 1), obs[:, 7:10], TOL) < TOL


@pytest.mark.parametrize('dims', [(32, 32, 32), (64, 32, 128), (32, 128, 64), (128, 64, 64), (512, 32, 64), (32, 64, 512)])
def test_blocked_dirac3d_passes_match_oracle(dims):
    """4 elements a thread below 2^18 points, 8 from there (the y-pass 4, 8 or 16)."""
    from instances import dirac3d_instance, dirac3d_obs
    from oracle.dirac3d import Dirac3DOracle, Dirac3DParams, spinor_particle_spin_up_3d
    prm = Dirac3DParams(*dims, 10., 8., 9., 1e-4, mass=1., c=137.036, A0='-1./sqrt(x*x+y*y+z*z+0.5) + 2.*t*z',
                        A1='-0.5*y', A2='0.5*x', A3='0.1*z')
    psi0 = spinor_particle_spin_up_3d(prm, (3., 1., 0.5), lambda x, y, z: np.exp(-(x * x + y * y + z * z) / 4.))
    inst = dirac3d_instance(prm, psi0, 3)
    inst.Run()
    obs, psi = Dirac3DOracle(prm).run(psi0, 3)
    assert rel_l2(inst.Psi_end, psi) < TOL
    assert obs_close(dirac3d_obs(inst), obs, TOL) < TOL
