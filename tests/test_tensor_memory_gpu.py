"""The damped p-pass of 16 elements a thread keeps its Caldeira-Leggett base in
tensor memory: CTAs of one warp (whose 16 per SM ask for more columns than there
are, so some wait for others to give theirs back), two and sixteen warps, against
the oracle.  Bars of the other complex128 passes (relative L2 1e-10, observables
1e-10 of their scale)."""
import numpy as np
import pytest

from oracle.common import rel_l2
from oracle.wigner2d import WignerOracle, WignerParams, wigner_harmonic_oscillator
from golden_cases import obs_close
from instances import wigner_instance, wigner_obs

pytestmark = pytest.mark.gpu
TOL = 1e-10


# warps a CTA: 1, 1, 2, 16 (two columns of 256 threads)
@pytest.mark.parametrize('n_x,n_p', [(4096, 128), (2048, 256), (1024, 512), (512, 4096)])
def test_damped_pass_matches_oracle(n_x, n_p):
    prm = WignerParams(n_x, n_p, 10., 8., 0.01, hbar=0.9, mass=1.3, d_theta=0.05, d_lambda=0.01, gamma=0.05,
                       potential='0.05*pow(x,4) - pow(x,2) + 0.1*x*sin(3.*t)',
                       dpotential='0.2*pow(x,3) - 2.*x + 0.1*sin(3.*t)', damping='CaldeiraLeggett',
                       fp_damping='p*p/sqrt(p*p + 0.5)')
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1.5, -0.5)
    inst = wigner_instance(prm, W0, 2)
    inst.Run()
    obs, W = WignerOracle(prm).run(W0, 3)
    assert rel_l2(inst.W_end_complex, W) < TOL
    got = wigner_obs(inst)
    assert obs_close(got[:, :9], obs[:3, 1:10], TOL) < TOL
    # the negative area sums the points below zero: those within rounding of zero enter one sum and not the other
    assert np.max(np.abs(got[:, 9] - obs[:3, 10])) < 1e-10
