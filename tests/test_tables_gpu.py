"""Host tables of lambda or theta that are not odd about 0: the ODM and the
Gross-Pitaevskii terms take them as given.  The register-blocked passes evaluate
one point of each pair +-lambda, +-theta and may only serve tables that are odd;
WIG_TILING selects the general passes, whose result is the reference here."""
import numpy as np
import pytest
import torch

from oracle.common import rel_l2
from oracle.wigner2d import WignerParams, wigner_harmonic_oscillator
from instances import gp_instance, wigner_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('form', ['odm', 'gp', 'gpodm'])
@pytest.mark.parametrize('d_lambda,d_theta', [(0.3, 0.), (0., 0.3), (0., 0.)])
def test_tables_not_odd_about_zero(monkeypatch, form, d_lambda, d_theta):
    """Offsets in units of the tables' spacing.  1e-11: both sides round at 1e-15 a transform and step, and
    the state's condition over 3 steps is near 1 (the offset tables change the result by 1e-4 and more)."""
    import pywignercuda_b200 as P
    set_grid = P.GPU_Wigner2D_FFT.SetPhaseSpaceGrid2D

    def shifted(self):
        set_grid(self)
        self.Lambda = self.Lambda + d_lambda * self.dLambda
        self.Theta = self.Theta + d_theta * self.dTheta
    prm = WignerParams(64, 128, 10., 8., 0.01, hbar=0.9, mass=1.3, d_theta=0.05, gamma=0.05,
                       potential='0.05*pow(x,4) - pow(x,2)', dpotential='0.2*pow(x,3) - 2.*x',
                       damping='ODM' if 'odm' in form else 'CaldeiraLeggett', fp_damping='p*p/sqrt(p*p + 0.5)',
                       L_material=2.)
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1.5, -0.5)
    monkeypatch.setattr(P.GPU_Wigner2D_FFT, 'SetPhaseSpaceGrid2D', shifted)

    def result(tiling):
        if tiling:
            monkeypatch.setenv('WIG_TILING', '0,0,0,0,0,0')
        else:
            monkeypatch.delenv('WIG_TILING', raising=False)
        inst = gp_instance(prm, 5., W0, 3) if form.startswith('gp') else wigner_instance(prm, W0, 3)
        W = torch.from_numpy(np.ascontiguousarray(W0, dtype=np.complex128)).cuda()
        obs = inst.propagate(W, 3)
        return W.cpu().numpy(), obs
    (W, obs), (ref, ref_obs) = result(False), result(True)
    assert rel_l2(W, ref) < 1e-11
    assert np.allclose(obs[:, :10], ref_obs[:, :10], rtol=1e-10, atol=1e-11)
