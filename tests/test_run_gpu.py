"""Run() issues the stretches between frames without waiting for them and collects
their samples on the device: the samples of one uninterrupted propagate call to
rounding (a stretch's end normalises W where a step would normalise on load), and
the same error for a state that is not finite."""
import numpy as np
import pytest
import torch

from oracle.wigner2d import WignerParams, wigner_harmonic_oscillator
from instances import wigner_instance, wigner_obs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('steps,skip', [(0, 1), (1, 1), (7, 3), (12, 4), (5, 100)])
@pytest.mark.parametrize('gamma', [0., 0.1])
def test_run_samples_match_one_propagate(steps, skip, gamma):
    prm = WignerParams(64, 32, 10., 8., 0.01, potential='0.5*pow(x,2) + 0.1*x*sin(t)', dpotential='x + 0.1*sin(t)',
                       gamma=gamma, d_theta=0.05, damping='CaldeiraLeggett', fp_damping='fabs(p)')
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1., 0.5)
    inst = wigner_instance(prm, W0, steps)
    inst.skipFrames = skip
    inst.Run()
    W = torch.from_numpy(np.ascontiguousarray(W0, dtype=np.complex128)).cuda()
    ref = inst.propagate(W, steps + 1)
    assert np.allclose(wigner_obs(inst), ref[:steps + 1, 1:11], rtol=1e-12, atol=1e-12)
    assert np.allclose(inst.W_end_complex, W.cpu().numpy(), rtol=0., atol=1e-13)
    assert inst.timeRangeIndexSaved == list(range(0, steps + 1, skip))


def test_run_reports_nonfinite_state():
    from pywignercuda_b200._lib import WignerNonFiniteError
    prm = WignerParams(64, 64, 10., 10., 0.01, potential='0.5*pow(x,2)', dpotential='x', gamma=0.1, d_theta=0.1,
                       damping='CaldeiraLeggett', fp_damping='fabs(p)')
    W0 = np.array(wigner_harmonic_oscillator(prm, 0, 1., 1., 0.), dtype=np.complex128)
    W0[5, 7] = float('nan')
    inst = wigner_instance(prm, W0, 4)
    inst.skipFrames = 2
    with pytest.raises(WignerNonFiniteError):
        inst.Run()
