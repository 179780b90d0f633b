"""A Run() whose state stops being finite ends there: the frames up to the last
finite sample are kept, no later one is kept or written, and the steps that are
left are not issued (but for those already under way, at most a buffer of the
frame writer each)."""
import numpy as np
import pytest

from oracle.wigner2d import WignerParams, wigner_harmonic_oscillator
from instances import wigner_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('gamma', [0., 0.1])
def test_run_stops_at_the_first_nonfinite_sample(gamma):
    from pywignercuda_b200._lib import WignerNonFiniteError
    # sqrt of a negative number from step 11 (t = 0.11) on; the samples from row 12 on are not finite
    prm = WignerParams(64, 64, 10., 10., 0.01, potential='0.5*pow(x,2) + 0.001*x*sqrt(0.105 - t)', dpotential='x',
                       gamma=gamma, d_theta=0.05, damping='CaldeiraLeggett', fp_damping='fabs(p)')
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1., 0.5)
    inst = wigner_instance(prm, W0, 400, skip_frames=2)
    stretches, stretch = [], inst._stretch

    def count(W, n_prop, t_index0, *args):
        stretches.append(t_index0)
        stretch(W, n_prop, t_index0, *args)
    inst._stretch = count
    with pytest.raises(WignerNonFiniteError):
        inst.Run()
    assert sorted(inst.frames) == [0, 2, 4, 6, 8, 10]
    assert all(np.isfinite(f).all() for f in inst.frames.values())
    # frame 12 is found bad before its buffer is given back, which frame 18 waits for
    assert stretches[-1] <= 18, stretches
