"""wig_run_observables gives the rows that the handle's last run recorded, and no
others: the device buffer keeps the size of the longest run so far, and its rest
holds samples of earlier runs."""
import ctypes

import numpy as np
import pytest
import torch

from oracle.wigner2d import WignerParams, wigner_harmonic_oscillator
from pywignercuda_b200 import _lib
from instances import wigner_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('many', [False, True])
def test_observables_of_the_last_run_only(many):
    prm = WignerParams(64, 64, 10., 10., 0.01, potential='0.5*pow(x,2)', dpotential='x', gamma=0.1, d_theta=0.05,
                       damping='CaldeiraLeggett', fp_damping='fabs(p)')
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1., 0.5)
    inst = wigner_instance(prm, W0, 4)
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    W = torch.from_numpy(np.ascontiguousarray(W0, dtype=np.complex128)).cuda()
    out = torch.full((101, _lib.WIG_NOBS), -7., dtype=torch.float64, device='cuda')
    assert lib.wig_run_observables(inst._handle, out.data_ptr(), 1, st) == 1            # no run yet
    inst.propagate(W, 100)
    if many:
        hs, Ws = (ctypes.c_void_p * 1)(inst._handle), (ctypes.c_void_p * 1)(W.data_ptr())
        obs = np.empty((4, _lib.WIG_NOBS))
        rows = (ctypes.POINTER(ctypes.c_double) * 1)(_lib.dptr(obs))
        assert lib.wig_run_many(hs, Ws, 1, 100, 3, _lib.WIG_RUN_CONTINUE, rows, st) == 0
    else:
        obs = inst.propagate(W, 3, t_index0=100, continue_run=True)
    assert lib.wig_run_observables(inst._handle, out.data_ptr(), 101, st) == 1
    assert 'recorded 4' in lib.wig_last_error().decode()
    assert bool((out == -7.).all())
    assert lib.wig_run_observables(inst._handle, out.data_ptr(), 4, st) == 0
    assert np.array_equal(out[:4].cpu().numpy(), obs)
    assert bool((out[4:] == -7.).all())
