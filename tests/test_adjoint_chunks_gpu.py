"""Adjoint sweeps longer than one chunk of gradient partials (the complex64 form
keeps those of 64 steps and sums them in one launch): the gradient rows and
dL/dW_0 of single steps, bit for bit, from a field that a kernel of the caller's
has written just before the sweep."""
import numpy as np
import pytest
import torch

from adjoint_twin import coherent

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('steps', [64, 65, 130])
@pytest.mark.parametrize('precision,gamma', [('c64', 0.), ('c64', 0.1), ('c128', 0.), ('c128', 0.1)])
def test_long_sweep_equals_steps(precision, gamma, steps):
    from pywignercuda_b200.adjoint import WignerControl
    n, step0 = 64, 3
    prop = WignerControl(n, n, x_amplitude=10., dt=0.01, gamma=gamma, d_theta=0.02, precision=precision)
    total = step0 + steps
    field = torch.from_numpy(np.random.default_rng(11).normal(0., 0.2, total)).cuda()
    W = coherent(n, 10., -1.0, 0.5, device='cuda').to(prop.dtype).contiguous()
    lam0 = coherent(n, 10., 1.0, -0.5, device='cuda').to(prop.dtype).contiguous()
    Y = torch.empty((steps, n, n), dtype=prop.dtype, device='cuda')
    U = torch.empty_like(Y) if gamma else None
    s = torch.zeros(total, dtype=torch.complex128, device='cuda') if gamma else None
    prop.forward_raw(W, field, step0, steps, Y, U, s)
    lam_a, lam_b = lam0.clone(), lam0.clone()
    g_a = torch.zeros((total, 3), dtype=torch.float64, device='cuda')
    g_b = torch.zeros_like(g_a)
    for k in reversed(range(steps)):
        prop.adjoint_step(lam_a, Y[k], field, step0 + k, g_a, U[k] if U is not None else None, s)
    eps = torch.full_like(field, 100.)
    torch.mul(field, 1., out=eps)
    prop.adjoint_sweep(lam_b, Y, eps, step0, g_b, U, s)
    torch.cuda.synchronize()
    assert torch.equal(lam_a, lam_b)
    assert torch.equal(g_a, g_b)
    assert bool((g_b[:step0] == 0.).all()) and bool((g_b[step0:, 0] != 0.).all())
