"""The entry points that make a fixed sequence of launches without a host wait can
be captured into a CUDA graph by a caller, their programmatic launches included;
the replays equal the direct calls bit for bit."""
import numpy as np
import pytest
import torch

from adjoint_twin import coherent
from oracle.wigner2d import WignerParams, wigner_harmonic_oscillator
from instances import gp_instance, wigner_instance

pytestmark = pytest.mark.gpu


def captured(call):
    """`call(stream)` once on a stream of its own, then captured there: the graph."""
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        call(st)
    st.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        call(st)
    return graph


@pytest.mark.parametrize('precision,gamma', [('c64', 0.), ('c64', 0.1), ('c128', 0.), ('c128', 0.1)])
def test_captured_gradient_equals_direct(precision, gamma):
    from pywignercuda_b200.adjoint import WignerControl
    n, T = 128, 7
    prop = WignerControl(n, n, x_amplitude=10., dt=0.01, gamma=gamma, d_theta=0.02, precision=precision)
    W0 = coherent(n, 10., -1.0, 0.5, device='cuda').to(prop.dtype).contiguous()
    lam0 = coherent(n, 10., 1.0, -0.5, device='cuda').to(prop.dtype).contiguous()
    eps = torch.zeros(T, dtype=torch.float64, device='cuda')
    W, lam = torch.empty_like(W0), torch.empty_like(lam0)
    Y = torch.empty((T, n, n), dtype=prop.dtype, device='cuda')
    U = torch.empty_like(Y) if gamma else None
    s = torch.zeros(T, dtype=torch.complex128, device='cuda') if gamma else None
    grad = torch.zeros((T, 3), dtype=torch.float64, device='cuda')
    drive = torch.from_numpy(np.random.default_rng(5).normal(0., 0.2, T)).cuda()
    scale = torch.ones((), dtype=torch.float64, device='cuda')

    def call(st):
        W.copy_(W0)
        lam.copy_(lam0)
        torch.mul(drive, scale, out=eps)                     # the field comes from a kernel of the caller's
        prop.forward_raw(W, eps, 0, T, Y, U, s, stream=st)
        torch.mul(drive, scale, out=eps)
        prop.adjoint_sweep(lam, Y, eps, 0, grad, U, s, stream=st)
    graph = captured(call)
    for k in (1., 0.3):
        scale.fill_(k)
        torch.cuda.synchronize()
        call(torch.cuda.current_stream())
        torch.cuda.synchronize()
        want = [t.clone() for t in (W, lam, grad)]
        for t in (W, lam, grad, eps, Y):
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for got, ref in zip((W, lam, grad), want):
            assert torch.equal(got, ref) and bool(ref.abs().sum() > 0.)


@pytest.mark.parametrize('form', ['cl', 'odm', 'gp'])
def test_captured_run_equals_direct(form):
    """wig_run without host samples, on a handle whose sample buffer has its size from an earlier run."""
    from pywignercuda_b200 import _lib
    prm = WignerParams(128, 64, 10., 8., 0.01, potential='0.05*pow(x,4) - pow(x,2)', dpotential='0.2*pow(x,3) - 2.*x',
                       gamma=0.05, d_theta=0.05, damping='ODM' if form == 'odm' else 'CaldeiraLeggett',
                       fp_damping='p*p/sqrt(p*p + 0.5)', L_material=2.)
    W0 = wigner_harmonic_oscillator(prm, 0, 1., 1., 0.5)
    inst = gp_instance(prm, 0.5, W0, 4) if form == 'gp' else wigner_instance(prm, W0, 4)
    W_in = torch.from_numpy(np.ascontiguousarray(W0, dtype=np.complex128)).cuda()
    W = W_in.clone()
    obs = torch.zeros((5, _lib.WIG_NOBS), dtype=torch.float64, device='cuda')
    lib = _lib.load()

    def call(st):
        W.copy_(W_in)
        assert lib.wig_run(inst._handle, W.data_ptr(), 0, 4, 0, None, st.cuda_stream) == 0, lib.wig_last_error()
        assert lib.wig_run_observables(inst._handle, obs.data_ptr(), 5, st.cuda_stream) == 0, lib.wig_last_error()
    graph = captured(call)
    call(torch.cuda.current_stream())
    torch.cuda.synchronize()
    want, want_obs = W.clone(), obs.clone()
    W.zero_()
    obs.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(W, want) and torch.equal(obs, want_obs)
    assert bool(torch.isfinite(obs).all())
