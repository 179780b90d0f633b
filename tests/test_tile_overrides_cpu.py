"""The tile overrides of the register-blocked passes (WIG_*_BTILING) are checked
on the host before any compile: a tile that leaves rows or columns of the grid
to no CTA, or that a CTA cannot run, is WIG_ERR_ARG."""
import ctypes

import pytest

from pywignercuda_b200 import _lib


def refused(monkeypatch, fn, desc, env, value):
    """The message of the refusal (asserted); the descriptor itself is accepted."""
    buf = ctypes.create_string_buffer(1 << 16)
    monkeypatch.setenv(env, value)
    assert getattr(_lib.load(), fn)(desc, buf, len(buf)) == 1, buf.value[:300]
    assert env in buf.value.decode()


def accepted(monkeypatch, fn, desc, env, value):
    buf = ctypes.create_string_buffer(1 << 16)
    monkeypatch.setenv(env, value)
    assert getattr(_lib.load(), fn)(desc, buf, len(buf)) == 0, buf.value[:300]


def adjoint_desc(n_x, n_p):
    d = _lib.WigaDesc()
    d.abi_version = _lib.ABI_VERSION
    d.n_x, d.n_p = n_x, n_p
    d.precision = _lib.WIGA_PREC_C128
    d.x_amplitude = d.p_amplitude = 10.
    d.hbar = d.mass = 1.
    d.dt = 0.005
    return d


# rows and columns that do not divide the grid, more than 1024 threads, more than 32 columns, no tile at all
@pytest.mark.parametrize('n_x,n_p,value', [(256, 128, '8,3,1'), (128, 256, '8,1,3'), (256, 128, '8,64,1'),
                                           (128, 64, '8,1,64'), (64, 64, '8,128,1')])
def test_adjoint_tile_refused(monkeypatch, n_x, n_p, value):
    refused(monkeypatch, 'wiga_jit_check', adjoint_desc(n_x, n_p), 'WIG_ADJ_BTILING', value)


def test_adjoint_tile_accepted(monkeypatch):
    accepted(monkeypatch, 'wiga_jit_check', adjoint_desc(256, 128), 'WIG_ADJ_BTILING', '4,2,2')


def dirac3_desc(*shape):
    d = _lib.Dirac3Desc()
    d.abi_version = _lib.ABI_VERSION
    d.n_x, d.n_y, d.n_z = shape
    d.constants = _lib.CONST_CUDA_F
    d.precision = _lib.PREC_C128
    d.x_amplitude = d.y_amplitude = d.z_amplitude = 8.
    d.mass, d.c, d.hbar, d.dt = 1., 137.036, 1., 1e-4
    return d


# lines of x, y and z that do not divide the grid, 2048 threads, 64 columns, no line, 5 elements a thread
@pytest.mark.parametrize('shape,value', [((256, 32, 32), '8,3,0,0,0,0,0,0,0'), ((64, 256, 32), '0,0,0,16,6,0,0,0,0'),
                                         ((64, 32, 256), '0,0,0,0,0,0,8,3,0'), ((256, 32, 32), '8,64,0,0,0,0,0,0,0'),
                                         ((64, 64, 64), '0,0,0,8,64,0,0,0,0'), ((64, 64, 64), '8,-4,0,0,0,0,0,0,0'),
                                         ((64, 64, 64), '0,0,0,0,0,0,5,0,0')])
def test_dirac3d_tile_refused(monkeypatch, shape, value):
    refused(monkeypatch, 'dirac3_jit_check', dirac3_desc(*shape), 'WIG_D3_BTILING', value)


def test_dirac3d_tile_accepted(monkeypatch):
    accepted(monkeypatch, 'dirac3_jit_check', dirac3_desc(64, 32, 32), 'WIG_D3_BTILING', '4,4,1,4,8,1,4,8,1')


def wigner_desc(n_x, n_p):
    d = _lib.WigDesc()
    d.abi_version = _lib.ABI_VERSION
    d.n_x, d.n_p = n_x, n_p
    d.x_amplitude = d.p_amplitude = 10.
    d.hbar = d.mass = 1.
    d.dt = 0.01
    return d


def dirac_desc(n_x, n_y):
    d = _lib.DiracDesc()
    d.abi_version = _lib.ABI_VERSION
    d.n_x, d.n_y = n_x, n_y
    d.x_amplitude = d.y_amplitude = 12.
    d.mass, d.c, d.hbar, d.dt = 1., 137.036, 1., 1e-4
    return d


ROWS = [('wig_jit_check', wigner_desc, 'WIG_BTILING', (256, 64), '4,%d,0,0,0,0,-1'),
        ('dirac_jit_check', dirac_desc, 'WIG_DIRAC_BTILING', (256, 64), '4,%d,0,0,0,0'),
        ('dirac3_jit_check', dirac3_desc, 'WIG_D3_BTILING', (256, 32, 32), '4,%d,0,0,0,0,0,0,0'),
        ('wiga_jit_check', adjoint_desc, 'WIG_ADJ_BTILING', (256, 64), '4,%d,0')]


@pytest.mark.parametrize('fn,desc,env,shape,value', ROWS, ids=[r[2] for r in ROWS])
def test_rows_beyond_the_hardware_barriers_refused(monkeypatch, fn, desc, env, shape, value):
    """Rows of 64 threads each take one of a CTA's 15 named barriers: 16 rows (1024 threads) have none."""
    refused(monkeypatch, fn, desc(*shape), env, value % 16)
    accepted(monkeypatch, fn, desc(*shape), env, value % 8)
