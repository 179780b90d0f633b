"""The mixed batched passes keep their FP64 sequences in registers: 16 elements a
thread from 512 points, 8 below, at 16 (x) and 12 (p) warps per SM.  The register
transform before them held 32 double2 a lane and spilled ~1.1 KB a thread."""
import ctypes

import pytest

from conftest import full_only
from pywignercuda_b200 import _lib


@pytest.mark.parametrize('warps', [4, full_only(2), full_only(8)])
def test_mixed_passes_hardly_spill(warps):
    """All size classes in one module; 8 bytes (p-pass) and 0 at 4 and 2 warps, 0 at 8: one more double2 a
    thread at most."""
    sizes = (ctypes.c_int32 * 5)(64, 128, 256, 512, 1024)
    buf = ctypes.create_string_buffer(1 << 17)
    rc = _lib.load().wigb_jit_check(sizes, 5, warps, 1, buf, len(buf))
    log = buf.value.decode()
    assert rc == 0, log
    lines = log.splitlines()
    for k in ('wigb_xpass', 'wigb_ppass'):
        at = [i for i, l in enumerate(lines) if "Compiling entry function '%s'" % k in l]
        assert at, k
        props = ' '.join(lines[at[0] + 1:at[0] + 3])
        spill = int(props.split(' bytes spill stores')[0].split()[-1])
        assert spill <= 24, (k, props)
