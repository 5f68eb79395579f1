"""The line FFT at lengths of every radix, one to three stages, and tiles with
ragged z: fftxyp2s, lapinv1, fftxys2p against the oracle.  The bound is 64
roundings of the transforms' lengths (log2(128^2) butterflies each way)."""
import ctypes as C

import numpy as np
import pytest

from epic_b200.abi import EpicContext
from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 6, 5), (8, 10, 16), (12, 18, 15), (20, 24, 31), (30, 36, 32), (40, 54, 17),
                                   (60, 72, 33), (80, 90, 47), (100, 108, 12), (120, 150, 9), (250, 16, 4)])
@pytest.mark.parametrize("path", [0, 2])
def test_line_fft_lengths(olib, glib, shape, path):
    rng = np.random.default_rng(5)
    f = rng.normal(size=(shape[0], shape[1], shape[2] + 3))
    out = []
    for lib, name in ((olib, "epic_oracle_test_spectral"), (glib, "epic_gpu_test_spectral")):
        ctx = EpicContext(lib, lib.default_config(*shape, (0.0, 0.0, 0.0), (2.0, 3.0, 1.0), n_per_cell=1))
        if lib is glib:
            glib.lib.epic_gpu_test_set_fft_path.argtypes = [C.c_void_p, C.c_int]
            assert glib.lib.epic_gpu_test_set_fft_path(ctx.h, path) == 0
        P = C.POINTER(C.c_double)
        call = getattr(lib.lib, name)
        call.argtypes = [C.c_void_p, C.c_int, P, P]
        r = np.zeros_like(f)
        assert call(ctx.h, 0, f.ctypes.data_as(P), r.ctypes.data_as(P)) == 0
        out.append(r[:, :, 1:-1])
    assert rel_err(out[1], out[0]) < 64 * np.finfo(np.float64).eps * np.log2(shape[0] * shape[1])
