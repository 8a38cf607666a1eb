"""The build's exponential exp(-E 2^e) on the GPU at the edges of its scales (both
shifts of the common form, the clamped ones, and what it leaves to the general form):
within 1 ulp of the host's extended-precision value, as at the scales in between."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-1, -13, -19, -20, -21, -43, -44, -45, -63, -64, -65, -90, -127, -128])
def test_scales(e, lib):
    from fgpu import _lib
    rng = np.random.default_rng(-e)
    bits = rng.integers(0, 62, size=60000)
    E = rng.integers(0, 2 ** 62, size=bits.size, dtype=np.uint64) >> (62 - bits).astype(np.uint64)
    E = np.concatenate([E, np.array([0, 1, 2, 2 ** 31, 2 ** 32, 2 ** 61, 2 ** 62 - 1], dtype=np.uint64)])
    y = np.empty(E.size)
    _lib.check(lib.fgpu_diag_exp_fixed(E.ctypes.data_as(C.POINTER(C.c_ulonglong)), e,
                                       y.ctypes.data_as(_lib.c_double_p), E.size))
    x = E.astype(np.longdouble) * np.longdouble(2.0) ** e
    with np.errstate(under="ignore"):
        ref = np.exp(-x).astype(np.float64)
    assert np.all(np.abs(y - ref) <= np.spacing(ref))
    assert np.all(y[E == 0] == 1.0)
