"""The FP64 Cholesky's reciprocal and reciprocal square root of a pivot, which start from an FP32 seed
(csrc/bss_chol_f64.cuh), on their own: whole solutions pass their tests with reciprocals good to 1e-11."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_every_seed():
    """1 / p is formed in integers with errors of a few 2^-56 and rounded once: one unit of the last
    place at most from the correctly rounded quotient.  1 / sqrt(p) ends in one FMA whose addend is off by
    less than half a unit, and the value it is compared with is rounded twice: two units."""
    from blockstructuredsolvers_gb300 import _lib
    rcp, rsqrt = ctypes.c_int32(-1), ctypes.c_int32(-1)
    _lib.check(_lib.load().bss_diag_pivot_selftest(ctypes.byref(rcp), ctypes.byref(rsqrt)))
    assert 0 <= rcp.value <= 1
    assert 0 <= rsqrt.value <= 2
