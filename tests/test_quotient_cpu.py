"""The correctly rounded quotient of the triangular solves (ppb_bdf.cuh:
quotient): b / a from the rounded reciprocal of a by multiply-adds alone must
be the IEEE quotient, bit for bit, over the range the solves use it in."""

import ctypes as C
import ctypes.util

import numpy as np
import pytest

_fma = C.CDLL(ctypes.util.find_library("m")).fma
_fma.restype = C.c_double
_fma.argtypes = [C.c_double] * 3


def quotient(b, a, y):
    q = b * y
    q = _fma(_fma(-a, q, b), y, q)
    return _fma(_fma(-a, q, b), y, q)


def mantissas(rng, n):
    """Random significands, and those next to 1, 2 and the middle."""
    m = 1.0 + rng.integers(0, 2 ** 52, n) * 2.0 ** -52
    edge = np.array([1.0, 1.0 + 2.0 ** -52, 1.5, 1.5 - 2.0 ** -52, 2.0 - 2.0 ** -51, 2.0 - 3 * 2.0 ** -52])
    m[: edge.size] = edge
    return m


# exponents of b and a: the solves take b within 2^+-500 (or zero) and a within 2^+-400
@pytest.mark.parametrize("eb,ea", [(0, 0), (-500, 399), (499, -400), (-500, -400), (499, 399), (-30, 12)])
def test_quotient_is_the_ieee_quotient(eb, ea):
    rng = np.random.default_rng(1000 * (eb + 500) + ea + 400)
    b = mantissas(rng, 4000) * 2.0 ** eb * rng.choice([-1.0, 1.0], 4000)
    a = rng.permutation(mantissas(rng, 4000)) * 2.0 ** ea * rng.choice([-1.0, 1.0], 4000)
    for x, d in zip(b.tolist(), a.tolist()):
        assert quotient(x, d, 1.0 / d) == x / d
    for d in a[:50].tolist():
        assert quotient(0.0, d, 1.0 / d) == 0.0
