"""The kernels' quotient and square root (qdiv, qsqrt: zero-safe forms of / and sqrt) have
the operators' bits in FP64 and FP32: on random doubles of every exponent, on values of
the sizes the schemes divide, and on zeros of both signs, subnormals, infinities and NaN
in either place."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-310, 2.2250738585072014e-308, 1e-45, -1e-39, 1.0, -1.0, 3.0, 1e-300,
                    -1e300, 1.7976931348623157e308, np.inf, -np.inf, np.nan])


def _pairs(kind):
    rng = np.random.default_rng(11)
    if kind == "special":
        a, b = np.meshgrid(SPECIAL, np.concatenate([SPECIAL, rng.uniform(-2, 2, 50)]))
        return a.ravel(), b.ravel()
    n = 1 << 20
    if kind == "bits":  # every exponent, both signs
        a = rng.integers(0, 1 << 63, size=n, dtype=np.int64).view(np.float64) * rng.choice([-1.0, 1.0], n)
        b = rng.integers(0, 1 << 63, size=n, dtype=np.int64).view(np.float64) * rng.choice([-1.0, 1.0], n)
        return a, b
    a = rng.uniform(-1, 1, n) * np.exp2(rng.integers(-60, 20, n))  # states, areas, jumps
    a[::3] = 0.0
    return a, rng.uniform(0.5, 1, n) * np.exp2(rng.integers(-30, 10, n))


@pytest.mark.parametrize("kind", ["special", "bits", "states"])
def test_quotients_have_the_operators_bits(native, cuda_ok, kind):
    a, b = (np.ascontiguousarray(x) for x in _pairs(kind))
    bad = (C.c_int64 * 5)(-1, -1, -1, -1, -1)
    pd = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
    with np.errstate(invalid="ignore"):
        assert native.subfv_probe_quotients(pd(a), pd(b), a.size, bad) == 0
    assert list(bad) == [0, 0, 0, 0, 0]
