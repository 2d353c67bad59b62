"""The double exponential, reciprocal and quotient of the cell models
(mb_math.cuh) against numpy's 80-bit long double.  Bars from their
construction, in units of the last place: mexp 0.5 (its last addition) + 2^-7
(the rounding of r (1 + r/2) relative to the table value); mrcp 0.5 + 2^-7 (the
hardware's approximation is good to 20 bits, so the first omitted term e^3 of
the Newton step is up to 2^-60 of the value, which is 2^-7 of a unit at worst);
mdiv 0.501 (its remainder correction leaves that term times 2^-53)."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _eval(fn, x, y=None):
    lib = C.CDLL(os.path.join(os.path.dirname(os.path.abspath(__file__)), "libmb_math_probe.so"))
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.ones_like(x) if y is None else np.ascontiguousarray(y, dtype=np.float64)
    out = np.empty_like(x)
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    assert lib.math_eval(C.c_int(fn), C.c_int(x.size), p(x), p(y), p(out)) == 0
    return out


def _ulps(got, ref):
    ref64 = ref.astype(np.float64)
    return np.max(np.abs(got.astype(np.longdouble) - ref) / np.spacing(np.abs(ref64)).astype(np.longdouble))


@pytest.mark.parametrize("lo,hi", [(-700.0, 700.0), (-40.0, 40.0), (-1.0, 1.0), (-1e-3, 1e-3)])
def test_exponential(lo, hi):
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(lo, hi, 400_000), [0.0, lo, hi],
                        # the edges of the table's intervals
                        (np.arange(-300, 300) + 0.5) * np.log(2.0) / 128 * (hi / 700.0 if hi >= 1 else hi)])
    assert _ulps(_eval(0, x), np.exp(x.astype(np.longdouble))) <= 0.52


def test_exponential_outside():
    """Beyond +-700 the value at about +-700 (the low word is kept: 0.07 at most)."""
    got = _eval(0, np.array([701.0, 1e5, 1e300, np.inf, -701.0, -1e5, -1e300, -np.inf]))
    assert (got[:4] >= np.exp(699.99)).all() and (got[:4] <= np.exp(700.07)).all()
    assert (got[4:] <= np.exp(-699.99)).all() and (got[4:] >= np.exp(-700.07)).all()
    assert np.isnan(_eval(0, np.array([np.nan, -np.nan]))).all()


def test_reciprocal_and_quotient():
    rng = np.random.default_rng(4)
    x = np.exp(rng.uniform(-690.0, 690.0, 400_000)) * rng.choice([-1.0, 1.0], 400_000)
    assert _ulps(_eval(1, x), 1.0 / x.astype(np.longdouble)) <= 0.5 + 2.0 ** -7
    a, b = np.exp(rng.uniform(-200, 200, 400_000)), np.exp(rng.uniform(-200, 200, 400_000))
    assert _ulps(_eval(2, a, b), a.astype(np.longdouble) / b.astype(np.longdouble)) <= 0.501
    # beyond the largest exponential the reciprocal is 0 or its subnormal value, not NaN
    assert np.all(np.abs(_eval(1, np.array([1.5e307, np.exp(700.0) * 1e3]))) < 1e-306)
    assert np.isnan(_eval(1, np.array([np.nan]))).all() and np.isnan(_eval(2, np.array([np.nan]))).all()
