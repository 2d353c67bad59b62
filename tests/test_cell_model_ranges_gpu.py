"""One step of the GPU cell models (mb_ode) from states outside their usual range
against the oracle's step: a model written with other quotients and its own
exponential has to be finite, and not a number, where the reference's formulas
are.

Bars, where a value is finite: FP64 1e-9 relative (a step is a few hundred roundings);
mixed 1e-3 relative (hardware exponentials, 1e-5 at arguments near 85)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

DT = 0.02


def _steps(model, precision, states):
    """(product, oracle) states after one step of every column of states."""
    from monoalg3d_c_b200 import OdeSolver
    n = states.shape[1]
    s = OdeSolver(model, n, DT, precision=precision)
    s.set_model_initial_conditions_gpu()
    s.set_state(states)
    s.solve_model_odes_gpu(1.0)
    got = s.state()
    s.close()
    ref = np.ascontiguousarray(states.T).copy()
    L = oracle.load()
    for row in ref:
        if model == "tt2006":
            L.orc_tt2006_step(row.ctypes.data, 0.0, DT, None)
        else:
            L.orc_torord_step(row.ctypes.data, 0.0, DT, 0, 0, None)
    return got, ref.T


def _torord(state, values):
    y = np.repeat(np.array(oracle.torord_initial_state(0))[:, None], len(values), axis=1)
    y[state] = values
    return y


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("state", [2, 4, 6, 9])
def test_concentration_below_zero_is_reported(state, precision):
    """A concentration whose logarithm, root or power does not exist makes V NaN, which the
    loop reports (MB_ERR_NAN), and does not leave finite numbers behind: subspace Ca, Na and
    K below the root of the ionic strength, myoplasmic Ca below zero."""
    scale = 1.0 if state == 9 else 1000.0
    y = _torord(state, -scale * np.array([1e-6, 3e-4, 0.5, 3.0]))
    got, ref = _steps("torord", precision, y)
    bad = np.isnan(ref[0])
    assert bad.any()
    assert np.array_equal(np.isnan(got[0]), bad)


@pytest.mark.parametrize("precision,low,high", [("fp64", -3000.0, 9000.0), ("mixed", -1400.0, 1100.0)])
def test_potential_far_out(precision, low, high):
    """ten Tusscher 2006 where the reference's formulas stay finite: m's time constant is a
    product and a sum of reciprocals whose own reciprocals overflow much earlier."""
    v = np.concatenate([np.linspace(low, high, 601), [399.5, 408.8, 430.0]])
    y = np.repeat(np.array(oracle.tt2006_initial_state())[:, None], v.size, axis=1)
    y[0] = v
    got, ref = _steps("tt2006", precision, y)
    assert np.isfinite(ref).all()
    np.testing.assert_allclose(got, ref, rtol=1e-9 if precision == "fp64" else 1e-3, atol=1e-9)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_vanishing_and_large_quotients(precision):
    """ToRORd states at which a quotient formed from products is 0/0 or overflows where the
    reference's nested form has its limit: no calcium with jca = 0, a huge junctional SR load."""
    y = _torord(8, [1e6, 1e5, 1.5, 1.5, 1.5, 1.5])
    y[2, 2] = y[9, 3] = y[2, 4] = y[9, 5] = 0.0
    y[29, 2] = y[29, 3] = 0.0
    got, ref = _steps("torord", precision, y)
    assert np.isfinite(ref).all()
    np.testing.assert_allclose(got, ref, rtol=1e-9 if precision == "fp64" else 1e-3, atol=1e-7)
