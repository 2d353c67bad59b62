"""The reverse sweep of the cell model's step (adj_cell) on both sides of each
of its branches: starting potentials below and above the -40 mV switch of the
h and j rates, at the L-type current's removable singularity (15 mV, where the
band's limit value is used) and beside it, and a loaded calcium state.

Bars: FP64 within 1e-6 of the oracle's FP64 tangent-linear loop, of the summed
magnitudes of the direction's terms (both differentiate the same FP64
arithmetic; the loop's solves stop at r.r <= 1e-24); mixed within 1e-3 of the
FP64 adjoint (FP32 Jacobian, as tests/test_adjoint_gpu.py has it)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("v0,loaded", [(-90.0, False), (-40.5, False), (-39.5, False), (14.0, False), (15.0, True),
                                       (30.0, True)])
def test_cell_reverse_sweep(v0, loaded):
    from monoalg3d_c_b200 import Stim
    from monoalg3d_c_b200.adjoint import Adjoint
    nx, ny, steps, every = 9, 7, 40, 8
    rng = np.random.default_rng(17)
    n = nx * ny
    sigma = 0.00013 * np.exp(0.3 * rng.standard_normal(n))
    gkr = np.exp(0.2 * rng.standard_normal(n)).astype(np.float32).astype(np.float64)
    sensors = rng.choice(n, size=5, replace=False)
    y0 = np.array(oracle.tt2006_initial_state())
    y0[0] = v0
    y0[1:3] = 0.3
    if loaded:
        y0[7:11] = 0.5
        y0[13:16] = (0.0008, 2.9, 0.05)
    kw = dict(initial_state=y0, initial_v=v0, cg_tolerance=1e-24, cg_max_iterations=500,
              stims=[Stim(kind="x_less_than", start=0.0, duration=0.4, current=-53.0, x_limit=300.0)])
    out = {}
    for precision in ("fp64", "mixed"):
        a = Adjoint(nx, ny, 1, sigma, gkr, sensors, nsteps=steps, sample_every=every, checkpoint_every=11,
                    precision=precision, **kw)
        target = a.forward(sigma, gkr) + rng.standard_normal((steps // every, 5))
        tr = a.forward(sigma, gkr)
        out[precision] = (target, tr)
        w = out["fp64"][1] - out["fp64"][0]          # the same misfit gradient for both
        out[precision] += a.backward(w)
        a.close()
    target, _, gs, gk = out["fp64"]
    _, _, ms, mk = out["mixed"]
    sc = np.ones((5, n))
    sc[1] = gkr
    for trial in range(2):
        d = rng.standard_normal(n)
        for g, m, x, key in ((gs, ms, sigma, "dsigma"), (gk, mk, gkr, "dgkr")):
            _, ref = oracle.tangent_misfit(nx, ny, 1, steps, every, sensors, target, assembly="per_cell",
                                           sigma_cell=sigma, current_scale=sc, **{key: x * d}, **kw)
            size = float(np.sum(np.abs(g * x * d)))
            assert size > 0
            ad = float(np.sum(g * x * d))
            assert abs(ad - ref) <= 1e-6 * size, f"{key} {trial}: adjoint {ad:.12e}, tangent {ref:.12e}"
            mixed = float(np.sum(m * x * d))
            assert abs(mixed - ad) <= 1e-3 * size, f"{key} {trial}: mixed {mixed:.9e}, FP64 {ad:.9e}"
