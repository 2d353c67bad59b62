"""ToRORd with several sub-steps per call (the kernels that keep the state in registers
between them) against the oracle: in tissues (dt_pde = 4 dt_ode) and cell-model
objects, cell types mixed, a cell count that is no multiple of a block, every variant.

Bars: FP64 as in test_oracle_parity_gpu.py (1e-8 of V, equal iteration counts); mixed 2e-3
of the oracle, as the mixed-precision tests have it, and bit for bit between variants."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule", ["reference_cpu", "true"])
@pytest.mark.parametrize("precision,variants", [("fp64", (0, 1, 2, 3, 7)), ("mixed", (0, 1, 4))])
def test_tissue_substeps(monkeypatch, precision, variants, rule):
    from monoalg3d_c_b200 import Stim, Tissue
    nx, ny, nz, steps = 23, 7, 3, 120
    rng = np.random.default_rng(8)
    kw = dict(model="torord", dt_pde=0.04, dt_ode=0.01, rl_rule=rule, celltype=rng.integers(0, 3, nx * ny * nz),
              active=(rng.random(nx * ny * nz) >= 0.15).astype(np.uint8),
              stims=[Stim(kind="x_less_than", start=0.0, duration=1.5, current=-53.0, x_limit=500.0)])
    o = oracle.Sim(nx, ny, nz, **kw)
    o.step(steps)
    ref = o.v()
    its, _ = o.last_cg()
    o.close()
    ok = np.isfinite(ref)
    first = None
    monkeypatch.setenv("MB_CG_VARIANT", "0")
    for variant in variants:
        monkeypatch.setenv("MB_ODE_VARIANT", str(variant))
        t = Tissue(nx, ny, nz, precision=precision, **kw)
        t.step(steps)
        v, state = t.v(), t.state()
        st = t.step_stats(steps - 1, 1)["its"][0]
        t.close()
        if precision == "fp64":
            assert st == its
            np.testing.assert_allclose(v[ok], ref[ok], rtol=1e-8, atol=1e-9)
        else:
            assert np.all(np.abs(v[ok] - ref[ok]) <= 2e-3 * (np.abs(ref[ok]) + 1.0))
        if first is None:
            first = v, state
        assert np.array_equal(v[ok], first[0][ok]) and np.array_equal(state, first[1]), f"variant {variant}"


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("steps", [2, 10])
def test_object_substeps(precision, steps):
    from monoalg3d_c_b200 import OdeSolver
    n, dt = 301, 0.01
    rng = np.random.default_rng(3)
    ct = rng.integers(0, 3, n).astype(np.uint8)
    s = OdeSolver("torord", n, dt, num_steps=steps, precision=precision)
    s.set_model_initial_conditions_gpu(celltype=ct)
    ref = s.state()
    stim = np.where(rng.random(n) < 0.5, -40.0, 0.0)
    for call in range(3):
        s.solve_model_odes_gpu(call * steps * dt, stim)
    got = s.state()
    s.close()
    cells = np.ascontiguousarray(ref.T)
    L = oracle.load()
    for c in range(n):
        for _ in range(3 * steps):
            L.orc_torord_step(cells[c].ctypes.data, float(stim[c]), dt, int(ct[c]), 0, None)
    # gates down to 1e-40 in the mixed form's FP32
    rtol, atol = (1e-9, 1e-30) if precision == "fp64" else (2e-3, 1e-7)
    np.testing.assert_allclose(got, cells.T, rtol=rtol, atol=atol)
