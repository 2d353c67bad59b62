"""The adjoint's transposed solves (explicit right-hand side, own unknown and control
block) on every CG kernel they can run on: flat shapes, clusters of 2^v blocks, fused
shapes, forced through MB_CG_VARIANT on a sheet with removed cells and rows of whole
4-cell groups; gradients against flat shape 0.

Bars: the solves stop at r.r <= 1e-24 lambda.lambda in every form and the forward loop at
r.r <= 1e-20, so FP64 gradients agree to 1e-7 of their largest entry; mixed to 1e-3 (FP32
Jacobian on states that differ by the solves' rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(monkeypatch, precision, variant):
    from monoalg3d_c_b200 import Stim
    from monoalg3d_c_b200.adjoint import Adjoint
    nx, ny, steps = 40, 30, 60
    n = nx * ny
    rng = np.random.default_rng(12)
    active = (rng.random(n) >= 0.1).astype(np.uint8)
    sigma = 0.00013 * np.exp(0.3 * rng.standard_normal(n))
    gkr = np.exp(0.2 * rng.standard_normal(n)).astype(np.float32).astype(np.float64)
    sensors = rng.choice(np.flatnonzero(active), 6, replace=False)
    monkeypatch.setenv("MB_CG_VARIANT", str(variant))
    a = Adjoint(nx, ny, 1, sigma, gkr, sensors, nsteps=steps, sample_every=10, checkpoint_every=16,
                precision=precision, active=active, cg_tolerance=1e-20,
                stims=[Stim(kind="x_less_than", start=0.0, duration=0.6, current=-53.0, x_limit=500.0)])
    tr = a.forward(sigma, gkr)
    g = a.backward(rng.standard_normal(tr.shape))
    a.close()
    return tr, g


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_every_solver_gives_the_same_gradient(monkeypatch, precision):
    from monoalg3d_c_b200._lib import lib
    from monoalg3d_c_b200.monodomain import cg_launch_shapes
    nf = cg_launch_shapes()
    c0 = nf + 2 + lib.mbk_zcg_variants()
    f0 = c0 + lib.mbk_ccg_variants()
    tr0, g0 = _gradient(monkeypatch, precision, 0)
    bar = 1e-7 if precision == "fp64" else 1e-3
    clusters = [c0 + c for c in range(lib.mbk_ccg_variants()) if c <= 3]       # 128 cells a block at least
    for v in [5, 12, 22] + clusters + [f0 + f for f in range(lib.mbk_ffcg_variants())]:
        tr, g = _gradient(monkeypatch, precision, v)
        np.testing.assert_allclose(tr, tr0, rtol=0, atol=1e-6 if precision == "fp64" else 1e-3)
        for a, b in zip(g, g0):
            assert np.abs(b).max() > 0
            assert np.abs(a - b).max() <= bar * np.abs(b).max(), f"kernel {v}: {np.abs(a - b).max() / np.abs(b).max():.2e}"
