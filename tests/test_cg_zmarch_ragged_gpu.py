"""The z-march CG on grids whose rows are no multiple of 4 cells (its vectors'
rows are padded): 1, 2 and 3 cells in the last group, rows that end just before,
at and after a 128-cell tile, few rows, one plane; every variant that takes
padded rows against the flat kernel, V written from outside in between (the
fused form's stored product is then stale).

FP64: the same iteration counts, V to 1e-8.  Mixed: counts within one, V within
1e-5 mV over the 16 steps (each solve stops at r.r <= 1e-16, 3e-7 mV)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(shape, precision, variant):
    from monoalg3d_c_b200 import Stim, Tissue
    nx, ny, nz = shape
    old = os.environ.get("MB_CG_VARIANT")
    os.environ["MB_CG_VARIANT"] = str(variant)
    try:
        t = Tissue(nx, ny, nz, model="tt2006", precision=precision, assembly="anisotropic", sigma_l=0.0002,
                   sigma_t=0.00004, fibre_angle_z=np.deg2rad(np.linspace(60.0, -60.0, nz) if nz > 1 else [30.0]),
                   stims=[Stim(kind="x_y_limits", start=0.0, duration=1.0, current=-53.0, min=(0.0, 0.0, 0.0),
                               max=(100.0 * nx / 3, 100.0 * ny / 2, 0.0)),
                          Stim(kind="x_y_limits", start=0.1, duration=1.0, current=-53.0,
                               min=(100.0 * (nx - 3), 0.0, 0.0), max=(100.0 * nx, 100.0 * ny, 0.0))])
    finally:
        os.environ.pop("MB_CG_VARIANT")
        if old is not None:
            os.environ["MB_CG_VARIANT"] = old
    kernel = t.tuning()["cg_kernel"]
    t.step(8)
    v = t.v()
    t.set_v(v + 0.5 * np.sin(np.arange(v.size)))
    t.step(8)
    v = t.v()
    t.sync()
    its = t.step_stats(0, 16)["its"]
    t.close()
    return kernel, v, its


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(9, 5, 4), (18, 7, 3), (31, 4, 5), (125, 3, 4), (127, 9, 3), (129, 6, 4), (130, 17, 3),
                                   (131, 5, 2), (258, 9, 3), (37, 11, 1)])
def test_ragged_rows_match_flat(shape, precision):
    from monoalg3d_c_b200._lib import lib
    from monoalg3d_c_b200.monodomain import cg_launch_shapes
    k0, v0, i0 = _run(shape, precision, 0)
    assert k0 == 0
    first = cg_launch_shapes() + 2
    # mixed 4..6 are the window form (whole rows only), FP64 has no 7..9
    takes = set(range(7)) if precision == "fp64" else {0, 1, 2, 3, 7, 8, 9}
    for z in range(lib.mbk_zcg_variants()):
        k, v, i = _run(shape, precision, first + z)
        assert k == (300 + z if z in takes else 0)
        if z not in takes:
            continue
        if precision == "fp64":
            assert np.array_equal(i, i0), f"variant {z}: iterations {i} against {i0}"
            np.testing.assert_allclose(v, v0, rtol=1e-8, atol=1e-9)
        else:
            assert np.abs(i - i0).max() <= 1, f"variant {z}: iterations {i} against {i0}"
            np.testing.assert_allclose(v, v0, rtol=0, atol=1e-5)
