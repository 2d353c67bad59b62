"""The CG kernels with one reduction per iteration -- the cluster kernel
(cg_cluster.cu) at every cluster size and the fused flat form (cg_flat.cu) in every
shape -- against the flat persistent kernel with two: blocks that own a few rows or less than a z-plane (neighbours two
blocks away), a last block that is partly or wholly empty, removed cells,
per-cell conductivity, 27-point rows, no preconditioner, and a first step whose
residual vanishes in one iteration (the recurred sums cancel).

FP64: the same iteration counts and V to 1e-8 (the bar of the CG variants).
Mixed: counts within one; both forms stop at r.r <= 1e-16, so a solve
differs by at most 2 sqrt(1e-16) / alpha = 3e-7 mV, 1e-5 over the 30 steps."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = {"cable": (130, 1, 1), "sheet": (97, 23, 1), "slab": (40, 33, 3), "thick": (24, 20, 9), "ragged": (31, 9, 8),
          "wide": (160, 96, 10)}


def _kw(form, nx, ny, nz):
    from monoalg3d_c_b200 import Stim
    n = nx * ny * nz
    rng = np.random.default_rng(5)
    kw = dict(stims=[Stim(kind="x_less_than", start=0.1, duration=1.0, current=-53.0, x_limit=500.0)])
    if form == "removed":
        kw.update(active=(rng.random(n) >= 0.2).astype(np.uint8), sigma=(0.00013,) * 3)
    elif form == "percell":
        kw.update(assembly="per_cell", sigma_cell=0.00013 * np.exp(0.3 * rng.standard_normal(n)))
    elif form == "rotating":
        kw.update(assembly="anisotropic", sigma_l=0.0002, sigma_t=0.00004,
                  fibre_angle_z=np.deg2rad(np.linspace(60.0, -60.0, nz)))
    elif form == "plain":
        kw.update(use_preconditioner=False)
    return kw


def _run(shape, precision, variant, **kw):
    from monoalg3d_c_b200 import Tissue
    old = os.environ.get("MB_CG_VARIANT")
    os.environ["MB_CG_VARIANT"] = str(variant)
    try:
        t = Tissue(*shape, model="torord", precision=precision, **kw)
    finally:
        os.environ.pop("MB_CG_VARIANT")
        if old is not None:
            os.environ["MB_CG_VARIANT"] = old
    kernel = t.tuning()["cg_kernel"]
    t.step(30)
    v = t.v()
    t.sync()
    st = t.step_stats(0, 30)
    t.close()
    return kernel, v, st["its"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,form", [("cable", "iso"), ("sheet", "removed"), ("slab", "iso"), ("slab", "plain"),
                                        ("thick", "percell"), ("thick", "removed"), ("ragged", "rotating"),
                                        ("slab", "rotating")])
def test_clusters_match_flat(shape, form, precision):
    from monoalg3d_c_b200._lib import lib
    from monoalg3d_c_b200.monodomain import cg_launch_shapes
    size = SHAPES[shape]
    kw = _kw(form, *size)
    k0, v0, i0 = _run(size, precision, 0, **kw)
    assert k0 == 0
    first = cg_launch_shapes() + 2 + lib.mbk_zcg_variants()
    ran = 0
    for c in range(lib.mbk_ccg_variants()):
        k, v, i = _run(size, precision, first + c, **kw)
        if k != 400 + c:
            assert (1 << c) * 128 > v.size, f"cluster of {1 << c} blocks not used"
            continue
        ran += 1
        ok = np.isfinite(v0)
        assert np.array_equal(ok, np.isfinite(v))
        if precision == "fp64":
            assert np.array_equal(i, i0), f"cluster of {1 << c}: iterations {i} against {i0}"
            np.testing.assert_allclose(v[ok], v0[ok], rtol=1e-8, atol=1e-9)
        else:
            assert np.abs(i - i0).max() <= 1, f"cluster of {1 << c}: iterations {i} against {i0}"
            np.testing.assert_allclose(v[ok], v0[ok], rtol=0, atol=1e-5)
    assert ran >= 1


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,form", [("cable", "iso"), ("sheet", "removed"), ("slab", "iso"), ("slab", "plain"),
                                        ("thick", "percell"), ("thick", "removed"), ("wide", "removed")])
def test_fused_shapes_match_flat(shape, form, precision):
    from monoalg3d_c_b200._lib import lib
    from monoalg3d_c_b200.monodomain import cg_launch_shapes
    size = SHAPES[shape]
    kw = _kw(form, *size)
    k0, v0, i0 = _run(size, precision, 0, **kw)
    assert k0 == 0
    first = cg_launch_shapes() + 2 + lib.mbk_zcg_variants() + lib.mbk_ccg_variants()
    ok = np.isfinite(v0)
    for f in range(lib.mbk_ffcg_variants()):
        k, v, i = _run(size, precision, first + f, **kw)
        if lib.mbk_ffcg_variant_groups(f) and size[0] % 4:
            assert k == 0
            continue
        assert k == 500 + f
        assert np.array_equal(ok, np.isfinite(v))
        if precision == "fp64":
            assert np.array_equal(i, i0), f"fused shape {f}: iterations {i} against {i0}"
            np.testing.assert_allclose(v[ok], v0[ok], rtol=1e-8, atol=1e-9)
        else:
            assert np.abs(i - i0).max() <= 1, f"fused shape {f}: iterations {i} against {i0}"
            np.testing.assert_allclose(v[ok], v0[ok], rtol=0, atol=1e-5)
