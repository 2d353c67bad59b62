"""The numbers MB_CG_VARIANT takes: 0..23 the flat shapes, 24 the tiled kernel, 25 the
resident one, 26.. the z-march variants, 36.. the clusters, 41.. the fused flat shapes.
A run that is pinned to a kernel by its number gets that kernel in every version."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("number,kernel,rotating", [(1, 1, False), (16, 16, False), (23, 23, True), (24, 100, False),
                                                    (25, 200, False), (26, 300, True), (33, 307, True),
                                                    (35, 309, True), (37, 401, False), (41, 500, False)])
def test_number_selects_its_kernel(monkeypatch, number, kernel, rotating):
    from monoalg3d_c_b200 import Stim, Tissue
    from monoalg3d_c_b200.monodomain import cg_launch_shapes
    assert cg_launch_shapes() == 24
    nx, ny, nz = 24, 12, 5
    kw = dict(assembly="anisotropic", sigma_l=0.0002, sigma_t=0.00004,
              fibre_angle_z=np.deg2rad(np.linspace(60, -60, nz))) if rotating else {}
    monkeypatch.setenv("MB_CG_VARIANT", str(number))
    t = Tissue(nx, ny, nz, precision="mixed", stims=[Stim(duration=1.0)], **kw)
    assert t.tuning()["cg_kernel"] == kernel
    t.close()
