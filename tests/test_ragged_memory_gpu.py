"""Creating a tissue of rotating fibres with ragged rows where there is room for the flat
kernel's vectors but not for the padded ones of the z-march kernel: the tissue runs on the
flat kernel.  The room is taken by allocations of the test's own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _create(monkeypatch, variant):
    from monoalg3d_c_b200 import MonoAlgError, Stim, Tissue
    nx, ny, nz = 77, 50, 40
    if variant is None:
        monkeypatch.delenv("MB_CG_VARIANT", raising=False)
    else:
        monkeypatch.setenv("MB_CG_VARIANT", str(variant))
    try:
        t = Tissue(nx, ny, nz, precision="mixed", assembly="anisotropic", sigma_l=0.0002, sigma_t=0.00004,
                   fibre_angle_z=np.deg2rad(np.linspace(60.0, -60.0, nz)), stims=[Stim(duration=1.0)])
    except MonoAlgError:
        return None
    t.step(20)
    v, kernel = t.v(), t.tuning()["cg_kernel"]
    t.close()
    return kernel, v


def test_falls_back_when_memory_is_short(monkeypatch):
    torch = pytest.importorskip("torch")
    plenty, flat = _create(monkeypatch, None), _create(monkeypatch, 0)
    assert plenty[0] >= 300 and flat[0] == 0
    _create(monkeypatch, 12)                              # load the kernels while there is room
    torch.cuda.synchronize()
    ran, fell_back = 0, 0
    for room in range(130, 20, -6):
        hog = []
        free = torch.cuda.mem_get_info()[0]
        if free > room * MB:
            hog.append(torch.empty(free - room * MB, dtype=torch.uint8, device="cuda"))
        least = _create(monkeypatch, 0)
        got = _create(monkeypatch, None) if least else None
        del hog
        torch.cuda.empty_cache()
        if least is None:
            break
        assert got is not None, f"{room} MB: the flat kernel's tissue fits, the default one is refused"
        np.testing.assert_allclose(got[1], flat[1], rtol=0, atol=1e-4)
        ran += 1
        fell_back += got[0] < 300
    assert ran >= 3 and fell_back >= 1
    assert _create(monkeypatch, None)[0] >= 300           # the refusal leaves no error behind
