"""Creating a tissue of rotating fibres with ragged rows where there is room for the flat
kernel's vectors but not for the padded ones of the z-march kernel: the tissue runs on the
flat kernel.  The room is taken by allocations of the test's own.  And what a tissue holds once
its kernel is chosen."""
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


@pytest.mark.parametrize("rotating", [True, False])
def test_kernels_not_chosen_keep_no_memory(monkeypatch, rotating):
    """After creation a tissue holds the vectors of the kernel it runs on and not those of the
    other candidates: as much as when that kernel is the only one."""
    torch = pytest.importorskip("torch")
    from monoalg3d_c_b200 import Stim, Tissue
    nx, ny, nz = 401, 101, 24
    kw = dict(assembly="anisotropic", sigma_l=0.0002, sigma_t=0.00004,
              fibre_angle_z=np.deg2rad(np.linspace(60.0, -60.0, nz))) if rotating else {}

    def held(variant):
        if variant is None:
            monkeypatch.delenv("MB_CG_VARIANT", raising=False)
        else:
            monkeypatch.setenv("MB_CG_VARIANT", str(variant))
        make = lambda: Tissue(nx, ny, nz, precision="mixed", stims=[Stim(duration=1.0)], **kw)  # noqa: E731
        make().close()                                    # kernels loaded
        before = torch.cuda.mem_get_info()[0]
        t = make()
        used, kernel = before - torch.cuda.mem_get_info()[0], t.tuning()["cg_kernel"]
        t.close()
        return used, kernel

    free, kernel = held(None)
    number = kernel if kernel < 100 else {100: 24, 200: 25}.get(kernel, 26 + kernel - 300 if kernel < 400 else
                                                              36 + kernel - 400 if kernel < 500 else 41 + kernel - 500)
    forced, again = held(number)
    assert again == kernel
    n = nx * ny * nz
    assert abs(free - forced) < 4 * n, f"kernel {kernel}: {free} bytes held, {forced} when it is the only candidate"
