"""What choosing its kernels adds to creating a small tissue: the tuners time a few
candidates, chosen by the tissue's size and operator, not every shape there is.

Bars: twice the time measured (the smallest of eight creations, so that only the host's
slowest moments could exceed it); with every shape a candidate the same differences were 5.3
and 11.6 ms."""
import time

import pytest

pytestmark = pytest.mark.gpu


def _create(monkeypatch, shape, **env):
    from monoalg3d_c_b200 import Stim, Tissue
    for k in ("MB_CG_VARIANT", "MB_ODE_VARIANT"):
        if k in env:
            monkeypatch.setenv(k, env[k])
        else:
            monkeypatch.delenv(k, raising=False)
    best = 1e9
    for _ in range(8):
        t0 = time.perf_counter()
        t = Tissue(*shape, model="tt2006", stims=[Stim(duration=1.0)])
        best = min(best, time.perf_counter() - t0)
        t.close()
    return 1e3 * best


@pytest.mark.parametrize("shape,bar_ms", [((400, 1, 1), 2.6), ((100, 100, 20), 7.0)])
def test_tuners_share(monkeypatch, shape, bar_ms):
    tuned = _create(monkeypatch, shape)
    fixed = _create(monkeypatch, shape, MB_CG_VARIANT="0", MB_ODE_VARIANT="0")
    assert tuned - fixed < bar_ms, f"{tuned:.1f} ms tuned, {fixed:.1f} ms with the kernels given"
