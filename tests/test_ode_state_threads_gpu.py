"""mb_ode_get_state / set_state of one cell-model object from several host threads at
once: every call works in a dense buffer of its own, whether the object keeps one
between calls (small states) or not (above 256 MiB)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,calls", [(3000, 30), (790_000, 2)])
def test_states_read_by_several_threads(cells, calls):
    from monoalg3d_c_b200 import OdeSolver
    s = OdeSolver("torord", cells, 0.02, precision="mixed")
    s.set_model_initial_conditions_gpu()
    s.solve_model_odes_gpu(0.0)
    ref = s.state()
    wrong = []

    def read():
        for _ in range(calls):
            if not np.array_equal(s.state(), ref):
                wrong.append(1)

    def write():
        for _ in range(calls):
            s.set_state(ref)

    threads = [threading.Thread(target=f) for f in (read, read, read, write)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    assert np.array_equal(s.state(), ref)
    s.close()
