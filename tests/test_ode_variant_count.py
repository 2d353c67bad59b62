"""The launch variants of a cell model that differ, which are those the tissue's tuner
times: several sub-steps per call have no staged or slot forms (host logic, no GPU)."""
import pytest


@pytest.mark.parametrize("model,precision,num_steps,adaptive,variants", [
    ("tt2006", "fp64", 1, 0, 10), ("tt2006", "mixed", 5, 0, 10), ("torord", "fp64", 1, 0, 10),
    ("torord", "mixed", 1, 0, 10), ("torord", "fp64", 2, 0, 4), ("torord", "mixed", 2, 0, 2),
    ("torord_endo", "fp64", 1, 0, 4), ("torord_endo", "fp64", 1, 1, 1)])
def test_variants_that_differ(model, precision, num_steps, adaptive, variants):
    from monoalg3d_c_b200._lib import lib
    from monoalg3d_c_b200.monodomain import MODELS, PRECISIONS
    assert lib.mbk_ode_variants(MODELS[model], PRECISIONS[precision], num_steps, adaptive) == variants
