"""The one-launch CSR CG (mb_csr_solve) against the oracle's cpu_conjugate_gradient:
one row, fewer rows than a warp takes, a last block partly empty, rows of 1 to 5
entries (four lanes a row) and of about 40 (sixteen), empty off-diagonals,
without preconditioner, an exact starting value and a limit of iterations.

Bars: the same iteration counts; x to 1e-10 relative to the largest value (both stop at
the same r.r, and differ by rounding, 1e-16 times the condition number, below
100 here)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def _spd(n, band, seed):
    """Diagonally dominant symmetric matrix with `band` random couplings per row,
    the diagonal first in each row (as the reference stores it)."""
    rng = np.random.default_rng(seed)
    rows = [dict() for _ in range(n)]
    for i in range(n):
        for j in rng.integers(0, n, band):
            if i != j:
                c = -rng.uniform(0.1, 1.0)
                rows[i][int(j)] = c
                rows[int(j)][i] = c
    ptr, col, val = [0], [], []
    for i, r in enumerate(rows):
        js = sorted(r)
        col += [i] + js
        val += [0.7 - sum(r.values())] + [r[j] for j in js]
        ptr.append(len(col))
    return np.array(ptr, dtype=np.int32), np.array(col, dtype=np.int32), np.array(val)


@pytest.mark.parametrize("n,band", [(1, 0), (7, 1), (130, 2), (3001, 0), (3001, 2), (20011, 1), (900, 20)])
@pytest.mark.parametrize("pre", [True, False])
def test_matches_oracle(n, band, pre):
    from monoalg3d_c_b200 import csr_conjugate_gradient
    ptr, col, val = _spd(n, band, n + band)
    rng = np.random.default_rng(9)
    b, x0 = rng.standard_normal(n), 0.1 * rng.standard_normal(n)
    for most in (200, 4):
        xr, ir, er = oracle.pcg(ptr, col, val, b, x0, 1e-20, most, pre)
        x, i, e = csr_conjugate_gradient(ptr, col, val, b, x0, 1e-20, most, pre)
        assert i == ir
        # r.r that cancels in one iteration is rounding: compare it where it is not
        assert e == pytest.approx(er, rel=1e-6, abs=1e-24)
        np.testing.assert_allclose(x, xr, rtol=0, atol=1e-10 * max(1.0, np.abs(xr).max()))
    again, i, _ = csr_conjugate_gradient(ptr, col, val, b, xr, 1.0 + er, 200, pre)
    assert i == 1 and np.array_equal(again, xr)          # already below the tolerance: nothing moves
