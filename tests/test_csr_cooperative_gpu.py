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


def _pcg(ptr, col, val, b, inv, tol):
    """Jacobi-PCG with the given 1/diag (its, x), the iteration of cpu_conjugate_gradient."""
    rows = np.repeat(np.arange(b.size), np.diff(ptr))
    mul = lambda p: np.bincount(rows, val * p[col], b.size)  # noqa: E731
    x, r = np.zeros_like(b), b.copy()
    p = inv * r
    rz, its = r @ p, 1
    while r @ r >= tol and its < 200:
        q = mul(p)
        alpha = rz / (p @ q)
        x += alpha * p
        r -= alpha * q
        z = inv * r
        rz, old = r @ z, rz
        p = z + rz / old * p
        its += 1
        if r @ r <= tol:
            break
    return its, x


@pytest.mark.parametrize("n,band", [(700, 2), (600, 20)])
def test_repeated_diagonal_entries(n, band):
    """A row whose diagonal comes in several entries is preconditioned by the last of
    them, wherever in the row they lie (the product takes their sum)."""
    from monoalg3d_c_b200 import csr_conjugate_gradient
    ptr, col, val = _spd(n, band, 5)
    rng = np.random.default_rng(6)
    out, cols, vals, inv = [0], [], [], np.empty(n)
    for i in range(n):
        c, v = list(col[ptr[i] + 1:ptr[i + 1]]), list(val[ptr[i] + 1:ptr[i + 1]])
        parts = val[ptr[i]] * rng.dirichlet(np.full(3, 4.0))
        at = sorted(rng.integers(0, len(c) + 1, 3), reverse=True)
        for k, d in zip(at, parts):
            c.insert(k, i)
            v.insert(k, d)
        cols += c
        vals += v
        inv[i] = 1.0 / v[len(c) - 1 - c[::-1].index(i)]
        out.append(len(cols))
    ptr, col, val = np.array(out, dtype=np.int32), np.array(cols, dtype=np.int32), np.array(vals)
    b = rng.standard_normal(n)
    its, x = _pcg(ptr, col, val, b, inv, 1e-20)
    got, i, _ = csr_conjugate_gradient(ptr, col, val, b, None, 1e-20, 200, True)
    assert 10 < its < 200 and abs(i - its) <= 1
    np.testing.assert_allclose(got, x, rtol=0, atol=1e-9 * np.abs(x).max())


@pytest.mark.parametrize("n,nnz,blocks", [(1, 1, 1), (128, 16 * 128, 1), (129, 16 * 129, 2), (900, 40 * 900, 29),
                                          (33, 17 * 33, 2)])
def test_blocks_cover_the_rows(n, nnz, blocks):
    """A small solve gets a block for every 512 lanes its rows take (4 or 16 lanes a row)."""
    from monoalg3d_c_b200._lib import lib
    assert lib.mbk_csr_pcg_blocks(n, nnz) == blocks


@pytest.mark.parametrize("n", [870_000, 1_400_003])
def test_beyond_l2(n):
    """Matrices that stay in L2 are solved in one launch, larger ones by a kernel per
    phase, with the same iterations: a chain of n rows on either side of the line
    (matrix and vectors 80 and 128 MB)."""
    from monoalg3d_c_b200 import csr_conjugate_gradient
    from monoalg3d_c_b200._lib import lib
    i = np.arange(n)
    col = np.stack([i, (i - 1) % n, (i + 1) % n], axis=1).reshape(-1)
    val = np.tile([2.5, -1.0, -1.0], n)
    val[1] = val[-1] = 0.0                     # no wrap-around
    ptr = np.arange(n + 1) * 3
    assert lib.mbk_csr_in_l2(n, 3 * n) == (n < 1_000_000)
    rng = np.random.default_rng(4)
    b = rng.standard_normal(n)
    for most in (200, 17):
        xr, ir, er = oracle.pcg(ptr.astype(np.int32), col.astype(np.int32), val, b, np.zeros(n), 1e-8, most, True)
        x, k, e = csr_conjugate_gradient(ptr, col, val, b, None, 1e-8, most, True)
        assert k == ir and e == pytest.approx(er, rel=1e-6)
        np.testing.assert_allclose(x, xr, rtol=0, atol=1e-10 * np.abs(xr).max())
