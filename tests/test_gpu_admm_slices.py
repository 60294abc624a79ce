"""The ADMM system on sliced rows: K v and the inner solve at sizes where the layout can go wrong
(windows of 256, slices of 32, empty rows, no constraint rows), and on a row too long for a lane,
which stays in CSR.

K v is compared with a product formed here in FP64: each row sums at most 300 products, so the two
orders of summation differ by at most 300 * 2^-53 of the row's absolute sum (3.4e-14; 1e-13 asked for).
The solve is checked by its residual, formed here, against the accuracy asked for (plus the rounding of
the recurrence, 1e-12 of max|rhs|)."""
import numpy as np
import pytest

from boxqp.admm import AdmmSystem

pytestmark = pytest.mark.gpu


def csr(rows, cols, vals, m):
    order = np.lexsort((cols, rows))
    ptr = np.zeros(m + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=m), out=ptr[1:])
    return ptr, cols[order].astype(np.int32), vals[order], rows[order]


def system(n, m, per_row, wide, rng):
    """H: random symmetric couplings plus a dominant diagonal; A: `per_row` entries a row, every seventh
    row empty, the first row `wide` entries."""
    a, b = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
    key = np.unique(np.minimum(a, b) * n + np.maximum(a, b))
    lo, hi = key // n, key % n
    lo, hi = lo[lo != hi], hi[lo != hi]
    w = rng.uniform(0.1, 1.0, len(lo))
    diag = rng.uniform(0.5, 2.0, n)
    np.add.at(diag, lo, w)
    np.add.at(diag, hi, w)
    i = np.arange(n)
    h = csr(np.concatenate([lo, hi, i]), np.concatenate([hi, lo, i]), np.concatenate([-w, -w, diag]), n)
    rows, cols = [], []
    for r in range(m):
        k = min(n, wide) if r == 0 else 0 if r % 7 == 3 else min(n, per_row)
        rows.append(np.full(k, r))
        cols.append(rng.choice(n, k, replace=False))
    rows = np.concatenate(rows) if m else np.zeros(0, np.int64)
    cols = np.concatenate(cols) if m else np.zeros(0, np.int64)
    return h, csr(rows, cols, rng.normal(size=len(rows)), m)


def times(mat, v, m):
    return np.bincount(mat[3], weights=mat[2] * v[mat[1]], minlength=m)[:m]


def transposed(mat, t, n):
    return np.bincount(mat[1], weights=mat[2] * t[mat[3]], minlength=n)[:n]


@pytest.mark.parametrize('n,m,per_row,wide', [(1, 1, 1, 1), (31, 0, 4, 4), (33, 7, 4, 4), (256, 255, 8, 8), (257, 300, 8, 100),
                                              (513, 257, 8, 127), (2000, 900, 8, 200), (5003, 1025, 5, 5)])
def test_product_and_solve(n, m, per_row, wide):
    rng = np.random.default_rng(n + m)
    h, a = system(n, m, per_row, wide, rng)
    rho = np.where(rng.random(m) < 0.3, 10.0, 0.1)
    sigma = 1e-6
    s = AdmmSystem(h[0], h[1], h[2], a[0], a[1], a[2], n)
    try:
        s.set_rho(rho, sigma)
        v = rng.normal(size=n)
        ref = times(h, v, n) + sigma * v + transposed(a, rho * times(a, v, m), n)
        size = times((h[0], h[1], np.abs(h[2]), h[3]), np.abs(v), n) + transposed(
            (a[0], a[1], np.abs(a[2]), a[3]), rho * times((a[0], a[1], np.abs(a[2]), a[3]), np.abs(v), m), n)
        assert np.all(np.abs(s.apply(v) - ref) <= 1e-13 * (size + 1.0))
        rhs = rng.normal(size=n)
        top = float(np.max(np.abs(rhs)))
        x, inner, resid = s.solve(rhs, np.zeros(n), 1e-9 * top, 4000)
        assert resid <= 1e-9 * top and inner > 0
        left = rhs - (times(h, x, n) + sigma * x + transposed(a, rho * times(a, x, m), n))
        assert np.max(np.abs(left)) <= 1e-9 * top + 1e-12 * top * (1.0 + float(np.max(size)))
    finally:
        s.close()


@pytest.mark.parametrize('n', [38912, 38913, 77825, 155649])
def test_product_and_solve_at_the_edges_of_the_grid(n):
    """1216 slices: a slice for each of eight warps on 152 SMs; one more; two blocks' worth and one more;
    and one more than the largest grid has warps (the rows and the bounds are those above)."""
    test_product_and_solve(n, 33, 4, 100)
