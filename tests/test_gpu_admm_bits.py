"""The ADMM inner solve against the CPU oracle that runs the kernels' order of sums: K x, x, the CG count
and the final max|r|, bit for bit.

The sizes are those where the order can go wrong: fewer rows than a warp or a block has, one past a block
(64 rows of the product, 256 elements of the vectors), one past the largest grid (38,912 rows, 155,648
elements: a second turn), empty and wide rows, no rows of A.  The oracle itself is held against a
product formed by numpy here (CPU)."""
import numpy as np
import pytest

from boxqp.admm import AdmmSystem
from oracle import oracle as O

SIZES = [(1, 1, 1, 1), (31, 0, 4, 4), (65, 7, 4, 4), (257, 300, 8, 100), (2000, 900, 8, 200), (38913, 33, 4, 100),
         (155649, 20001, 3, 200)]


def csr(rows, cols, vals, m):
    order = np.lexsort((cols, rows))
    ptr = np.zeros(m + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=m), out=ptr[1:])
    return ptr, cols[order].astype(np.int32), vals[order], rows[order]


def system(n, m, per_row, wide, rng):
    """H: random symmetric couplings plus a dominant diagonal; A: about `per_row` entries a row, every
    seventh row empty, the first row `wide` entries."""
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
    count = np.where(np.arange(m) % 7 == 3, 0, min(n, per_row))
    count[:1] = min(n, wide)
    key = np.unique(np.repeat(np.arange(m), count) * n + rng.integers(0, n, int(count.sum())))
    return h, csr(key // n, key % n, rng.normal(size=len(key)), m)


def case(n, m, per_row, wide):
    rng = np.random.default_rng(n + m)
    h, a = system(n, m, per_row, wide, rng)
    rho = np.where(rng.random(m) < 0.3, 10.0, 0.1)
    return h, a, rho, rng.normal(size=n), 0.1 * rng.normal(size=n)


def times(mat, v, rows):
    return np.bincount(mat[3], weights=mat[2] * v[mat[1]], minlength=rows)[:rows]


@pytest.mark.parametrize('n,m,per_row,wide', SIZES)
def test_the_oracle_solves_the_system(n, m, per_row, wide):
    """The two orders of a row's sum differ by at most 300 * 2^-53 of its absolute sum (3.4e-14; 1e-13
    asked for); the residual is that of numpy's product."""
    h, a, rho, rhs, x0 = case(n, m, per_row, wide)
    sigma, top = 1e-6, float(np.max(np.abs(rhs)))
    x, inner, resid, product = O.admm_solve(h, a, n, rho, sigma, rhs, x0, 1e-9 * top, 4000)

    def k_times(v, size=False):
        f = np.abs if size else (lambda z: z)
        hh, aa = (h[0], h[1], f(h[2]), h[3]), (a[0], a[1], f(a[2]), a[3])
        t = rho * times(aa, f(v), m)
        return times(hh, f(v), n) + sigma * f(v) + np.bincount(a[1], weights=aa[2] * t[a[3]], minlength=n)

    assert np.all(np.abs(product - k_times(x0)) <= 1e-13 * (k_times(x0, True) + 1.0))
    assert inner > 0 and resid <= 1e-9 * top
    assert np.max(np.abs(rhs - k_times(x))) <= 1e-9 * top + 1e-12 * (top + float(np.max(k_times(x, True))))


@pytest.mark.gpu
@pytest.mark.parametrize('n,m,per_row,wide', SIZES)
def test_the_bits_of_the_inner_solve(n, m, per_row, wide):
    h, a, rho, rhs, x0 = case(n, m, per_row, wide)
    sigma, accuracy = 1e-6, 1e-9 * float(np.max(np.abs(rhs)))
    s = AdmmSystem(*h[:3], *a[:3], n)
    try:
        s.set_rho(rho, sigma)
        for most in (3, 4000):
            ref, inner_ref, resid_ref, product = O.admm_solve(h, a, n, rho, sigma, rhs, x0, accuracy, most)
            x, inner, resid = s.solve(rhs, x0, accuracy, most)
            assert np.array_equal(s.apply(x0), product)
            assert (inner, resid) == (inner_ref, resid_ref)
            assert np.array_equal(x, ref)
    finally:
        s.close()
