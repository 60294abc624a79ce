"""Sliced instances with a dense window: 256 rows of 60 to 127 entries in an instance of short rows, more
entries than the admission and the residual pass stage in shared memory (1.2 times an average window;
5,120), so that both read them from global memory.  The dense window is the first, one inside, or the
last and partial one.  Bars as in the tests of the other sliced sizes: the bit-exact engine equals the
oracle bit for bit, the FP64 objective agrees to 1e-10, the mixed answer is verified by the oracle at 1e-6
and its objective agrees to 1e-7."""
import numpy as np
import pytest

import boxqp
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def problem(n, first, rows):
    """Lower triplets: about three couplings a row, and 60 to 100 more for each of `rows` rows from
    `first` on."""
    rng = np.random.default_rng(n + first)
    dense = np.arange(first, first + rows)
    others = np.setdiff1d(np.arange(n), dense)
    extra = rng.integers(60, 101, rows)
    a = np.concatenate([rng.integers(0, n, 3 * n)] + [np.full(k, r) for r, k in zip(dense, extra)])
    b = np.concatenate([rng.integers(0, n, 3 * n)] + [rng.choice(others, k, replace=False) for k in extra])
    key = np.unique(np.maximum(a, b) * n + np.minimum(a, b))
    row, col = key // n, key % n
    row, col = row[row != col], col[row != col]
    w = rng.uniform(0.1, 1.0, len(row))
    diag = rng.uniform(0.5, 2.0, n)
    np.add.at(diag, row, w)
    np.add.at(diag, col, w)
    i = np.arange(n)
    return (np.concatenate([row, i]), np.concatenate([col, i]), np.concatenate([-w, diag]), rng.uniform(-2, 2, n),
            np.zeros(n), rng.uniform(0.5, 2.0, n))


@pytest.mark.parametrize('n,first,rows', [(8192, 0, 256), (8192, 512, 256), (8292, 8192, 100)])
def test_a_dense_window(n, first, rows):
    args = problem(n, first, rows)
    rowptr, col, val = boxqp.csr_from_lower(n, *args[:3])[:3]
    lengths = np.diff(rowptr)
    average = rowptr[-1] / n
    window = int(lengths[first:first + rows].sum())
    assert lengths.max() <= 127 and average < 20 and window > max(5120, 1.2 * 256 * average + 256)
    status, x_ref, st_ref = O.solve_box(*args, tol=1e-8, threads=1)
    eng = boxqp.Engine(0)
    try:
        x, st = eng.solve(rowptr, col, val, *args[3:], boxqp.options_struct(1e-8, 60.0, 200000, 'fp64_exact'))
        assert boxqp.STATUS_NAMES[st.status] == status and st.iterations == st_ref['iterations']
        assert np.array_equal(x, x_ref)
        x, st = eng.solve(rowptr, col, val, *args[3:], boxqp.options_struct(1e-8, 60.0, 200000, 'fp64'))
        assert boxqp.STATUS_NAMES[st.status] == status
        assert abs(st.objective - st_ref['objective']) <= 1e-10 * (1 + abs(st_ref['objective']))
        x, st = eng.solve(rowptr, col, val, *args[3:], boxqp.options_struct(1e-6, 60.0, 200000, 'mixed'))
        assert boxqp.STATUS_NAMES[st.status] == 'optimal' and st.polish_rounds > 0
        assert O.check(*args, x, tol=1e-6)['verified'] == 1.0
        assert abs(st.objective - st_ref['objective']) <= 1e-7 * (1 + abs(st_ref['objective']))
    finally:
        eng.close()
