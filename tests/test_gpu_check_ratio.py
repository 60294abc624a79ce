"""The check's stationarity residual, max |x - P(x - g)| / (1 + |x|), ranks rows by FP32 bounds and
divides in FP64 only where a row can be the largest: it must be the plain FP64 form's number, bit for
bit.

Matrix entries and x are small multiples of 2^-10, so Q x is exact in any order of summation, and every other
operation is the same single rounding here and there: no tolerance.  The objective is a sum of n
terms in another order: 4 n eps of the sum of their magnitudes bounds the difference.
"""
import ctypes

import numpy as np
import pytest
import torch

import boxqp

pytestmark = pytest.mark.gpu


def rows(n, kind, rng):
    """Tridiagonal CSR, x, c: ratios spread over magnitudes, all the same, or below FP32's range."""
    x = rng.integers(0, 1024, n) / 1024.0
    c = rng.integers(-2048, 2048, n) / 1024.0 * 2.0 ** rng.integers(-30, 1, n)
    if kind == 'equal':
        x, c = np.full(n, 0.5), np.full(n, -0.75)
    if kind == 'tiny':
        x = np.zeros(n)
        c = -rng.uniform(0.5, 1.0, n) * 2.0 ** rng.integers(-1000, -55, n).astype(float)
    if kind == 'near':  # neighbours within FP32 rounding of each other
        x = np.full(n, 0.25)
        c = -0.125 - rng.integers(0, 64, n) * 2.0 ** -50
    i = np.arange(n)
    row = np.concatenate([i[1:], i, i[:-1]])
    col = np.concatenate([i[:-1], i, i[1:]])
    val = np.concatenate([np.full(n - 1, -0.25), np.full(n, 1.0), np.full(n - 1, -0.25)])
    at = np.lexsort((col, row))
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(np.bincount(row, minlength=n))
    g = x.copy()
    g[1:] -= 0.25 * x[:-1]
    g[:-1] -= 0.25 * x[1:]
    return rowptr, col[at].astype(np.int32), val[at], x, c, g


@pytest.mark.parametrize('kind', ['spread', 'equal', 'tiny', 'near'])
@pytest.mark.parametrize('n', [1, 31, 33, 513, 608 * 512, 608 * 512 + 1, 700001])
def test_check_stationarity_is_the_fp64_quotient(n, kind):
    rng = np.random.default_rng(n)
    rowptr, col, val, x, c, gq = rows(n, kind, rng)
    lower, upper = np.zeros(n), np.full(n, 1.0)
    dev = [torch.from_numpy(a).cuda() for a in (rowptr, col, val, x, c, lower, upper)]
    st = boxqp.Stats()
    rc = boxqp.lib().bqp_check_device(n, *[d.data_ptr() for d in dev], 1e-6, 0.0, 0, ctypes.byref(st))
    assert rc == 0
    g = gq + c
    ratio = np.abs(x - np.maximum(lower, np.minimum(upper, x - g))) / (1.0 + np.abs(x))
    assert st.stationarity_residual == ratio.max()
    assert st.primal_residual == 0.0
    terms = np.concatenate([0.5 * x * gq, c * x])
    assert abs(st.objective - terms.sum()) <= 4 * n * 2.0 ** -52 * np.abs(terms).sum()
