"""The box iteration's division by L, known in advance: the quotient that IEEE division gives, bit for bit.

One step from x = w = 0 with an empty product is 0 - c / L, which numpy forms with the same two
rounded operations.  Divisors lie inside, at and outside the range for which the short form holds
(2^-100 .. 2^100), dividends over all exponents, at the edges of theirs (2^-823 .. 2^824), subnormal, zero."""
import numpy as np
import pytest

import boxqp

pytestmark = pytest.mark.gpu

EDGE = 2.0 ** 100
DIVISORS = [1.0, 3.0, 7.0 / 3.0, np.nextafter(2.0, 0.0), np.nextafter(1.0, 2.0), 1.3e5, EDGE, np.nextafter(EDGE, 0.0),
            np.nextafter(EDGE, np.inf), 1.0 / EDGE, np.nextafter(1.0 / EDGE, 0.0), np.nextafter(1.0 / EDGE, 1.0), 3.1 * EDGE,
            0.3 / EDGE, 1.7e300, 1.7e-300, 1.7e308, 2.3e-308, 4e-320]


def dividends(n, rng):
    bits = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    exponent = rng.integers(0, 2047, n, dtype=np.uint64)
    exponent[:n // 4] = rng.choice(np.array([0, 1, 198, 199, 200, 201, 1845, 1846, 1847, 1848, 2046], np.uint64), n // 4)
    exponent[n // 4:n // 2] = rng.integers(1000, 1046, n // 2 - n // 4, dtype=np.uint64)
    bits[:n // 8] = rng.choice(np.array([0, 1, (1 << 52) - 1, 1 << 51], np.uint64), n // 8)
    sign = rng.integers(0, 2, n, dtype=np.uint64)
    return (sign << np.uint64(63) | exponent << np.uint64(52) | bits).view(np.float64)


@pytest.mark.parametrize('sliced', [True, False])
def test_division_by_a_known_divisor(sliced):
    n = 200003
    rng = np.random.default_rng(11)
    c = dividends(n, rng)
    c[:3] = [0.0, -0.0, 5e-324]
    # a zero matrix: one entry a row, or (a row too long for a lane: the CSR kernel) 200 in the first
    long = np.arange(200) if not sliced else np.arange(1)
    rowptr = np.concatenate([[0], np.arange(len(long), len(long) + n)]).astype(np.int32)
    col = np.concatenate([long, np.arange(1, n)]).astype(np.int32)
    rng.shuffle(c)
    free = np.full(n, 1.7976931348623157e308)
    for L in DIVISORS:
        box = boxqp.make_cuda_box(rowptr, col, np.zeros(len(col)), c, -free, free, L)
        box.step(0.0)
        with np.errstate(over='ignore', under='ignore'):
            expected = np.clip(0.0 - (0.0 + c) / L, -free, free)
        got = box.primal()
        assert np.array_equal(got.view(np.uint64), expected.view(np.uint64)), (L, np.flatnonzero(got != expected)[:5])
