"""Instances with a row too long for a lane keep the CSR: the structure that the engine picks for their
FP64 steps must not be slower than the block-staged one it had before there were sliced rows.

The bound is the resolution of the step timer on these sizes (steps of 20 to 400 us, back to back): the
wrong structures are 1.5 to 3 times slower; 1.2 is allowed, the best of three timings on each side."""
import numpy as np
import pytest

import boxqp
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def problem(n, epv, hub):
    """Random couplings, and row 0 coupled to `hub` others (lower triplets)."""
    rng = np.random.default_rng(n + hub)
    a = np.concatenate([rng.integers(0, n, epv * n), np.zeros(hub, np.int64)])
    b = np.concatenate([rng.integers(0, n, epv * n), rng.choice(np.arange(1, n), hub, replace=False)])
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


@pytest.mark.parametrize('n,epv,hub', [(16384, 1, 500), (16384, 5, 4000), (100000, 3, 40000)])
def test_structure_of_fp64_steps_on_long_rows(n, epv, hub):
    p = problem(n, epv, hub)
    csr = boxqp.csr_from_lower(n, *p[:3])
    eng, best = boxqp.Engine(0), {}
    try:
        for variant in (-1, 0):
            o = boxqp.options_struct(1e-6, 20.0, 50, 'fp64', kernel_variant=variant)
            ident = eng.submit(*csr[:3], *p[3:], o)
            eng.wait(ident)
            x, st = eng.fetch(ident, n)
            assert abs(st.objective - O.check(*p, x)['objective']) <= 1e-10 * (1 + abs(st.objective))
            best[variant] = min(eng.profile_step(ident, 30)[0] for _ in range(3))
            eng.release(ident)
    finally:
        eng.close()
    assert best[-1] <= 1.2 * best[0], best
