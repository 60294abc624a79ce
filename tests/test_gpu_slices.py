"""Sliced rows (rows ordered by length within windows of 256, 32 to a warp, entries interleaved):
the sizes where the layout can go wrong, against the CPU oracle.

The bit-exact engine sums every row in column order whatever the layout, so its iterates, iteration
counts and primal must be the oracle's bit for bit; the FP64 engine runs the same iteration with
fused products, so its objective agrees to rounding accumulated over the run (1e-10 relative).
"""
import numpy as np
import pytest

import boxqp
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def engine():
    eng = boxqp.Engine(0)
    yield eng
    eng.close()


def problem(n, rng, hub=0, empty=False, epv=3):
    """Random diagonally dominant Hessian (lower triplets); `hub`: row 0 couples to that many others;
    `empty`: every fifth row has no entry at all."""
    dead = np.zeros(n, bool)
    if empty:
        dead[4::5] = True
    live = np.flatnonzero(~dead)
    pairs = set()
    for _ in range(epv * len(live)):
        a, b = rng.choice(live, 2)
        if a != b:
            pairs.add((max(a, b), min(a, b)))
    for j in live[1:hub + 1]:
        pairs.add((j, live[0]))
    row = np.array([p[0] for p in sorted(pairs)], np.int64)
    col = np.array([p[1] for p in sorted(pairs)], np.int64)
    w = rng.uniform(0.1, 1.0, len(row))
    diag = rng.uniform(0.5, 2.0, n)
    np.add.at(diag, row, w)
    np.add.at(diag, col, w)
    keep = live
    hrow, hcol = np.concatenate([row, keep]), np.concatenate([col, keep])
    hval = np.concatenate([-w, diag[keep]])
    return hrow, hcol, hval, rng.uniform(-2, 2, n), np.zeros(n), rng.uniform(0.5, 2.0, n)


def rows_of(n, hrow, hcol, hval):
    rowptr, col, val = boxqp.csr_from_lower(n, hrow, hcol, hval)
    return rowptr, col, val, int(np.max(np.diff(rowptr)))


CASES = [(1, 0, False), (31, 0, False), (32, 0, False), (33, 0, True), (255, 0, False), (256, 0, True), (257, 0, False),
         (513, 126, False),   # the longest row a sliced instance may have (127 entries)
         (514, 127, False),   # one more entry: the CSR kernels
         (4099, 40, True)]


@pytest.mark.parametrize('n,hub,empty', CASES)
def test_sliced_rows_match_the_oracle(engine, n, hub, empty):
    rng = np.random.default_rng(100 * n + hub)
    args = problem(n, rng, hub, empty)
    rowptr, col, val, longest = rows_of(n, *args[:3])
    if hub:
        assert longest >= hub + 1
    status, x_ref, st_ref = O.solve_box(*args, tol=1e-8, threads=1)
    o = boxqp.options_struct(1e-8, 60.0, 200000, 'fp64_exact')
    x, st = engine.solve(rowptr, col, val, *args[3:], o)
    assert boxqp.STATUS_NAMES[st.status] == status
    assert st.iterations == st_ref['iterations']
    assert np.array_equal(x, x_ref)
    o = boxqp.options_struct(1e-8, 60.0, 200000, 'fp64')
    x, st = engine.solve(rowptr, col, val, *args[3:], o)
    assert boxqp.STATUS_NAMES[st.status] == status
    assert abs(st.objective - st_ref['objective']) <= 1e-10 * (1 + abs(st_ref['objective']))
    assert O.check(*args, x, tol=1e-8)['verified'] == 1.0


def test_resolve_and_batch_of_sliced_solves_keep_their_bits(engine):
    """Solo, re-run and in a batch with instances of other sizes (small and large pieces)."""
    rng = np.random.default_rng(7)
    insts = [problem(n, rng) for n in (257, 2049)] + [problem(70001, rng, epv=2)]
    o = boxqp.options_struct(1e-6, 60.0, 200000, 'fp64')
    csr = [rows_of(len(p[3]), *p[:3])[:3] for p in insts]
    solo = [engine.solve(*c, *p[3:], o)[0] for c, p in zip(csr, insts)]
    ids = [engine.submit(*c, *p[3:], o) for c, p in zip(csr, insts)]
    for again in range(2):
        for i, p, ref in zip(ids, insts, solo):
            engine.wait(i)
            assert np.array_equal(engine.fetch(i, len(p[3]))[0], ref)
        if not again:
            engine.resolve(ids)
    for i in ids:
        engine.release(i)


@pytest.mark.parametrize('n,hub,empty', CASES)
def test_sliced_mixed_engine_is_verified(engine, n, hub, empty):
    """The mixed engine (FP32 steps, FP64 checks and polish on the same layout): verified at 1e-6 by the
    oracle, the objective within 1e-7 of the oracle's (the bar of the engine's parity tests)."""
    rng = np.random.default_rng(100 * n + hub)
    args = problem(n, rng, hub, empty)
    rowptr, col, val, _ = rows_of(n, *args[:3])
    _, _, st_ref = O.solve_box(*args, tol=1e-9, threads=1)
    o = boxqp.options_struct(1e-6, 60.0, 200000, 'mixed')
    x, st = engine.solve(rowptr, col, val, *args[3:], o)
    assert boxqp.STATUS_NAMES[st.status] == 'optimal'
    assert O.check(*args, x, tol=1e-6)['verified'] == 1.0
    assert abs(st.objective - st_ref['objective']) <= 1e-7 * (1 + abs(st_ref['objective']))


@pytest.mark.parametrize('n', [2, 256, 513, 1025, 70001])
def test_sliced_chains_keep_the_row_order(engine, n):
    """Tridiagonal rows (the end rows are shorter, so the order within the first and last window is not
    the row order): the polish's chains must follow the rows, or CG needs tens of iterations."""
    inst = boxqp.planted('tridiagonal', n=n, lower_triplets=True)
    o = boxqp.options_struct(1e-6, 60.0, 200000, 'mixed')
    x, st = engine.solve(inst['rowptr'], inst['col'], inst['val'], inst['c'], inst['lower'], inst['upper'], o)
    assert boxqp.STATUS_NAMES[st.status] == 'optimal'
    assert st.polish_iterations <= 15
    args = (inst['hrow'], inst['hcol'], inst['hval'], inst['c'], inst['lower'], inst['upper'])
    assert O.check(*args, x, tol=1e-6)['verified'] == 1.0
