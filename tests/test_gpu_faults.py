"""Allocations of the engine that fail (on the host, injected: no device call is made for them): what
the failure ends, and that the engine goes on with the right answers.

Answers are compared bit for bit with those of an engine in which nothing failed."""
import numpy as np
import pytest

import boxqp

pytestmark = pytest.mark.gpu


def problem(seed, n):
    p = boxqp.planted('graph10k', seed=seed, n=n)
    return tuple(p[k] for k in ('rowptr', 'col', 'val', 'c', 'lower', 'upper'))


@pytest.fixture()
def engine():
    eng = boxqp.Engine(0)
    yield eng
    eng.close()


@pytest.fixture(scope='module')
def reference():
    """x of a solve in an engine of its own, by seed, size and precision."""
    eng, known = boxqp.Engine(0), {}

    def solve(seed, n, precision):
        if (seed, n, precision) not in known:
            known[seed, n, precision] = eng.solve(*problem(seed, n), options(precision))[0]
        return known[seed, n, precision]
    yield solve
    eng.close()


def options(precision):
    return boxqp.options_struct(1e-7, 20.0, 200000, precision)


def done(engine, ident, n):
    assert engine.wait(ident, 60.0)
    x, st = engine.fetch(ident, n)
    assert boxqp.STATUS_NAMES[st.status] == 'optimal'
    return x


@pytest.mark.parametrize('precision', ['fp64', 'fp64_exact', 'mixed'])
def test_a_launch_that_cannot_be_set_up_leaves_nothing_running(engine, reference, precision):
    """Its solves' records were armed on the device; the next launch, of another solve, must not wait for
    them, and a re-run of them must still give their answer."""
    engine.inject_oom('launch')
    failed = engine.submit(*problem(70, 3000), options(precision))
    with pytest.raises(boxqp.EngineError, match='injected'):
        engine.wait(failed, 60.0)
    other = engine.submit(*problem(71, 5000), options(precision))
    assert np.array_equal(done(engine, other, 5000), reference(71, 5000, precision))
    engine.resolve([failed])
    assert np.array_equal(done(engine, failed, 3000), reference(70, 3000, precision))
    # a re-run that fails, then the release of the solve whose record it left armed
    engine.inject_oom('launch')
    engine.resolve([failed])
    with pytest.raises(boxqp.EngineError, match='injected'):
        engine.wait(failed, 60.0)
    engine.release(failed)
    engine.resolve([other])
    assert np.array_equal(done(engine, other, 5000), reference(71, 5000, precision))
    engine.release(other)
    # its slot is taken again
    again = engine.submit(*problem(70, 3000), options(precision))
    assert np.array_equal(done(engine, again, 3000), reference(70, 3000, precision))


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('n', [3000, 150000])
def test_no_record_for_the_gate(engine, reference, n, precision):
    """The solve ends before any of its memory is in use on a stream; those around it keep their answers
    (sizes of the staged upload and of the copied one)."""
    before = engine.submit(*problem(72, n), options(precision))
    done(engine, before, n)
    engine.inject_oom('gate_record')
    failed = engine.submit(*problem(73, n), options(precision))
    after = engine.submit(*problem(74, n), options(precision))
    with pytest.raises(boxqp.EngineError, match='convexity gate'):
        engine.wait(failed, 60.0)
    assert np.array_equal(done(engine, after, n), reference(74, n, precision))
    engine.resolve([before])
    assert np.array_equal(done(engine, before, n), reference(72, n, precision))
    held = engine.load()['resident_bytes']
    engine.release(failed)
    assert engine.load()['resident_bytes'] == held


def test_no_buffer_for_the_upload(engine, reference):
    """A solve of sliced rows goes on over its CSR: the exact engine with the same bits, the FP64 engine
    with those of the CSR structure it names (two lanes a row), the mixed one verified.  A solve that
    runs over its CSR anyway and needs the buffer ends out of memory, as it always did."""
    n = 30000
    assert engine.load()['resident_bytes'] == 0
    for precision in ('fp64_exact', 'fp64', 'mixed'):
        engine.inject_oom('upload_buffer')
        ident = engine.submit(*problem(75, n), options(precision))
        x = done(engine, ident, n)
        ref = reference(75, n, precision)
        if precision == 'fp64_exact':
            assert np.array_equal(x, ref)
        elif precision == 'fp64':
            named = boxqp.options_struct(1e-7, 20.0, 200000, precision, kernel_variant=2)
            assert np.array_equal(x, engine.solve(*problem(75, n), named)[0])
        else:
            st = engine.fetch(ident, n)[1]
            fstar = boxqp.planted('graph10k', seed=75, n=n)['fstar']
            assert st.verified and abs(st.objective - fstar) <= 1e-7 * (1 + abs(fstar))
        engine.resolve([ident])
        assert np.array_equal(done(engine, ident, n), x)
        engine.release(ident)
    csr = boxqp.options_struct(1e-7, 20.0, 200000, 'mixed', kernel_variant=8)
    engine.inject_oom('upload_buffer')
    ident = engine.submit(*problem(75, n), csr)
    with pytest.raises(boxqp.EngineError, match='upload buffer'):
        engine.wait(ident, 60.0)
    engine.release(ident)
    assert np.array_equal(engine.solve(*problem(75, n), options('mixed'))[0], reference(75, n, 'mixed'))
    assert engine.load()['resident_bytes'] == 0
