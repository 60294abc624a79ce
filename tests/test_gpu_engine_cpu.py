"""The engine thread leaves its core to others while a launch of milliseconds runs: launches of about 1.8 ms
one after the other take less than 0.7 of a core (polling throughout takes all of it, naps about a
third)."""
import time

import pytest

import boxqp

pytestmark = pytest.mark.gpu


def test_cpu_share_of_a_stream_of_launches():
    p = boxqp.planted('graph10k', seed=1, n=10000)
    eng = boxqp.Engine(0)
    try:
        ident = eng.submit(*(p[k] for k in ('rowptr', 'col', 'val', 'c', 'lower', 'upper')),
                           boxqp.options_struct(1e-7, 60.0, 200000, 'fp64'))
        eng.wait(ident)
        cpu, wall, launches = time.process_time(), time.perf_counter(), 0
        while time.perf_counter() - wall < 1.0:
            eng.resolve([ident])
            eng.wait(ident)
            launches += 1
        share = (time.process_time() - cpu) / (time.perf_counter() - wall)
    finally:
        eng.close()
    assert launches > 10 and share < 0.7, (launches, share)
