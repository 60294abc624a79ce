"""The autotuner's choice per class (CPU): no timing noise decides between variants that share a kernel,
because the variant also names the order of the mixed engine's FP32 sums."""
from boxqp import autotune


def test_a_committed_variant_stays_within_the_noise():
    times = {'-1': 0.01000, '0': 0.00998, '64': 0.01002, '1': 0.01001, '2': 0.00999, '4': 0.02}
    for committed in (-1, 0, 64, 1, 2):
        assert autotune.choose(times, committed) == committed
    assert autotune.choose(times, 4) == 0          # another kernel, twice as slow
    assert autotune.choose(times, None) == 0       # no committed choice: the fastest
    assert autotune.choose(times, 8) == 0          # one that was not timed


def test_every_class_of_the_committed_table_has_a_timed_variant():
    for e in autotune.load_table()['entries']:
        assert e['ms'][str(e['variant'])] <= (1 + autotune.KEEP) * min(e['ms'].values()), e
