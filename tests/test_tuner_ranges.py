"""The autotuner's search ranges hold no two values that select the same code."""
from horsepower_gb300 import autotune as T


def test_ranges_hold_distinct_values():
    assert T.KNOBS["radix_pass"][1] == [0, 2]  # 1 is an alias of 2
    for name, (_, values) in T.KNOBS.items():
        assert len(set(values)) == len(values) > 1, name
