"""The tuning sweep's choice (no GPU): a setting that leads the default by more
than two sweeps differ, in total and without trailing it anywhere, else the
default."""
from tetragpu_gb300 import tune


def test_select():
    base = [9.0, 1.0, 3.0, 5.0]
    buckets = [1, 2, 3]
    pick = lambda **others: tune.select({"default": base, **others}, buckets)  # noqa: E731
    assert pick() == "default"
    assert pick(a=[1.0, 1.0, 2.99, 4.98]) == "default"            # a lead of 0.3 %
    assert pick(a=[9.0, 0.95, 2.9, 4.9]) == "a"
    assert pick(a=[9.0, 1.02, 2.8, 4.7]) == "default"             # ahead in total, behind in a bucket
    assert pick(a=[9.0, 0.95, 2.9, 4.9], b=[9.0, 0.94, 2.8, 4.9]) == "b"
    assert tune.select({"a": [2.0, 1.0], "b": [1.0, 2.0]}, [0]) == "b"   # a sweep without the default
