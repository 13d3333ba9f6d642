"""VARIANCE/STD with many groups: the partitioned path only where it pays, equal
results on both sides of the line."""
import numpy as np
import pytest

from parity import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,groups,accumulators,mode", [
    (1_100_000, 50_000, 1, 0), (1_100_000, 50_000, 4, 0), (2_100_000, 5_000, 4, 0), (2_100_000, 100_000, 4, 2),
    (2_100_000, 900_000, 4, 0), (3_600_000, 1_500_000, 4, 2), (4_000_000, 100_000, 1, 0), (6_100_000, 300_000, 1, 2),
    (6_100_000, 2_500_000, 1, 0)])
def test_var_route(n, groups, accumulators, mode):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(n + groups)
    keys = [cb.Column.from_numpy(rng.integers(0, groups, n) * 1_000_003)]
    reqs = [(cb.Column.from_numpy(rng.normal(size=n), rng.random(n) > 0.1), [agg.variance(1), agg.std(1)])]
    if accumulators == 4:
        reqs.append((cb.Column.from_numpy(rng.integers(-1000, 1000, n)), [agg.sum(), agg.min(), agg.max()]))
    gb, *_ = run_both(keys, reqs)
    assert gb.stats()["mode"] == mode
