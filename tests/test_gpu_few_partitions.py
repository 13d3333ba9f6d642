"""Partitions fewer than the SMs, cut into pieces that merge through the global
table: even and skewed rows, with and without a heavy key."""
import numpy as np
import pytest

from parity import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [70_001, 1_100_003, 2_000_000])
@pytest.mark.parametrize("groups", [1, 300, 5_000, 18_000])
@pytest.mark.parametrize("hot", [0.0, 0.6])
def test_few_partitions_in_pieces(n, groups, hot):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(groups + n)
    key = (rng.random(n) ** (3 if groups == 300 else 1) * groups).astype(np.int64) * 1_000_003
    key[rng.random(n) < hot] = -1  # the all-ones key word
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n), rng.random(n) > 0.1), [agg.sum(), agg.min(), agg.count()]),
            (cb.Column.from_numpy(rng.normal(size=n).astype(np.float32)), [agg.sum(), agg.max()])]
    gb, *_ = run_both([cb.Column.from_numpy(key)], reqs, tuning={"force_mode": 2})
    assert gb.stats()["mode"] == 2
