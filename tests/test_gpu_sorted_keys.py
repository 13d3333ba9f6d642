"""Keys in sorted order, and hot keys: rows of one key meet in a warp, and are
folded there before they update a table."""
import numpy as np
import pytest

from parity import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_words", [False, True])
@pytest.mark.parametrize("n,groups,mode", [(70_001, 40, None), (200_000, 900, 1), (900_000, 2_900, 1), (1_100_000, 2_000, 1),
                                           (1_500_000, 20_000, 2), (1_500_000, 400_000, 2), (8_400_000, 30, 1)])
def test_sorted_keys(n, groups, mode, two_words):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(n + groups)
    key = np.sort(rng.integers(0, groups, n)) - 3  # an all-ones key among them
    keys = [cb.Column.from_numpy(key)] + ([cb.Column.from_numpy((key % 2).astype(np.int32), rng.random(n) > 0.001)] if two_words else [])
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n), rng.random(n) > 0.1), [agg.sum(), agg.min(), agg.count()]),
            (cb.Column.from_numpy(rng.normal(size=n).astype(np.float32)), [agg.sum(), agg.max()])]
    gb, *_ = run_both(keys, reqs, include_null_keys=two_words)
    if mode is not None and not two_words:
        assert gb.stats()["mode"] == mode


@pytest.mark.parametrize("n,groups,mode", [(880_000, 2_900, 1), (1_500_000, 60_000, 2), (6_000_000, 16_000, 2)])
@pytest.mark.parametrize("share", [0.06, 0.7])
def test_a_hot_key_among_many(n, groups, mode, share):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(n)
    key = rng.integers(0, groups, n) * 1_000_003
    key[rng.random(n) < share] = 77
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n)), [agg.sum(), agg.max()]),
            (cb.Column.from_numpy(rng.normal(size=n), rng.random(n) > 0.1), [agg.sum(), agg.min()])]
    gb, *_ = run_both([cb.Column.from_numpy(key)], reqs)
    if n > 1_000_000 or share > 0.1:
        assert gb.stats()["mode"] == mode


@pytest.mark.parametrize("n,groups", [(300_000, 30), (1_500_000, 65), (1_500_000, 250)])
def test_sorted_keys_with_many_accumulators(n, groups):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(groups)
    keys = [cb.Column.from_numpy(np.sort(rng.integers(0, groups, n)))]
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n) if i % 2 else rng.normal(size=n)), [agg.sum(), agg.min(), agg.max()])
            for i in range(7)]
    gb, *_ = run_both(keys, reqs)
    assert gb.stats()["mode"] == 1


@pytest.mark.parametrize("n,groups", [(1_200_000, 8_000), (2_000_000, 16_000), (7_000_001, 16_000)])
def test_long_tailed_keys_in_few_partitions(n, groups):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(n + groups)
    top = (groups + 1.0) ** -0.1
    key = np.minimum(((1 - rng.random(n) * (1 - top)) ** -10.0 - 1).astype(np.int64), groups - 1) * 1_000_003
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n)), [agg.sum(), agg.min()]),
            (cb.Column.from_numpy(rng.normal(size=n), rng.random(n) > 0.1), [agg.sum(), agg.max()])]
    gb, *_ = run_both([cb.Column.from_numpy(key)], reqs)
    assert gb.stats()["mode"] == 2
