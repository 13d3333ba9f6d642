"""Records of more than 64 bytes over thousands of partitions, against the
oracle: the launch shapes that only wide rows with many groups reach."""
import numpy as np
import pytest

from parity import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_words,nullable", [(False, False), (False, True), (True, False), (True, True)])
def test_wide_records_over_8192_partitions(two_words, nullable):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(5 + 2 * two_words + nullable)
    n = 4_200_000
    rows = np.arange(n, dtype=np.int64)
    keys = [cb.Column.from_numpy(rng.permutation(rows) * 1_000_003)]  # every row its own group
    if two_words:
        keys.append(cb.Column.from_numpy((rows % 9).astype(np.int32)))
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n), rng.random(n) > 0.1 if nullable else None),
             [agg.sum(), agg.min(), agg.max()]) for _ in range(8)]
    gb, *_ = run_both(keys, reqs)
    st = gb.stats()
    assert st["mode"] == 2
    # slot: key words, a row count, a null count per nullable column, 24 accumulators; an odd
    # number of 8-byte (two-word keys: 16-byte) units.  Beyond 4096 partitions at 78% fill of
    # ~220 KB of slots and tags there are 8192.
    unit = 16 if two_words else 8
    units = -(-(8 * (1 + two_words) + 4 + 4 * 8 * nullable + 24 * 8 + 7) // unit)
    slot = (units | 1) * unit
    assert st["est_groups"] > 4096 * 0.78 * (220 * 1024 // (slot + 4))


@pytest.mark.parametrize("columns,groups", [(8, 400_000), (8, 1_500_000), (6, 1_300_000), (4, 2_500_000)])
def test_wide_records_over_hundreds_to_thousands_of_partitions(columns, groups):
    """Both sides of the line between two CTAs per SM and one."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(columns + groups)
    n = 1_500_007
    key = rng.integers(0, groups, n) * 2_654_435_761
    reqs = [(cb.Column.from_numpy(rng.integers(-10**9, 10**9, n), rng.random(n) > 0.2 if c % 2 else None),
             [agg.sum(), agg.min(), agg.max()]) for c in range(columns)]
    gb, *_ = run_both([cb.Column.from_numpy(key)], reqs, tuning={"force_mode": 2})
    assert gb.stats()["mode"] == 2


@pytest.mark.parametrize("two_words", [False, True])
@pytest.mark.parametrize("nullable", [False, True])
@pytest.mark.parametrize("hot", [0, 3, 900])
def test_wide_records_with_hot_keys(hot, nullable, two_words):
    """96-byte records are read four words at a time: without hot keys, and with keys whose rows are folded per
    warp first.  The columns' types put their words at every place of a record."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(hot + nullable)
    n = 150_001
    key = rng.integers(0, 30_000, n)
    if hot:
        key = np.where(rng.random(n) < 0.7, rng.integers(0, hot, n), key)
    keys = [cb.Column.from_numpy(key * 1_000_003)]
    if two_words:
        keys.append(cb.Column.from_numpy((key % 11).astype(np.int32)))
    kinds = [np.int64, np.float64, np.uint64, np.int64, np.float64, np.int64, np.float64, np.int32]
    if not (nullable or two_words):
        kinds[-1] = np.int64
    reqs = [(cb.Column.from_numpy(rng.integers(0, 1000, n).astype(k), rng.random(n) > 0.1 * (j % 3) if nullable else None),
             [agg.sum(), agg.min(), agg.max(), agg.count()][j % 2:]) for j, k in enumerate(kinds)]
    gb, *_ = run_both(keys, reqs, tuning={"force_mode": 2})
    assert gb.stats()["mode"] == 2
