"""Group counts at the partitioned path's capacity, against the oracle: 16384
partitions, and the global table beyond what they hold."""
import numpy as np
import pytest

from parity import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,columns,two_words,nullable,mode", [
    (6_000_000, 7, False, False, 2), (6_200_000, 6, True, False, 2), (5_600_000, 8, False, False, 2), (5_600_000, 8, False, True, 0)])
def test_groups_beyond_8192_partitions(n, columns, two_words, nullable, mode):
    """64-byte records and 240-byte slots: about 900 slots a table, so 6M groups need more than 8192 tables at 78%
    fill.  96-byte records with masks keep to 8192 partitions, and take the global table beyond them."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(n)
    rows = np.arange(n, dtype=np.int64)
    keys = [cb.Column.from_numpy(rng.permutation(rows) * 1_000_003)]
    if two_words:
        keys.append(cb.Column.from_numpy((rows % 5).astype(np.int32)))
    reqs = [(cb.Column.from_numpy(rng.integers(-1000, 1000, n) if c % 2 else rng.normal(size=n),
                                  rng.random(n) > 0.1 if nullable else None),
             [agg.sum(), agg.min(), agg.max(), agg.sum_of_squares()]) for c in range(columns)]
    gb, *_ = run_both(keys, reqs)
    assert gb.stats()["mode"] == mode


def test_float32_sums_keep_the_partitioned_path():
    """FLOAT32 sums are held in 64 bits, which widens the slots: 7.2M groups of eight such columns were beyond the
    tables that 32-bit sums had fitted."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(2)
    n = 7_200_000
    keys = [cb.Column.from_numpy(rng.permutation(np.arange(n, dtype=np.int64)) * 1_000_003)]
    reqs = [(cb.Column.from_numpy(rng.normal(size=n).astype(np.float32)), [agg.sum(), agg.min(), agg.sum_of_squares()])
            for _ in range(8)]
    gb, *_ = run_both(keys, reqs)
    assert gb.stats()["mode"] == 2
