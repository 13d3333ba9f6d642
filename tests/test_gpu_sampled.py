"""Few groups on large inputs, sized from a sample of the rows: what happens to
groups that the sample does not see."""
import numpy as np
import pytest

from parity import run_both
from test_gpu_record import _fmix64

pytestmark = pytest.mark.gpu

CHUNKS = 4096  # sampled runs of 128 rows


def _run_starts(n):
    s = np.arange(CHUNKS, dtype=np.int64)
    stratum = n // CHUNKS
    return s * stratum + (_fmix64(s) % np.uint64(stratum - 128)).astype(np.int64)


def _reqs(rng, n):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    return [(cb.Column.from_numpy(rng.integers(-10**6, 10**6, n)), [agg.sum(), agg.min(), agg.max(), agg.count()]),
            (cb.Column.from_numpy(rng.normal(size=n), rng.random(n) > 0.1), [agg.sum(), agg.mean()])]


def test_more_missed_rows_than_the_list_holds_redo_the_call():
    """70,000 one-row groups on unsampled rows: the call ends with the count of every row, not the sample's."""
    import cudf_b200 as cb
    n, hidden = (8 << 20) + 77, 70_000
    rng = np.random.default_rng(7)
    key = rng.integers(0, 5, n)
    seen = np.zeros(n, bool)
    seen[(_run_starts(n)[:, None] + np.arange(128)).ravel()] = True
    key[rng.permutation(np.nonzero(~seen)[0])[:hidden]] = 1000 + np.arange(hidden)
    gb, uk, *_ = run_both([cb.Column.from_numpy(key)], _reqs(rng, n))
    assert uk.num_rows() == 5 + hidden
    assert abs(gb.stats()["est_groups"] - (5 + hidden)) < 0.1 * hidden


@pytest.mark.parametrize("product", [False, True])
def test_a_stretch_of_missed_groups_costs_no_second_pass(product):
    """Sorted keys with one stretch of one-row groups between two sampled runs (about 3,900 rows of 8M): the call
    stays with the sample's five groups, in the shared stage and in the generic kernel (PRODUCT)."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    n = (8 << 20) + 77
    rng = np.random.default_rng(8)
    key = np.sort(rng.integers(0, 5, n))
    start = _run_starts(n)
    gap = np.diff(start) - 128
    i = int(np.argmax(gap))
    a, hidden = int(start[i]) + 128, int(gap[i])
    assert hidden > 3000
    key[a:a + hidden] = 1000 + rng.permutation(hidden)
    reqs = _reqs(rng, n)
    if product:
        reqs = [(cb.Column.from_numpy(rng.integers(-1, 2, n)), [agg.product(), agg.sum()])]
    gb, uk, *_ = run_both([cb.Column.from_numpy(key)], reqs)
    assert uk.num_rows() == 5 + hidden
    assert gb.stats()["est_groups"] < 10 and gb.stats()["mode"] == 1
