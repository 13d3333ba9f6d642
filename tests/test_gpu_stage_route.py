"""A few thousand groups: the shared stage keeps those that the whole of shared
memory holds, from 1M rows on; equal results on both sides of each line."""
import numpy as np
import pytest

from parity import run_both

pytestmark = pytest.mark.gpu


def _requests(plan, rng, n):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg

    def f32():
        return cb.Column.from_numpy(rng.lognormal(size=n).astype(np.float32))

    return {"2 sums": lambda: [(f32(), [agg.sum()]) for _ in range(2)],
            "6 sums": lambda: [(f32(), [agg.sum()]) for _ in range(6)],
            "sums, argmax": lambda: [(f32(), [agg.sum(), agg.argmax()]) for _ in range(2)],
            "var": lambda: [(cb.Column.from_numpy(rng.normal(size=n), rng.random(n) > 0.1), [agg.variance(1)])]}[plan]()


@pytest.mark.parametrize("plan,n,groups,mode", [
    ("2 sums", 1_100_000, 4_000, 1), ("2 sums", 1_100_000, 4_600, 2), ("2 sums", 600_000, 4_000, 0),
    ("6 sums", 2_000_000, 2_400, 1), ("6 sums", 2_000_000, 2_800, 2),
    ("sums, argmax", 1_100_000, 1_900, 1), ("sums, argmax", 1_100_000, 2_600, 0),
    ("var", 1_100_000, 3_300, 1), ("var", 1_100_000, 4_200, 0)])
def test_stage_route(plan, n, groups, mode):
    import cudf_b200 as cb
    rng = np.random.default_rng(n + groups)
    key = rng.integers(0, groups, n) * 1_000_003
    key[:groups] = np.arange(groups) * 1_000_003
    gb, uk, *_ = run_both([cb.Column.from_numpy(key)], _requests(plan, rng, n))
    assert uk.num_rows() == groups
    assert gb.stats()["mode"] == mode


@pytest.mark.parametrize("plan", ["2 sums", "sums, argmax", "var"])
@pytest.mark.parametrize("groups,hint,redone", [(2_000, 2_000, False), (40_000, 2_000, True), (300_000, 20_000, True)])
def test_a_caller_s_estimate_far_too_low_is_dropped(plan, groups, hint, redone):
    """A right estimate holds; one that the tables overflow on is replaced by the count of every row."""
    import cudf_b200 as cb
    rng = np.random.default_rng(groups)
    n = 1_100_000
    key = rng.integers(0, groups, n) * 1_000_003
    gb, uk, *_ = run_both([cb.Column.from_numpy(key)], _requests(plan, rng, n), tuning={"groups_hint": hint})
    st = gb.stats()
    assert st["retries"] == int(redone)
    assert abs(st["est_groups"] - uk.num_rows()) < 0.08 * uk.num_rows()


@pytest.mark.parametrize("plan", ["2 sums", "sums, argmax"])
@pytest.mark.parametrize("key", ["i64", "two words"])
def test_generic_stage_tables_of_any_size(plan, key):
    """The generic kernel's table need not be a power of two: keys at its ends, and more groups than it holds."""
    import cudf_b200 as cb
    rng = np.random.default_rng(3)
    n = 1_100_000
    k = rng.integers(0, 1_800, n)
    keys = [cb.Column.from_numpy(k * 1_000_003)] + ([cb.Column.from_numpy((k % 3).astype(np.int32))] if key == "two words" else [])
    for hint in (1_500, 700):
        run_both(keys, _requests(plan, rng, n), tuning={"force_mode": 1, "groups_hint": hint, "block": 256})
