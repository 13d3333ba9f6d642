"""The engine over a caller's device memory resource, at the edges of what the
hooks promise."""
import numpy as np
import pytest
import torch

from device_mr import DeviceResource, aggregate_with
from oracle import oracle as O
from parity import compare, gpu_pairs, host_cols

pytestmark = pytest.mark.gpu


def _check(keys, reqs, uk, res):
    torch.cuda.synchronize()
    o = O.groupby(host_cols(keys), [(host_cols([r.values])[0], [int(a.kind) for a in r.aggregations]) for r in reqs],
                  nthreads=8)
    compare(o, gpu_pairs(uk), [gpu_pairs(t) for t in res], [[int(a.kind) for a in r.aggregations] for r in reqs], None)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("two_words", [False, True])
@pytest.mark.parametrize("kinds", ["i32 f32", "f64 i64 i16", "f64 i64 f64 f32", "f64 i64 f64 i64 f32 i32 i8",
                                   "f64 i64 f64 i64 f64 i64 f64 i64"])
def test_blocks_aligned_to_16_bytes_are_enough(mode, two_words, kinds):
    """Records of every size, tables and results in blocks at 16 mod 32."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(len(kinds) + mode)
    n, groups = 200_003, 700 if mode == 1 else 40_000
    key = rng.integers(0, groups, n) * 1_000_003
    keys = [cb.Column.from_numpy(key)] + ([cb.Column.from_numpy((key % 7).astype(np.int32))] if two_words else [])
    dtype = {"i8": np.int8, "i16": np.int16, "i32": np.int32, "i64": np.int64, "f32": np.float32, "f64": np.float64}
    reqs = [cb.GroupByRequest(cb.Column.from_numpy((rng.integers(-100, 100, n)).astype(dtype[k]),
                                                   rng.random(n) > 0.1 if j == 0 else None),
                              [agg.sum(), agg.min(), agg.max(), agg.count()]) for j, k in enumerate(kinds.split())]
    gb = cb.GroupBy(cb.Table(keys)).set_tuning(force_mode=mode)
    mr = DeviceResource(shift=16)
    uk, res = aggregate_with(gb, reqs, mr)
    assert gb.stats()["mode"] == mode
    _check(keys, reqs, uk, res)
    del uk, res
    assert not mr.live


@pytest.mark.parametrize("tuning", [{}, {"force_mode": 2}])
def test_rows_that_do_not_fit_as_records_take_the_global_table(tuning):
    """32-byte records of 1.1M rows are 35 MB: a resource that gives 20 MB blocks holds every column
    and the 50k groups' table, so the call still runs."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(3)
    n = 1_100_000
    keys = [cb.Column.from_numpy(rng.integers(0, 50_000, n))]
    reqs = [cb.GroupByRequest(cb.Column.from_numpy(rng.integers(-9, 9, n), rng.random(n) > 0.1), [agg.sum(), agg.max()])]
    reqs.append(cb.GroupByRequest(cb.Column.from_numpy(rng.normal(size=n)), [agg.sum()]))
    gb = cb.GroupBy(cb.Table(keys))
    if tuning:
        gb.set_tuning(**tuning)
    mr = DeviceResource(limit=20_000_000)
    uk, res = aggregate_with(gb, reqs, mr)
    assert mr.refused and gb.stats()["mode"] == 0 and gb.stats()["retries"] == 1
    _check(keys, reqs, uk, res)
    del uk, res
    assert not mr.live


def test_a_call_that_fails_for_memory_leaves_the_next_one_alone():
    """The blocks of a failed call go back, and the thread's next call, on another stream, gives its own result."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(4)
    n = 1_100_000
    keys = [cb.Column.from_numpy(rng.integers(0, 50_000, n))]
    reqs = [cb.GroupByRequest(cb.Column.from_numpy(rng.integers(-9, 9, n)), [agg.sum(), agg.max()])]
    gb = cb.GroupBy(cb.Table(keys))
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    for limit in (200_000, 1_000_000):
        small = DeviceResource(limit=limit)
        with pytest.raises(MemoryError):
            aggregate_with(gb, reqs, small)
        assert not small.live
        uk, res = aggregate_with(gb, reqs, DeviceResource(), stream=other)
        _check(keys, reqs, uk, res)
