"""The partitioned path's row records against the oracle: every record size,
key widths, column offsets, row counts around the tile edges, and values at the
ends of their types."""
import numpy as np
import pytest

from oracle import oracle as O
from parity import run_both

pytestmark = pytest.mark.gpu

# value columns per schema: records of 16, 32, 48, 64 and 96 bytes
SCHEMAS = {
    16: ["i32", "f32"],
    32: ["f64", "i64", "u8", "i16"],
    48: ["f64", "i64", "f64", "f32", "bool"],
    64: ["f64", "i64", "f64", "i64", "f32", "i32", "i8"],
    96: ["f64", "i64", "f64", "i64", "f64", "i64", "f64", "u64"],
}
DTYPE = {"i8": np.int8, "u8": np.uint8, "i16": np.int16, "i32": np.int32, "i64": np.int64, "u64": np.uint64,
         "f32": np.float32, "f64": np.float64, "bool": np.uint8}


def _values(rng, kind, n):
    dt = DTYPE[kind]
    if kind == "bool":
        return rng.integers(0, 2, n).astype(dt)
    if kind in ("f32", "f64"):
        v = rng.normal(size=n).astype(dt)
        v[rng.random(n) < 0.002] = np.nan
        v[rng.random(n) < 0.001] = -0.0
        return v
    info = np.iinfo(dt)
    v = rng.integers(max(info.min, -1000), min(info.max, 1000), n, endpoint=True).astype(dt)
    ends = rng.random(n)
    v[ends < 0.001] = info.min
    v[ends > 0.999] = info.max
    return v


def _column(cb, rng, arr, nullable, offset, type_id=None):
    valid = rng.random(arr.shape[0]) > 0.15 if nullable else None
    c = cb.Column.from_numpy(arr, valid, type_id)
    return cb.Column(c.type_id, c.data, c.mask, size=arr.shape[0] - offset, offset=offset)


@pytest.mark.parametrize("offset", [0, 3])
@pytest.mark.parametrize("nullable", [False, True])
@pytest.mark.parametrize("key", ["i32", "i64", "i64+i32", "i8+i16"])
@pytest.mark.parametrize("size", sorted(SCHEMAS))
@pytest.mark.parametrize("n", [1, 511, 3073, 40_961, 300_007])
def test_record_shapes(n, size, key, nullable, offset):
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(n * 7 + size)
    rows = n + offset
    ids = rng.integers(0, max(1, n // 3), rows)
    parts = {"i32": [ids.astype(np.int32)], "i64": [ids * 1_000_003 - 5],
             "i64+i32": [ids * 1_000_003, (ids % 7).astype(np.int32)],
             "i8+i16": [(ids % 100).astype(np.int8), (ids % 3000).astype(np.int16)]}[key]
    two = "+" in key
    keys = [_column(cb, rng, k, two, offset) for k in parts]
    # integral sums and sums of squares of values near the ends wrap alike; a
    # float column with huge values would only loosen its own bound
    reqs = []
    for j, kind in enumerate(SCHEMAS[size]):
        aggs = [agg.sum(), agg.min(), agg.max(), agg.count()]
        if j == 0:
            aggs += [agg.mean(), agg.sum_of_squares()]
        c = _column(cb, rng, _values(rng, kind, rows), nullable, offset, O.BOOL8 if kind == "bool" else None)
        reqs.append((c, aggs))
    run_both(keys, reqs, include_null_keys=two, tuning={"force_mode": 2})


@pytest.mark.parametrize("groups", [5_000, 900_000, 2_500_000])
def test_table_fill_and_partition_counts(groups):
    """Few, hundreds and thousands of partitions with tables near their fill
    limit; every group has about two rows."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(groups)
    n = max(2 * groups, 1_100_000) + 13
    key = rng.integers(0, groups, n).astype(np.int64) * 2_654_435_761
    v = rng.integers(-10**9, 10**9, n)
    f = rng.normal(size=n)
    wide = [agg.sum(), agg.min(), agg.max(), agg.mean()]
    gb, *_ = run_both([cb.Column.from_numpy(key)],
                      [(cb.Column.from_numpy(v, rng.random(n) > 0.1), wide), (cb.Column.from_numpy(f), wide)],
                      tuning={"force_mode": 2, "part_fill_pct": 85})
    assert gb.stats()["mode"] == 2


@pytest.mark.parametrize("mode,n,groups", [(1, 400_000, 3), (1, 2_000_000, 900), (2, 2_000_000, 1), (2, 3_000_000, 4_000),
                                           (0, 400_000, 5)])
def test_float32_sums_round_once(mode, n, groups):
    """FLOAT32 sums, means and sums of squares accumulate in 64 bits: however
    many rows a group has, SUM is the float nearest to the exact sum up to the
    64-bit additions' own error (n * 2^-52 of sum|x|, far below half a float
    step), so at most one float step away."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(groups)
    key = rng.integers(0, groups, n).astype(np.int64)
    x = rng.lognormal(size=n).astype(np.float32)
    gb = cb.GroupBy(cb.Table([cb.Column.from_numpy(key)]))
    gb.set_tuning(force_mode=mode)
    uk, res = gb.aggregate([cb.GroupByRequest(cb.Column.from_numpy(x), [agg.sum(), agg.mean(), agg.sum_of_squares()])])
    got = uk[0].to_numpy()[0]
    x64 = x.astype(np.float64)
    total = np.bincount(key, x64, groups)[got]
    count = np.bincount(key, minlength=groups)[got]
    squares = np.bincount(key, x64 * x64, groups)[got]
    for values, exact in ((res[0][0], total), (res[0][2], squares)):
        v = values.to_numpy()[0]
        assert v.dtype == np.float32
        assert np.all(np.abs(v.astype(np.float64) - exact) <= np.spacing(exact.astype(np.float32)))
    assert np.allclose(res[0][1].to_numpy()[0], total / count, rtol=n * 2.0**-52, atol=0)


def _fmix64(k):
    k = k.astype(np.uint64)
    with np.errstate(over="ignore"):
        k ^= k >> np.uint64(33)
        k *= np.uint64(0xff51afd7ed558ccd)
        k ^= k >> np.uint64(33)
        k *= np.uint64(0xc4ceb9fe1a85ec53)
        k ^= k >> np.uint64(33)
    return k


@pytest.mark.parametrize("hidden", [0, 40, 70_000])
@pytest.mark.parametrize("width", [1, 3])
def test_sampled_sketch_with_groups_it_misses(hidden, width):
    """Few groups on a large input are sized from a sample of 4096 runs of 128
    rows.  Groups placed on rows that the sample does not visit still come out:
    they find room in the shared tables, are listed, or (more than the list
    holds) the call is redone from a pass over all rows."""
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    n, chunks = (8 << 20) + 77, 4096
    rng = np.random.default_rng(hidden + width)
    key = rng.integers(0, 5, n).astype(np.int64)
    stratum = n // chunks
    s = np.arange(chunks, dtype=np.int64)
    start = s * stratum + (_fmix64(s) % np.uint64(stratum - 128)).astype(np.int64)
    seen = np.zeros(n, bool)
    seen[(start[:, None] + np.arange(128)).ravel()] = True
    rows = rng.permutation(np.nonzero(~seen)[0])[:hidden]
    key[rows] = 1000 + np.arange(hidden)
    v = rng.integers(-10**6, 10**6, n)
    f = rng.normal(size=n)
    reqs = [(cb.Column.from_numpy(v), [agg.sum(), agg.min(), agg.max(), agg.count()]),
            (cb.Column.from_numpy(f, rng.random(n) > 0.1), [agg.sum(), agg.mean()]),
            (cb.Column.from_numpy(f), [agg.max()])][:width]
    gb, uk, *_ = run_both([cb.Column.from_numpy(key)], reqs)
    assert uk.num_rows() == 5 + hidden
    assert gb.stats()["mode"] == (1 if hidden < 70_000 else gb.stats()["mode"])
