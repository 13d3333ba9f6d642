"""Rows per tile of a batch: a caller's setting is taken as given, the defaults
shrink for small batches, and the stats report the size that is used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [300_000, 70_000, 5_000, 0, 40_000]


def _stats():
    import cudf_b200 as cb
    from cudf_b200 import aggregation as agg
    rng = np.random.default_rng(1)
    inst = [(cb.Table([cb.Column.from_numpy(rng.integers(0, 50, n).astype(np.int32))]),
             [cb.GroupByRequest(cb.Column.from_numpy(rng.integers(0, 9, n)), [agg.sum()])]) for n in ROWS]
    batch = cb.BatchGroupBy(inst, use_graph=False)
    batch.run()
    assert [batch.result(i)[0].num_rows() for i in range(len(ROWS))] == [50, 50, 50, 0, 50]
    return batch.stats()


def _tiles(tile_rows):
    return sum(-(-n // tile_rows) for n in ROWS)


@pytest.fixture
def autotune():
    from cudf_b200 import autotune
    yield autotune
    autotune.set_batch_tuning([], autotune.BATCH_LAUNCH_DEFAULT)


@pytest.mark.parametrize("tile_rows", [1024, 16384, 65536, 262144])
def test_tiles_are_as_set(autotune, tile_rows):
    autotune.set_batch_tuning([], {"block": 512, "tile_rows": tile_rows, "smem_bytes": 96 * 1024})
    st = _stats()
    assert st["tile_rows"] == tile_rows and st["tiles"] == _tiles(tile_rows)


def test_default_tiles_shrink_and_are_reported(autotune):
    autotune.load()
    st = _stats()
    assert 1024 <= st["tile_rows"] < 65536 and st["tiles"] == _tiles(st["tile_rows"])
