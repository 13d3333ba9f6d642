"""Repeated calls through the engine's default memory pool find the blocks that
the calls before them freed (in a process of its own: the pool is per process)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# bench.py's default workload
SCRIPT = r'''
import torch
import bench
import cudf_b200 as cb
from cudf_b200 import aggregation as agg
key, vals, masks = bench.make_inputs_device(bench.N_ROWS, bench.SEED, torch.device("cuda", 0))
aggs = [agg.sum(), agg.count(), agg.min(), agg.max(), agg.mean()]
types = [cb.TypeId.INT64, cb.TypeId.FLOAT64, cb.TypeId.FLOAT32]
reqs = [cb.GroupByRequest(cb.Column(t, v, m), aggs) for t, v, m in zip(types, vals, masks)]
gb = cb.GroupBy(cb.Table([cb.Column(cb.TypeId.INT64, key)]))
seen, out = [], None
for _ in range(16):
    out = gb.aggregate(reqs)  # the result before it is freed when this one is there
    seen.append(out[0][0].data.data_ptr())
assert gb.stats()["mode"] == 2
print(len(set(seen[6:])))
'''


def test_equal_calls_alternate_between_two_result_blocks():
    """Two result blocks are alive at a time.  A third address means that the pool remapped freed pages
    (milliseconds in the driver, on every call) because another allocation took part of the free block."""
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split()[-1]) <= 2
