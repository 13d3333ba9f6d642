"""A device memory resource for tests: torch's allocator behind the engine's
gb_allocator hooks, with blocks at a chosen offset and a limit on their size."""
import ctypes

import torch

from cudf_b200 import _lib
from cudf_b200.column import Table
from cudf_b200.groupby import GroupBy, _out_column, _ResultOwner

_ALLOC = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p)
_FREE = ctypes.CFUNCTYPE(None, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, ctypes.c_void_p)


class GbAllocator(ctypes.Structure):
    _fields_ = [("allocate", _ALLOC), ("deallocate", _FREE), ("ctx", ctypes.c_void_p)]


class DeviceResource:
    """Blocks at `shift` bytes past a multiple of 512; larger ones than `limit` are refused."""

    def __init__(self, shift=0, limit=None):
        self.live, self.sizes, self.refused = {}, [], []
        self.shift, self.limit = shift, limit
        self.hooks = GbAllocator(_ALLOC(self._allocate), _FREE(self._deallocate), None)

    def _allocate(self, ctx, size, stream):
        if self.limit is not None and size > self.limit:
            self.refused.append(size)
            return None
        base = torch.cuda.caching_allocator_alloc(size + self.shift, stream=stream or 0)
        assert base % 512 == 0
        self.live[base + self.shift] = base
        self.sizes.append(size)
        return base + self.shift

    def _deallocate(self, ctx, ptr, size, stream):
        torch.cuda.caching_allocator_delete(self.live.pop(ptr))


def aggregate_with(gb: GroupBy, requests, mr: DeviceResource, stream=None):
    """gb.aggregate(requests) with every allocation made through `mr`."""
    L = _lib.lib()
    reqs = (_lib.GbRequest * max(1, len(requests)))()
    keep = []
    for i, r in enumerate(requests):
        aggs = (_lib.GbAgg * max(1, len(r.aggregations)))(
            *[_lib.GbAgg(int(a.kind), int(a.param)) for a in r.aggregations])
        keep.append(aggs)
        reqs[i] = _lib.GbRequest(r.values.gb_view(), len(r.aggregations), aggs)
    out = ctypes.POINTER(_lib.GbResult)()
    s = stream if stream is not None else torch.cuda.current_stream()
    _lib.check(L.gb_aggregate(gb._h, reqs, len(requests), int(s.cuda_stream), ctypes.byref(mr.hooks), ctypes.byref(out)))
    owner = _ResultOwner(out)
    res = out.contents
    keys = Table([_out_column(res.keys[k], owner) for k in range(res.num_keys)])
    return keys, [Table([_out_column(res.results[r][j], owner) for j in range(res.num_results[r])])
                  for r in range(res.num_requests)]
