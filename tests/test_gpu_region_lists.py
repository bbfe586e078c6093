"""The ray queues as builds make them on the device, against the host statement
of the SM-affine schedule (mrf_test_region_lists) per view: equal element for
element, for ray, view and region counts around the edges -- one ray, no ray in
BP, fewer rays than regions, more views than rays, blocks' remainders, ties,
all rays of one length, shares of 0 and 100 per cent."""
import ctypes as C

import numpy as np
import pytest

from mrfmap_gb300 import lib as L
from mrfmap_gb300.params import MapParams

pytestmark = pytest.mark.gpu
U32 = C.POINTER(C.c_uint32)


def _p(a):
    return a.ctypes.data_as(U32)


def _records(a):
    return np.ascontiguousarray(a, dtype=np.int32).ctypes.data_as(C.POINTER(C.c_int32))


def _host(records, regions, share):
    n = len(records)
    home, left = np.zeros(max(n, 1), np.uint32), np.zeros(max(n, 1), np.uint32)
    starts = np.zeros(regions + 1, np.uint32)
    nh, nl = C.c_int64(), C.c_int64()
    rec = np.ascontiguousarray(records if n else np.zeros((1, 3)), dtype=np.int32)
    st = L.load().mrf_test_region_lists(_records(rec), n, regions, share, _p(home), C.byref(nh), _p(starts),
                                        _p(left), C.byref(nl))
    assert st == 0, L.load().mrf_last_error()
    return home[:nh.value], starts, left[:nl.value]


@pytest.mark.parametrize("n,views,regions,share,kind", [
    (1, 1, 152, 75, "mixed"), (1, 1, 1, 100, "one length"), (5, 1, 152, 75, "mixed"), (255, 1, 16, 75, "mixed"),
    (256, 2, 1, 90, "mixed"), (257, 3, 7, 0, "mixed"), (300, 2, 152, 75, "none"), (6000, 1, 152, 75, "mixed"),
    (6001, 5, 3, 100, "one length"), (40000, 4, 152, 60, "ties"), (20, 64, 152, 75, "mixed"),
    (64000, 64, 152, 75, "mixed"), (307200, 1, 152, 75, "mixed"), (921600, 3, 300, 75, "longest"),
])
def test_device_queues_match_the_host(native_lib, n, views, regions, share, kind):
    rng = np.random.default_rng(n + regions)
    n_pre = rng.integers(0, 2000, n)
    n_pre[rng.random(n) < 0.2] = 0
    if kind == "one length":
        n_pre[:] = 40
    if kind == "ties":
        n_pre = rng.choice([0, 4, 300, 65532], n)
    if kind == "longest":
        n_pre[rng.random(n) < 0.01] = 65532
    n_post = np.minimum(n_pre, rng.integers(0, 2500, n)) if kind != "one length" else n_pre
    kdyn = np.full(n, 65535) if kind == "none" else rng.integers(0, 1000, n) if kind != "one length" else 0 * n_pre
    records = np.ascontiguousarray(np.stack([n_pre, n_post, kdyn], 1), dtype=np.int32)
    lists, queue = np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    starts, lefts = np.zeros((views, regions + 1), np.uint32), np.zeros(3 * views, np.uint32)
    lib = L.load()
    m = L.MRFMap(MapParams(res=0.1, dims=(1.0, 1.0, 1.0), rows=4, cols=4, fx=4.0, fy=4.0, cx=2.0, cy=2.0))
    try:
        st = lib.mrf_test_region_lists_device(m.handle, _records(records), n, views, regions, share, _p(lists),
                                              _p(starts), _p(lefts), _p(queue))
        assert st == 0, lib.mrf_last_error()
    finally:
        m.close()
    at = 0
    for v in range(views):
        p0, p1 = n * v // views, n * (v + 1) // views
        home, row, left = _host(records[p0:p1], regions, share)
        act = len(home) + len(left)
        assert np.array_equal(lists[at:at + act], p0 + np.concatenate([home, left]))
        assert np.array_equal(starts[v], at + row)
        assert lefts[v] == at + len(home)
        assert tuple(lefts[views + 2 * v:views + 2 * v + 2]) == (0, len(left))
        bp = np.flatnonzero((n_pre[p0:p1] > 0) & (kdyn[p0:p1] < n_post[p0:p1]))
        assert np.array_equal(queue[at:at + act], p0 + bp[np.argsort(-n_pre[p0:p1][bp], kind="stable")])
        at += act
