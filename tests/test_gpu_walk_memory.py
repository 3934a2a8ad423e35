"""The device walk with less and less memory: pools and slots that cannot be
had, and lists for which there is room only without them.  It succeeds down to
little more than the lists themselves, as counting and filling needs, with the
host walk's entries every time, and then fails with an error."""
import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import ics, tree
from changa_gb300.walk import gpu_walk, same_entries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [0, 8])
@pytest.mark.parametrize("order", [2, 4])
def test_walk_with_less_memory(cuda_ok, order, groups):
    n = 30000
    p = ics.plummer(n, ics.rng_for(9), soft=0.05)
    L = tree.build_lists(p["pos"], p["mass"], p["soft"], n_bucket=8, theta=0.6, order=order)
    nb = len(L.bucket_starts)
    lists = 8 * sum(r.n_entries for r in (L.cells, L.plist, L.softcells) if r is not None)
    # node records and the group arrays are below 2 KB a bucket, and a group's
    # lists and frontier are shared by its buckets, so below all lists / 2
    least = lists + 2048 * nb + (lists // 2 if groups else 0)
    lib = N.cuda_lib()
    lib.changa_walk_set_groups(groups, 1)
    passes, limit = [], 16 * least
    try:
        while True:
            lib.changa_walk_set_test_memory(int(limit))
            tm = {}
            try:
                got = gpu_walk(L, timings=tm)
            except Exception:
                assert limit < least
                break
            assert same_entries(L.cells, got[0], nb) and same_entries(L.plist, got[1], nb)
            if order == 4:
                assert same_entries(L.softcells, got[2], nb)
            passes.append(tm["passes"])
            limit *= 0.9
    finally:
        lib.changa_walk_set_test_memory(0)
        lib.changa_walk_set_groups(32, 10240)
    # all three ways in turn: gathered, the pools given up for the lists, no pools
    assert passes[0] == 1 and passes[-1] == 2 and 3 in passes
    assert limit > lists / 2
    assert same_entries(L.cells, gpu_walk(L)[0], nb)


@pytest.mark.parametrize("groups", [0, 8])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("n_bucket", [8, 300])
def test_walk_whose_pools_run_short(cuda_ok, n_bucket, order, groups):
    """Pools of a chunk per bucket and list: warps that find them short, and
    those that start after, only count; the counts and the filled lists are the
    host walk's."""
    p = ics.plummer(12000, ics.rng_for(10), soft=0.3)
    L = tree.build_lists(p["pos"], p["mass"], p["soft"], n_bucket=n_bucket, theta=0.6, order=order)
    nb = len(L.bucket_starts)
    lib = N.cuda_lib()
    lib.changa_walk_set_groups(groups, 1)
    lib.changa_walk_set_pool_factor(0.0)
    try:
        tm = {}
        got = gpu_walk(L, timings=tm)
    finally:
        lib.changa_walk_set_pool_factor(1.2)
        lib.changa_walk_set_groups(32, 10240)
    assert tm["passes"] == 3
    assert same_entries(L.cells, got[0], nb) and same_entries(L.plist, got[1], nb)
    if order == 4:
        assert same_entries(L.softcells, got[2], nb)
