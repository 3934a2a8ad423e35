"""The device walk where its branches change: coordinates at which the FP32
screen cannot decide (exact ties on a regular lattice, structure far smaller
than its distance from the origin, extreme units, a period that FP32 cannot
hold), group lists longer than their slots, and bucket lists longer than the
pools hold.  Every decision is an FP64 one, so the entries equal the host
walk's exactly."""
import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import ics, tree
from changa_gb300.walk import gpu_walk, same_entries

pytestmark = pytest.mark.gpu


def check(L, **kw):
    tm = {}
    cells, plist, soft = gpu_walk(L, timings=tm, **kw)
    nb = len(L.bucket_starts)
    assert same_entries(L.cells, cells, nb) and same_entries(L.plist, plist, nb)
    if L.order == 4:
        assert same_entries(L.softcells, soft, nb)
    return tm


@pytest.mark.parametrize("groups", [0, 8])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("scale,shift,period", [
    (1.0, 0.0, 0.0), (1.0, 0.0, 1.0), (0.1, 0.0, 0.1), (1e-3, 1000.0, 0.0), (1e-6, 1.0, 0.0),
    (1e-14, 0.0, 0.0), (1e-25, 0.0, 0.0), (1e14, 1e15, 0.0), (1e25, 0.0, 0.0)])
def test_walk_of_a_regular_lattice(cuda_ok, scale, shift, period, order, groups):
    g = (np.stack(np.meshgrid(*[np.arange(16)] * 3, indexing="ij"), -1).reshape(-1, 3) - 7.5) / 16
    pos = g * scale + shift
    n = len(pos)
    L = tree.build_lists(pos, np.full(n, 1.0 / n), np.full(n, 0.01 * scale), n_bucket=8, theta=0.7,
                         order=order, period=period)
    lib = N.cuda_lib()
    lib.changa_walk_set_groups(groups, 1)
    try:
        check(L)
    finally:
        lib.changa_walk_set_groups(32, 10240)


@pytest.mark.parametrize("order", [2, 4])
def test_walk_groups_outgrow_their_slots(cuda_ok, order):
    """Groups of one bucket hold that bucket's whole lists, here more than the
    3072 particles of a slot."""
    p = ics.plummer(6000, ics.rng_for(3), soft=0.05)
    L = tree.build_lists(p["pos"], p["mass"], p["soft"], n_bucket=64, theta=0.3, order=order)
    assert np.diff(L.plist.markers).max() > 3072
    lib = N.cuda_lib()
    lib.changa_walk_set_groups(1, 1)
    try:
        check(L)
    finally:
        lib.changa_walk_set_groups(32, 10240)


@pytest.mark.parametrize("groups", [0, 8])
@pytest.mark.parametrize("theta,passes", [(0.7, 1), (0.15, 3)])
def test_walk_of_a_small_tree_appends(cuda_ok, theta, passes, groups):
    """Pools of 1024 entries (a fifth more) per bucket and list and a chunk of
    256 each: enough, or replaced by the fill pass; either way the arrays that
    count + fill write, when both walk in one phase."""
    p = ics.plummer(8000, ics.rng_for(4), soft=0.05)
    L = tree.build_lists(p["pos"], p["mass"], p["soft"], n_bucket=8, theta=theta)
    long = max(L.cells.n_entries, L.plist.n_entries) / len(L.bucket_starts)
    assert (long > 1229 + 256) == (passes == 3)
    lib = N.cuda_lib()
    lib.changa_walk_set_groups(groups, 1)
    try:
        assert check(L)["passes"] == passes
        if not groups:
            one, two = gpu_walk(L), gpu_walk(L, method="two_pass")
            for a, b in zip(one[:2], two[:2]):
                assert np.array_equal(a.to_host()[0], b.to_host()[0])
                assert np.array_equal(a.to_host()[1], b.to_host()[1])
    finally:
        lib.changa_walk_set_groups(32, 10240)
