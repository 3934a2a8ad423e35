"""Values that the far-first list kernels must neither spread nor lose: sources
that are not in a bucket's list, masses that are infinite or not a number,
sums that overflow, and the last bits of the lane groups' sums."""
import ctypes as C
import math
from types import SimpleNamespace

import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import gravity
from changa_gb300.tree import ListRequest

pytestmark = pytest.mark.gpu

HERE = (3 | 3 << 3 | 3 << 6) << 22  # the replica at the origin


def evaluate(call, sources, targets, lists):
    """`call` on buckets of one list each: lists holds (first target, targets,
    source indices)."""
    import torch
    idx = np.concatenate([np.asarray(l[2], np.int32) for l in lists])
    entries = np.stack([idx, np.full(len(idx), HERE, np.int32)], 1)
    markers = np.concatenate([[0], np.cumsum([len(l[2]) for l in lists])]).astype(np.int32)
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
         (entries, markers, np.array([l[0] for l in lists], np.int32),
          np.array([l[1] for l in lists], np.int32), sources, targets)]
    r = N.ChangaListRequest()
    r.list, r.markers, r.starts, r.sizes = (x.data_ptr() for x in t[:4])
    r.n_buckets, r.n_entries = len(lists), len(idx)
    v = torch.zeros((len(targets), 5), dtype=torch.float64, device="cuda")
    N.check(call(t[4].data_ptr(), len(sources), t[5].data_ptr(), len(targets), C.byref(r), 0.0,
                 v.data_ptr(), torch.cuda.current_stream().cuda_stream))
    return v.cpu().numpy()


@pytest.fixture(params=[17, 18])
def variant(cuda_ok, request):
    """A warp per bucket, a CTA per bucket."""
    lib = N.cuda_lib()
    saved = [lib.changa_gb300_get_list_variant(k) for k in (4, 5)]
    for k in (4, 5):
        assert lib.changa_gb300_set_list_variant(k, request.param) == 0
    yield request.param
    for k, s in zip((4, 5), saved):
        lib.changa_gb300_set_list_variant(k, s)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n_list", [1, 5, 31])
def test_a_mass_that_is_not_in_the_list(variant, bad, n_list):
    """Particle 0 has no finite mass and is in no list; the buckets' sources
    are all within the softening, so no block has a far source."""
    rng = np.random.default_rng(n_list)
    parts = np.concatenate([np.full((64, 1), 0.5), np.full((64, 1), 10.0),
                            rng.uniform(-1, 1, (64, 3))], 1)
    sizes = [1, 3, 16]
    lists, at = [], 1
    for s in sizes:
        lists.append((at, s, rng.choice(np.arange(21, 64), n_list, replace=False)))
        at += s
    call = N.cuda_lib().changa_part_forces_mixed
    want = evaluate(call, parts, parts, lists)
    parts[0, 0] = bad
    got = evaluate(call, parts, parts, lists)
    assert np.isfinite(want).all() and (want[1:at, 3] < 0).all()
    assert np.array_equal(got[1:at], want[1:at])


@pytest.mark.parametrize("name", ["part_forces_mixed", "cell_forces_mixed", "part_forces_fp64",
                                  "cell_forces_fp64"])
def test_a_marker_far_below_zero_is_an_empty_list(variant, name):
    """A list that ends 2^31 before it begins holds nothing; the length of the
    next one is that of its entries."""
    import torch
    rng = np.random.default_rng(4)
    targets = np.concatenate([np.ones((40, 1)), np.full((40, 1), 0.1), rng.normal(size=(40, 3))], 1)
    sources = targets
    if name.startswith("cell"):
        sources = np.zeros((40, 12))
        sources[:, 1], sources[:, 2], sources[:, 3:6] = 0.1, 1.0, rng.normal(size=(40, 3)) + 5
    entries = np.stack([np.arange(40), np.full(40, HERE)], 1).astype(np.int32)
    markers = np.array([7, -2 ** 31, 40, 40], np.int32)  # lists 7.., 0..40 and an empty one
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
         (entries, markers, np.array([0, 10, 30], np.int32), np.array([10, 20, 10], np.int32),
          sources, targets)]
    r = N.ChangaListRequest()
    r.list, r.markers, r.starts, r.sizes = (x.data_ptr() for x in t[:4])
    r.n_buckets, r.n_entries = 3, 40
    v = torch.zeros((40, 5), dtype=torch.float64, device="cuda")
    call = getattr(N.cuda_lib(), "changa_" + name)
    N.check(call(t[4].data_ptr(), 40, t[5].data_ptr(), 40, C.byref(r), 0.0, v.data_ptr(),
                 torch.cuda.current_stream().cuda_stream))
    v = v.cpu().numpy()
    want = evaluate(call, sources, targets, [(0, 10, []), (10, 20, range(40))])
    assert (want[10:30, 3] < 0).all() and np.array_equal(v, want)


def test_the_groups_sums_keep_fp64_bits(variant):
    """One target, every group one source of mass m1 and, a block later, one
    of m2 below m1's last bit, all at distance 1: a group's compensated sum is
    m1 + m2 exactly, of 49 bits, and the join of the G groups may lose no more
    than G - 1 FP64 additions would."""
    block = 32 if variant == 17 else 128
    groups = block // 2
    rng = np.random.default_rng(11)
    parts, lists, want = [[1.0, 0.0, 0.0, 0.0, 0.0]], [], []
    for _ in range(40):
        m = [(rng.integers(1 << 23, 1 << 24, groups) | 1) * 2.0 ** -23,
             (rng.integers(1 << 23, 1 << 24, groups) | 1) * 2.0 ** -49]
        at = len(parts)
        for mass in np.stack([np.concatenate(m), np.zeros(2 * groups)], 1).ravel():
            d = np.zeros(3)
            d[rng.integers(3)] = rng.choice([-1.0, 1.0])
            parts.append([mass, 0.0, *d])
        lists.append((0, 1, np.arange(at, len(parts))))
        want.append(math.fsum(m[0]) + math.fsum(m[1]))
    parts = np.array(parts)
    unit = len(parts)
    parts = np.concatenate([parts, [[1.0, 0.0, 1.0, 0.0, 0.0]]])
    call = N.cuda_lib().changa_part_forces_mixed
    assert evaluate(call, parts, parts, [(0, 1, [unit])])[0, 3] == -1.0  # 1 / sqrt(1) is exact
    got = [-evaluate(call, parts, parts, [l])[0, 3] for l in lists]
    want = np.array(want)
    assert (np.abs(got - want) <= (groups - 1) * 2.0 ** -53 * want).all()


@pytest.mark.parametrize("variant", [17, 18])
def test_an_infinite_potential_of_the_fp32_form(cuda_ok, variant):
    """A mass of 3e38 at distance 1/2, whose potential of 6e38 is past FP32,
    among finite ones in the other groups: the potential is infinite and so is
    the acceleration toward it, not NaN."""
    lib = N.cuda_lib()
    parts = np.zeros((100, 5), np.float32)
    parts[:, 0] = 1.0
    parts[1:, 2:] = np.random.default_rng(2).uniform(1, 2, (99, 3))
    parts[40] = 3e38, 0.0, 0.5, 0.0, 0.0
    one = lambda x: np.array([x], np.int32)
    entries = np.stack([np.arange(1, 100), np.full(99, HERE)], 1).astype(np.int32)
    empty = ListRequest(entries[:0], one(0), one(0)[:0], one(0)[:0], one(0)[:0])
    inp = gravity.DropInInputs(SimpleNamespace(
        n=100, order=2, period=0.0, cells=empty, abi_moments=lambda: np.zeros((4, 12), np.float32),
        plist=ListRequest(entries, np.array([0, 99], np.int32), one(0), one(1), one(0)),
        abi_parts=lambda: parts))
    saved = lib.changa_gb300_get_list_variant(1)
    assert lib.changa_gb300_set_list_variant(1, variant) == 0
    try:
        got = gravity.dropin_step(inp).copy()
    finally:
        lib.changa_gb300_set_list_variant(1, saved)
        inp.free()
    assert got[0, 3] == -np.inf and got[0, 0] == np.inf


@pytest.mark.parametrize("xx", [1e-3, 3.3e-5, 7e-7])
def test_a_near_cells_small_moment(variant, xx):
    """A cell at distance 1 along x, near because another target's softening
    is large but softening none of its own pair: there 1/r is exact, the trace
    terms are M = 3 tr and cancel, and the acceleration is 3 xx (1 - 5/2).
    Five FP32 roundings of that: its moment is not read off the trace."""
    tgt = np.array([[1.0, 0.0, 0.0, 0.0, 0.0], [1.0, 10.0, 0.1, 0.1, 0.1]])
    cell = np.zeros((1, 12))
    cell[0, 2:6] = 3.0, -1.0, 0.0, 0.0
    cell[0, 6], cell[0, 9], cell[0, 11] = xx, 1.0, 1.0 - xx  # half the trace is 1
    got = evaluate(N.cuda_lib().changa_cell_forces_mixed, cell, tgt, [(0, 2, [0])])
    assert abs(got[0, 0] / (-4.5 * xx) - 1.0) < 5 * 2.0 ** -24


@pytest.mark.parametrize("cell", [False, True])
@pytest.mark.parametrize("form,n", [("fp64", 1), ("fp64", 2), ("fp64", 5), ("mixed", 5)])
def test_a_mass_that_is_not_a_number_leaves_dtgrav(variant, cell, form, n):
    """Such a source makes the acceleration NaN; dtGrav's maximum is that of
    the others, as fmax takes it."""
    rng = np.random.default_rng(8)
    tgt = np.concatenate([np.ones((n, 1)), np.zeros((n, 1)), rng.uniform(0, 0.1, (n, 3))], 1)
    src = np.zeros((70, 12 if cell else 5))
    src[:, 2 if cell else 0] = rng.uniform(1, 2, 70)
    src[:, (3 if cell else 2):(6 if cell else 5)] = rng.uniform(1, 2, (70, 3))
    call = getattr(N.cuda_lib(), "changa_%s_forces_%s" % ("cell" if cell else "part", form))
    want = evaluate(call, src, tgt, [(0, n, [k for k in range(70) if k != 33])])
    src[33, 2 if cell else 0] = np.nan
    got = evaluate(call, src, tgt, [(0, n, range(70))])
    assert np.isnan(got[:, :4]).all() and (want[:, 4] > 0).all()
    assert np.array_equal(got[:, 4], want[:, 4])
