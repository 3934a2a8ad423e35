"""The far-first list kernels (a warp per bucket, a CTA per bucket, and the
rule between them) at the edges of their tiles: bucket sizes around whole
warps, halves and thirds of a warp and the CTA kernel's target chunk, list
lengths around one and several blocks of both, sources inside and outside the
softening, of one mass and of several, with and without replica offsets."""
import ctypes as C

import numpy as np
import pytest

import oracle
from changa_gb300 import _native as N
from changa_gb300.tree import ListRequest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 8, 11, 16, 17, 20, 31, 32, 33, 63, 64, 65, 100]
LENGTHS = [0, 1, 2, 31, 32, 33, 64, 127, 128, 129, 257]


def request(rng, n_sources, period):
    sizes = np.array([s for s in SIZES for _ in LENGTHS], np.int32)
    lens = np.array([n for _ in SIZES for n in LENGTHS], np.int64)
    starts = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    markers = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    lst = np.empty((int(lens.sum()), 2), np.int32)
    lst[:, 0] = rng.integers(0, n_sources, len(lst))
    o = rng.integers(-1, 2, (len(lst), 3)) if period else np.zeros((len(lst), 3), np.int64)
    lst[:, 1] = ((o[:, 0] + 3) | ((o[:, 1] + 3) << 3) | ((o[:, 2] + 3) << 6)) << 22
    return ListRequest(lst, markers, starts, sizes, np.arange(len(sizes), dtype=np.int32))


def device(req):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda()
         for x in (req.list, req.markers, req.starts, req.sizes)]
    r = N.ChangaListRequest()
    r.list, r.markers, r.starts, r.sizes = (x.data_ptr() for x in t)
    r.n_buckets, r.n_entries = req.n_buckets, req.n_entries
    return r, t


def bound(req, mass, pos, tgt, soft_min, period):
    """Sum over each target's list of m / max(r, h)^2 (and of m / max(r, h)):
    the scale that every pair's rounding is relative to."""
    acc, pot = np.zeros(len(tgt)), np.zeros(len(tgt))
    for b in range(req.n_buckets):
        e = slice(req.markers[b], req.markers[b + 1])
        s = slice(req.starts[b], req.starts[b] + req.sizes[b])
        code = req.list[e, 1] >> 22
        off = period * (np.stack([code & 7, (code >> 3) & 7, (code >> 6) & 7], 1) - 3)
        d = (pos[req.list[e, 0]] + off)[None] - tgt[s][:, None]
        r = np.maximum(np.linalg.norm(d, axis=2), soft_min)
        acc[s] += (mass[req.list[e, 0]] / r ** 2).sum(1)
        pot[s] += (mass[req.list[e, 0]] / r).sum(1)
    return acc, pot


@pytest.mark.parametrize("variant", [17, 18, 19])
@pytest.mark.parametrize("masses", ["one", "several"])
@pytest.mark.parametrize("period", [0.0, 1.0])
def test_far_first_kernels_at_tile_edges(cuda_ok, variant, masses, period):
    import torch
    rng = np.random.default_rng(20261203 + variant)
    n = 6000
    parts = np.empty((n, 5))
    parts[:, 0] = 1.0 / n if masses == "one" else rng.choice([1.0, 3.0, 7.5], n) / n
    parts[:, 1] = rng.choice([1e-3, 0.02, 0.1], n)
    parts[:, 2:] = rng.uniform(-0.5, 0.5, (n, 3))
    at = 0  # the buckets' targets are compact, so that most sources are far
    for size in [s for s in SIZES for _ in LENGTHS]:
        parts[at:at + size, 2:] = rng.uniform(-0.5, 0.5, 3) + rng.uniform(-0.02, 0.02, (size, 3))
        at += size
    assert at <= n
    nm = 512
    mom = np.zeros((nm, 12))
    mom[:, 0] = 0.05
    mom[:, 1] = rng.choice([1e-3, 0.1], nm)
    mom[:, 2] = rng.uniform(0.5, 2.0, nm) / nm
    mom[:, 3:6] = rng.uniform(-0.5, 0.5, (nm, 3))
    d = rng.normal(0, 0.01, (nm, 4, 3))
    q = np.einsum("nki,nkj->nij", d, d) / 4 * mom[:, 2, None, None]
    mom[:, 6:] = np.stack([q[:, 0, 0], q[:, 0, 1], q[:, 0, 2], q[:, 1, 1], q[:, 1, 2], q[:, 2, 2]], 1)
    lib = N.cuda_lib()
    dp, dm = torch.from_numpy(parts).cuda(), torch.from_numpy(mom).cuda()
    cases = [(5, lib.changa_part_forces_mixed, request(rng, n, period), dp, n, parts),
             (4, lib.changa_cell_forces_mixed, request(rng, nm, period), dm, nm, mom)]
    for kernel, call, req, src, n_src, host in cases:
        cell = kernel == 4
        ref = (oracle.cell_forces if cell else oracle.part_forces)(host, parts, req, fperiod=period)
        start = rng.normal(0, 1e-6, (n, 5))  # results are added to what vars holds
        start[:, 4] = 0.0
        v = torch.from_numpy(start).cuda()
        r, keep = device(req)
        saved = lib.changa_gb300_get_list_variant(kernel)
        assert lib.changa_gb300_set_list_variant(kernel, variant) == 0
        try:
            s = torch.cuda.current_stream().cuda_stream
            N.check(call(src.data_ptr(), n_src, dp.data_ptr(), n, C.byref(r), period,
                         v.data_ptr(), s))
            v = v.cpu().numpy() - np.concatenate([start[:, :4], np.zeros((n, 1))], 1)
        finally:
            lib.changa_gb300_set_list_variant(kernel, saved)
        col = (2, slice(3, 6)) if cell else (0, slice(2, 5))
        # a pair's separation is known to 2^-24 of coordinates below 2, which
        # at the smallest softened separation (2 x 1e-3, spline-flat below)
        # is 6e-5 relative and three times that in 1/r^3; a cell's quadrupole
        # adds at most (0.02 / r)^2 of its monopole at r above 0.02
        acc, pot = bound(req, host[:, col[0]], host[:, col[1]], parts[:, 2:], 2e-3, period)
        rel = np.abs(v[:, :3] - ref[:, :3]).max(1) / np.maximum(acc, 1e-30)
        assert rel.max() < 2e-4 and np.median(rel[acc > 0]) < 2e-6, (rel.max(), np.median(rel))
        relp = np.abs(v[:, 3] - ref[:, 3]) / np.maximum(pot, 1e-30)
        assert relp.max() < 1e-4 and np.median(relp[pot > 0]) < 1e-6, relp.max()
        np.testing.assert_allclose(v[:, 4], ref[:, 4], rtol=4e-4)
        assert not v[acc == 0, :3].any() or np.abs(v[acc == 0, :3]).max() < 1e-20


@pytest.mark.parametrize("masses", ["one", "several"])
@pytest.mark.parametrize("period", [0.0, 1.0])
def test_fp64_kernel_at_tile_edges(cuda_ok, masses, period):
    """The plain FP64 form over the same sizes and lengths, buckets of more
    targets than a CTA has threads, and coincident sources and targets."""
    import torch
    rng = np.random.default_rng(20261207)
    sizes = np.array([s for s in SIZES + [255, 256, 257, 300] for _ in LENGTHS], np.int32)
    n = int(sizes.sum()) + 100
    parts = np.empty((n, 5))
    parts[:, 0] = 1.0 / n if masses == "one" else rng.choice([1.0, 3.0, 7.5], n) / n
    parts[:, 1] = rng.choice([0.0, 1e-3, 0.02, 0.1], n)
    parts[:, 2:] = rng.uniform(-0.5, 0.5, (n, 3))
    at = 0
    for size in sizes:
        parts[at:at + size, 2:] = rng.uniform(-0.5, 0.5, 3) + rng.uniform(-0.02, 0.02, (size, 3))
        at += size
    nm = 512
    mom = np.zeros((nm, 12))
    mom[:, 0], mom[:, 1] = 0.05, rng.choice([0.0, 1e-3, 0.1], nm)
    mom[:, 2] = rng.uniform(0.5, 2.0, nm) / nm
    mom[:, 3:6] = rng.uniform(-0.5, 0.5, (nm, 3))
    mom[:64, 3:6] = parts[rng.integers(0, at, 64), 2:]  # cells centred on a target
    mom[:, 6:] = rng.uniform(-1e-4, 1e-4, (nm, 6)) * mom[:, 2:3]
    lib = N.cuda_lib()
    dp, dm = torch.from_numpy(parts).cuda(), torch.from_numpy(mom).cuda()
    for cell in (False, True):
        n_src, host = (nm, mom) if cell else (n, parts)
        req = request(rng, n_src, period)
        more = sizes[len(req.sizes):]
        lens = np.tile(LENGTHS, len(more) // len(LENGTHS))
        lst = np.zeros((int(lens.sum()), 2), np.int32)
        lst[:, 0] = rng.integers(0, n_src, len(lst))
        lst[:, 1] = (3 | 3 << 3 | 3 << 6) << 22
        req = ListRequest(np.concatenate([req.list, lst]),
                          np.concatenate([req.markers, req.markers[-1] + np.cumsum(lens)])
                          .astype(np.int32),
                          np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32), sizes,
                          np.arange(len(sizes), dtype=np.int32))
        ref = (oracle.cell_forces if cell else oracle.part_forces)(host, parts, req, fperiod=period)
        v = torch.zeros((n, 5), dtype=torch.float64, device="cuda")
        r, keep = device(req)
        call = lib.changa_cell_forces_fp64 if cell else lib.changa_part_forces_fp64
        N.check(call((dm if cell else dp).data_ptr(), n_src, dp.data_ptr(), n, C.byref(r), period,
                     v.data_ptr(), torch.cuda.current_stream().cuda_stream))
        v = v.cpu().numpy()
        col = (2, slice(3, 6)) if cell else (0, slice(2, 5))
        acc, pot = bound(req, host[:, col[0]], host[:, col[1]], parts[:, 2:], 1e-5, period)
        # separations are exact differences of coordinates below 2 to 2^-53,
        # at distances of 1e-5 and more (closer pairs are softened or rare)
        assert np.isfinite(v).all()
        ok = np.isfinite(ref).all(1)  # the oracle divides by r = 0 for a cell on its target
        assert ok.sum() >= n - 64
        assert (np.abs(v - ref)[ok, :3].max(1) / np.maximum(acc[ok], 1e-30)).max() < 1e-9
        assert (np.abs(v - ref)[ok, 3] / np.maximum(pot[ok], 1e-30)).max() < 1e-9
        np.testing.assert_allclose(v[ok, 4], ref[ok, 4], rtol=1e-9)


@pytest.mark.parametrize("cut,n_rep", [(2.6, 1), (2.6, 2), (4.6, 1)])
@pytest.mark.parametrize("whole", [True, False])
def test_ewald_fp64_replicas_and_tables(cuda_ok, cut, n_rep, whole):
    """The FP64 Ewald term with more replicas than one culled batch, a ragged
    particle count, and a table whose vectors are not whole (which takes the
    sine and cosine of each)."""
    import torch
    from changa_gb300 import gravity
    rng = np.random.default_rng(5)
    n = 1001
    parts = np.empty((n, 5))
    parts[:, 0], parts[:, 1] = 1.0 / n, 1e-3
    parts[:, 2:] = rng.uniform(0, 1, (n, 3)) ** 2
    m = parts[:, 0]
    cm = (m[:, None] * parts[:, 2:]).sum(0) / m.sum()
    d = parts[:, 2:] - cm
    q = np.einsum("n,ni,nj->ij", m, d, d)
    root = np.array([0.8, 1e-3, m.sum(), *cm, q[0, 0], q[0, 1], q[0, 2], q[1, 1], q[1, 2], q[2, 2]])
    ref = oracle.ewald_forces(parts, root, 1.0, n_rep, cut, 2.8)
    p = gravity.EwaldConfig(1.0, n_rep, cut, 2.8).params(root)
    if not whole:
        p._keep[:, :3] *= 1 + 1e-12
    dp = torch.from_numpy(parts).cuda()
    v = torch.zeros((n, 5), dtype=torch.float64, device="cuda")
    N.check(N.cuda_lib().changa_ewald_forces(N.CHANGA_FORM_FP64, dp.data_ptr(), n, None, n,
                                             C.byref(p), v.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream))
    v = v.cpu().numpy()
    # the tables differ by 1e-12; near the root the recursion of the g_n loses
    # up to (alpha r)^-6 = (4 * 1.2e-3)^-3 of 2^-53 of the O(1) terms
    assert np.abs(v[:, :4] - ref[:, :4]).max() < 1e-8
    assert np.median(np.abs(v[:, :4] - ref[:, :4])) < 1e-11


@pytest.mark.parametrize("extra", [-1, 0, 1, 40000])
def test_dropin_list_around_two_default_chunks(cuda_ok, extra):
    """A drop-in list of just under, at and over two default upload chunks
    (32 MiB for lists this long), against the same list in one upload.  The
    sources lie in one octant of every target at separations above 0.4, so
    nothing cancels: a block of 32 terms is summed in FP32 (32 x 2^-24 = 2e-6
    of the sum) before it joins the compensated total, and twice that for two
    orders of summation is below 1e-5."""
    from types import SimpleNamespace
    from changa_gb300 import gravity
    rng = np.random.default_rng(5)
    n_entries, nb, nt, n = (8 << 20) + extra, 4001, 8, 40000
    n_tgt = nb * nt
    pos = rng.uniform(0.5, 1.0, (n, 3))
    pos[:n_tgt] = rng.uniform(0.0, 0.05, (n_tgt, 3))
    parts = np.concatenate([np.full((n, 1), 1.0 / n), np.full((n, 1), 1e-3), pos], 1).astype(np.float32)
    lst = np.empty((n_entries, 2), np.int32)
    lst[:, 0] = rng.integers(n_tgt, n, n_entries)
    lst[:, 1] = 0x49 * 3 << 22  # the replica at the origin
    markers = np.linspace(0, n_entries, nb + 1).astype(np.int32)
    starts = np.arange(nb, dtype=np.int32) * nt
    sizes = np.full(nb, nt, np.int32)
    empty = ListRequest(np.empty((0, 2), np.int32), np.zeros(1, np.int32), np.empty(0, np.int32),
                        np.empty(0, np.int32), np.empty(0, np.int32))
    inp = gravity.DropInInputs(SimpleNamespace(
        n=n, order=2, period=0.0, plist=ListRequest(lst, markers, starts, sizes, np.arange(nb)),
        cells=empty, abi_moments=lambda: np.zeros((4, 12), np.float32), abi_parts=lambda: parts))
    lib = N.cuda_lib()
    try:
        got = gravity.dropin_step(inp).copy()
        lib.changa_gb300_set_host_chunk_bytes(1 << 30)
        try:
            whole = gravity.dropin_step(inp).copy()
        finally:
            lib.changa_gb300_set_host_chunk_bytes(0)  # the default
    finally:
        inp.free()
    assert (whole[:n_tgt, :3] > 0).all() and not whole[n_tgt:].any()
    np.testing.assert_allclose(got, whole, rtol=1e-5)


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("period", [0.0, 4.0])
def test_hexadecapole_kernels_at_tile_edges(cuda_ok, variant, period):
    """Every number of lane groups a bucket can have (1 to 32) and list lengths
    around their blocks.  Cells of radius 0.01 at separations above 0.2: the
    monopole dominates a pair, so its some 30 roundings are below 2e-6 of M / r^2
    and a block's FP32 sum adds at most 32 x 2^-24 = 2e-6."""
    import torch
    rng = np.random.default_rng(20261206)
    n = 6000
    parts = np.concatenate([np.full((n, 1), 1.0 / n), np.full((n, 1), 1e-4),
                            rng.uniform(-0.5, 0.2, (n, 3))], 1)
    nm = 512
    mom = np.zeros((nm, 27))
    mom[:, 0] = 0.01
    mom[:, 1] = 1e-4
    mom[:, 2] = rng.uniform(0.5, 2.0, nm) / nm
    mom[:, 3:6] = rng.uniform(0.5, 1.0, (nm, 3))
    mom[:, 6:] = rng.normal(0, 0.3, (nm, 21)) * mom[:, 2, None]
    sizes = np.array([s for s in range(1, 34) for _ in LENGTHS], np.int32)
    lens = np.array([k for _ in range(1, 34) for k in LENGTHS], np.int64)
    assert sizes.sum() <= n + 2000
    starts = (np.concatenate([[0], np.cumsum(sizes)[:-1]]) % (n - 40)).astype(np.int32)
    markers = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    lst = np.empty((int(lens.sum()), 2), np.int32)
    lst[:, 0] = rng.integers(0, nm, len(lst))
    o = rng.integers(-1, 2, (len(lst), 3)) if period else np.zeros((len(lst), 3), np.int64)
    lst[:, 1] = ((o[:, 0] + 3) | ((o[:, 1] + 3) << 3) | ((o[:, 2] + 3) << 6)) << 22
    req = ListRequest(lst, markers, starts, sizes, np.arange(len(sizes), dtype=np.int32))
    # buckets share particles where the starts wrap, so each is evaluated for itself
    first = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    rows = np.concatenate([np.arange(s, s + k) for s, k in zip(starts, sizes)])
    own = np.ascontiguousarray(parts[rows])
    req.starts = first[:-1].copy()
    geom = np.zeros((len(sizes), 10))
    for b in range(len(sizes)):
        x = own[first[b]:first[b + 1], 2:]
        geom[b, :3], geom[b, 3] = x.mean(0), 1e-4
        geom[b, 4:7], geom[b, 7:] = x.min(0), x.max(0)
    ref = oracle.cell_forces_hex(mom, own, req, geom, fperiod=period)
    lib = N.cuda_lib()
    dp, dm = torch.from_numpy(own).cuda(), torch.from_numpy(mom).cuda()
    v = torch.zeros((len(own), 5), dtype=torch.float64, device="cuda")
    r, keep = device(req)
    none = N.ChangaListRequest()
    saved = lib.changa_gb300_get_hex_variant()
    assert lib.changa_gb300_set_hex_variant(variant) == 0
    try:
        N.check(lib.changa_gravity_step_hexa(N.CHANGA_FORM_MIXED, dm.data_ptr(), nm, dp.data_ptr(), len(own),
                                             C.byref(r), C.byref(none), C.byref(none), period, None,
                                             v.data_ptr(), torch.cuda.current_stream().cuda_stream))
        v = v.cpu().numpy()
    finally:
        lib.changa_gb300_set_hex_variant(saved)
    acc, pot = bound(req, mom[:, 2], mom[:, 3:6], own[:, 2:], 1e-4, period)
    assert (np.abs(v[:, :3] - ref[:, :3]).max(1) <= 5e-6 * acc).all()
    assert (np.abs(v[:, 3] - ref[:, 3]) <= 5e-6 * pot).all()
    np.testing.assert_allclose(v[:, 4], ref[:, 4], rtol=2e-5)
