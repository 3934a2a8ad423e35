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
