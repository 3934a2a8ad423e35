"""Hexadecapole evaluations whose cell lists are empty: the device walk keeps
every bucket in its requests, so a bucket without accepted cells is an empty
list, a request may hold no entry at all, and its list may then be null."""
import ctypes as C

import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import gravity, ics, tree
from changa_gb300.walk import gpu_walk

from helpers import force_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1, 2])
def hex_variant(cuda_ok, request):
    lib = N.cuda_lib()
    saved = lib.changa_gb300_get_hex_variant()
    assert lib.changa_gb300_set_hex_variant(request.param) == 0
    yield request.param
    lib.changa_gb300_set_hex_variant(saved)


@pytest.mark.parametrize("form", ["mixed", "fp64"])
@pytest.mark.parametrize("n,n_bucket,soft", [(40, 64, 0.05), (60, 16, 0.05), (4000, 16, 20.0)])
def test_device_lists_without_accepted_cells(hex_variant, form, n, n_bucket, soft):
    """One bucket; a few buckets that open every cell; softenings that send
    every accepted cell to the softened lists.  The host lists leave empty
    buckets out, and give the same sums but for their order (up to 4000 terms
    of one sign in blocks of 32 in FP32: 32 x 2^-24 of the sum, against net
    forces of at least a thousandth of it)."""
    p = ics.plummer(n, ics.rng_for(n), soft=soft)
    L = tree.build_lists(p["pos"], p["mass"], p["soft"], n_bucket=n_bucket, theta=0.7, order=4)
    assert L.cells.n_entries == 0 and (L.softcells.n_entries > 0) == (soft > 1)
    reqs = gpu_walk(L)
    assert reqs[0].n_buckets == len(L.bucket_starts) and reqs[0].n_entries == 0
    host = gravity.DeviceSystem(L).step(form).cpu().numpy()
    dev = gravity.DeviceSystem(L, device_reqs=reqs).step(form).cpu().numpy()
    assert np.isfinite(dev).all()
    assert force_rel_err(dev, host).max() < (2e-3 if form == "mixed" else 1e-10)


def test_request_without_a_list(hex_variant):
    """No entry and no list at all, for buckets of every lane group: nothing
    is added, and dtGrav's maximum is taken with zero."""
    import torch
    rng = np.random.default_rng(3)
    sizes = np.arange(1, 34, dtype=np.int32)
    n = int(sizes.sum())
    parts = np.concatenate([np.ones((n, 1)), np.full((n, 1), 1e-3), rng.normal(size=(n, 3))], 1)
    starts = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    t = [torch.from_numpy(x).cuda() for x in
         (np.zeros(len(sizes) + 1, np.int32), starts, sizes, parts, np.ones((1, 27)))]
    r, none = N.ChangaListRequest(), N.ChangaListRequest()
    r.list = None
    r.markers, r.starts, r.sizes = (x.data_ptr() for x in t[:3])
    r.n_buckets, r.n_entries = len(sizes), 0
    v = torch.from_numpy(rng.normal(size=(n, 5))).cuda()
    want = v.clone()
    want[:, 4].clamp_(min=0.0)
    N.check(N.cuda_lib().changa_gravity_step_hexa(
        N.CHANGA_FORM_MIXED, t[4].data_ptr(), 1, t[3].data_ptr(), n, C.byref(r), C.byref(none),
        C.byref(none), 0.0, None, v.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(v, want)
