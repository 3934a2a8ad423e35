"""Drop-in requests on several streams at once: a cell list that goes up whole,
and after it on the same stream a particle list that goes up in chunks.  Each
stream's sums are the bits that its requests alone give, whatever else is in
flight."""
import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import gravity
from changa_gb300.tree import ListRequest

pytestmark = pytest.mark.gpu


def lists(seed):
    """2 MiB of cell entries and 72 MiB of particle entries for 4000 buckets."""
    rng = np.random.default_rng(seed)
    nb, nt, nm = 4000, 8, 500
    n_tgt = nb * nt
    n = n_tgt + 5000
    pos = rng.uniform(0.5, 1.0, (n, 3))
    pos[:n_tgt] = rng.uniform(0.0, 0.05, (n_tgt, 3))
    parts = np.concatenate([rng.uniform(1, 2, (n, 1)) / n, np.full((n, 1), 1e-3), pos],
                           1).astype(np.float32)
    mom = np.zeros((nm, 12), np.float32)  # {radius, soft, M, cm, xx, xy, xz, yy, yz, zz}
    mom[:, 1], mom[:, 2], mom[:, 3:6] = 1e-3, 1.0 / nm, rng.uniform(0.5, 1.0, (nm, 3))
    out = []
    for n_entries, lo, hi in ((1 << 18, 0, nm), (9 << 20, n_tgt, n)):
        lst = np.empty((n_entries, 2), np.int32)
        lst[:, 0] = rng.integers(lo, hi, n_entries)
        lst[:, 1] = (3 | 3 << 3 | 3 << 6) << 22
        out.append(ListRequest(lst, np.linspace(0, n_entries, nb + 1).astype(np.int32),
                               np.arange(nb, dtype=np.int32) * nt, np.full(nb, nt, np.int32),
                               np.arange(nb)))
    return n_tgt, SimpleNamespace(n=n, order=2, period=0.0, cells=out[0], plist=out[1],
                                  abi_parts=lambda: parts, abi_moments=lambda: mom)


def test_requests_in_flight_on_several_streams(cuda_ok):
    import torch
    lib, rt = N.cuda_lib(), gravity._cudart()
    cases = [lists(k) for k in range(3)]
    inps = [gravity.DropInInputs(c[1]) for c in cases]
    streams = [torch.cuda.Stream() for _ in inps]
    dev = []
    try:
        alone = [gravity.dropin_step(i, stream=s.cuda_stream).copy()
                 for i, s in zip(inps, streams)]
        for i, s in zip(inps, streams):
            d = [C.c_void_p() for _ in range(3)]
            lib.DataManagerTransferLocalTree(i.moments.ptr, i.moments.nbytes, i.parts.ptr,
                                             i.parts.nbytes, i.vars.ptr, i.vars.nbytes,
                                             *[C.byref(x) for x in d], s.cuda_stream, i.n, None)
            dev.append(d)
        torch.cuda.synchronize()
        for k in (0, 1):
            for i, s, d in zip(inps, streams, dev):
                lst, mk, st, sz, req = i.reqs[k]
                r = N.CudaRequest()
                r.stream = s.cuda_stream
                r.d_localMoments, r.d_localParts, r.d_localVars = d
                r.list, r.bucketMarkers, r.bucketStarts, r.bucketSizes = (lst.ptr, mk.ptr, st.ptr,
                                                                          sz.ptr)
                r.numInteractions, r.numBucketsPlusOne = req.n_entries, req.n_buckets + 1
                r.fperiod, r.node = 0.0, k == 0
                (lib.TreePieceCellListDataTransferLocal if k == 0 else
                 lib.TreePiecePartListDataTransferLocal)(C.byref(r))
        for i, s, d in zip(inps, streams, dev):
            lib.TransferParticleVarsBack(i.out.ptr, i.out.nbytes, d[2], s.cuda_stream, None)
        torch.cuda.synchronize()
        for (n_tgt, _), i, v in zip(cases, inps, alone):
            assert (v[:n_tgt, :3] > 0).all() and np.array_equal(i.out.array, v)
    finally:
        for d in dev:
            for x in d:
                rt.cudaFree(x)
        for i in inps:
            i.free()
