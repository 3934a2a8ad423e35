"""The launches of one evaluation overlap (cells, particles, softened cells,
the Ewald term: each starts while the one before it drains and waits for it
before it adds to the sums).  Evaluated one call after another they give the
same bits, whatever the number and size of the buckets: a CTA or a warp per
bucket, launches that fill the GPU and launches that leave it nearly idle,
repeated so that a missing wait has many chances to show."""
import ctypes as C

import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import gravity, ics, tree

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["mixed", "fp64"])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("n,n_bucket", [(40, 64), (1200, 8), (3000, 64), (9000, 12), (30000, 8)])
@pytest.mark.parametrize("periodic", [False, True])
def test_overlapped_evaluation_equals_separate_calls(cuda_ok, form, order, n, n_bucket, periodic):
    import torch
    rng = ics.rng_for(n)
    p = ics.nfw_halos(n, rng, soft=2e-3) if periodic else ics.plummer(n, rng, soft=0.05)
    period = 1.0 if periodic else 0.0
    L = tree.build_lists(p["pos"], p["mass"], p["soft"], n_bucket=n_bucket, theta=0.7, period=period,
                         order=order, **(dict(n_replicas=1) if periodic else {}))
    ds = gravity.DeviceSystem(L, ewald=gravity.EwaldConfig(1.0, 1, 2.6, 2.8) if periodic else None)
    whole = ds.step(form).clone()
    for _ in range(20):
        assert torch.equal(ds.step(form), whole)
    lib, s = N.cuda_lib(), torch.cuda.current_stream().cuda_stream
    if order == 2:
        cells, parts = ((lib.changa_cell_forces_mixed, lib.changa_part_forces_mixed)
                        if form == "mixed" else
                        (lib.changa_cell_forces_fp64, lib.changa_part_forces_fp64))
        v = torch.zeros_like(whole)
        for call, src, req in ((cells, ds.moments, ds.reqs[0]), (parts, ds.parts, ds.reqs[1])):
            N.check(call(src.data_ptr(), src.shape[0], ds.parts.data_ptr(), n, C.byref(req["c"]),
                         period, v.data_ptr(), s))
    else:  # one list at a time: the step with the other lists empty
        v = torch.zeros_like(whole)
        none = N.ChangaListRequest()
        for k in range(3):
            reqs = [C.byref(ds.reqs[j]["c"] if j == k else none) for j in range(3)]
            N.check(lib.changa_gravity_step_hexa(gravity.FORMS[form], ds.moments.data_ptr(),
                                                 ds.moments.shape[0], ds.parts.data_ptr(), n, *reqs,
                                                 period, None, v.data_ptr(), s))
    if periodic and order == 2:
        N.check(lib.changa_ewald_forces(gravity.FORMS[form], ds.parts.data_ptr(), n, None, n,
                                        C.byref(ds.ewald_params), v.data_ptr(), s))
    if periodic and order == 4:
        none = N.ChangaListRequest()
        N.check(lib.changa_gravity_step_hexa(gravity.FORMS[form], ds.moments.data_ptr(),
                                             ds.moments.shape[0], ds.parts.data_ptr(), n,
                                             *[C.byref(none)] * 3, period, C.byref(ds.ewald_params),
                                             v.data_ptr(), s))
    assert torch.equal(v, whole)
