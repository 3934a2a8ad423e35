"""The device walk of clouds far smaller than their distance from the origin,
where the FP32 opening test's margin is smallest against its error: random
positions, whose distances to the opening radii fall at all places of the
undecided band.  The entries equal the host walk's exactly."""
import numpy as np
import pytest

from changa_gb300 import _native as N
from changa_gb300 import tree
from changa_gb300.walk import gpu_walk, same_entries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [0, 8])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("log", [-22, -20, -19, -18, -17, -15])
def test_cloud_far_from_the_origin(cuda_ok, log, order, groups):
    rng = np.random.default_rng(100 - log)
    n, at = 30000, 520.0
    ext = at * 2.0 ** log
    pos = at + ext * rng.normal(0, 0.3, (n, 3)).clip(-1, 1)
    L = tree.build_lists(pos, np.full(n, 1.0 / n), np.full(n, 1e-3 * ext), n_bucket=8, theta=0.6,
                         order=order)
    lib = N.cuda_lib()
    lib.changa_walk_set_groups(groups, 1)
    try:
        cells, plist, soft = gpu_walk(L)
    finally:
        lib.changa_walk_set_groups(32, 10240)
    nb = len(L.bucket_starts)
    assert same_entries(L.cells, cells, nb) and same_entries(L.plist, plist, nb)
    if order == 4:
        assert same_entries(L.softcells, soft, nb)
