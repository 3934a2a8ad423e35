"""The replicas that the FP64 Ewald term culls in FP32 must lie beyond the cut,
also where the cut is small against the offsets that FP32 rounds."""
import ctypes as C

import numpy as np
import pytest

import oracle
from changa_gb300 import _native as N
from changa_gb300 import gravity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [0.7, 1.0, 3e-5])
@pytest.mark.parametrize("cut", [1e-4, 3e-3, 0.4])
def test_replica_just_inside_the_cut(cuda_ok, cut, L):
    """Each warp's 32 particles at one place, a box length less a little from
    the root's centre, so that the first replica (not in the hole, n_rep 0) is
    within a few 1e-4 of the cut; its term is of the order of the others."""
    import torch
    rng = np.random.default_rng(3)
    n = 3008
    parts = np.zeros((n, 5))
    parts[:, 0] = 1.0 / n
    parts[:, 2] = (L * (1 - cut * (1 - rng.uniform(1e-5, 4e-4, n // 32)))).repeat(32)
    root = np.zeros(12)
    root[0], root[2] = 0.8 * L, 1.0
    ref = oracle.ewald_forces(parts, root, L, 0, cut, 2.8)
    p = gravity.EwaldConfig(L, 0, cut, 2.8).params(root)
    dp = torch.from_numpy(parts).cuda()
    v = torch.zeros((n, 5), dtype=torch.float64, device="cuda")
    N.check(N.cuda_lib().changa_ewald_forces(N.CHANGA_FORM_FP64, dp.data_ptr(), n, None, n,
                                             C.byref(p), v.data_ptr(),
                                             torch.cuda.current_stream().cuda_stream))
    # the recursion of the g_n near the root loses up to (4 x 1.2e-3)^-3 of
    # 2^-53 of terms of size 1 / L
    v = v.cpu().numpy()
    assert np.abs(v[:, 3] - ref[:, 3]).max() * L < 1e-8
    assert np.abs(v[:, :3] - ref[:, :3]).max() * L * L < 1e-8
