"""The FP64 form's reciprocal square root, read off the potential of single
pairs: one target at the origin, one source of mass 1 at (x, 0, 0), both
without softening, whose potential is -1/sqrt(x^2) with x^2 rounded once."""
import ctypes as C

import numpy as np
import pytest

from changa_gb300 import _native as N

pytestmark = pytest.mark.gpu


def test_reciprocal_root_over_the_exponents(cuda_ok):
    """Every binary exponent of x from 2^-48 to 2^60 (x^2 over 217 of them),
    mantissas at random and next to the powers of two.  The series is cut
    below 2^-58; x y, e and the final sum round to 2^-53 each, the first two
    halved: at most 2^-52 of the root."""
    import torch
    rng = np.random.default_rng(1)
    man = np.concatenate([rng.uniform(1, 2, 180), [1.0, np.sqrt(2.0), 1.5],
                          1 + 2.0 ** -52 * np.arange(1, 9), 2 - 2.0 ** -52 * np.arange(1, 9)])
    x = (man[:, None] * 2.0 ** np.arange(-48, 61)[None]).ravel()
    n = len(x)
    targets = np.zeros((n, 5))
    sources = np.zeros((n, 5))
    sources[:, 0], sources[:, 2] = 1.0, x
    here = (3 | 3 << 3 | 3 << 6) << 22
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
         (np.stack([np.arange(n), np.full(n, here)], 1).astype(np.int32),
          np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), np.ones(n, np.int32),
          sources, targets)]
    r = N.ChangaListRequest()
    r.list, r.markers, r.starts, r.sizes = (a.data_ptr() for a in t[:4])
    r.n_buckets, r.n_entries = n, n
    v = torch.zeros((n, 5), dtype=torch.float64, device="cuda")
    N.check(N.cuda_lib().changa_part_forces_fp64(
        t[4].data_ptr(), n, t[5].data_ptr(), n, C.byref(r), 0.0, v.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    root = 1 / np.sqrt((x * x).astype(np.longdouble))
    err = np.abs(-v[:, 3].cpu().numpy() - root) / root
    assert err.max() <= 2.0 ** -52, float(err.max())
