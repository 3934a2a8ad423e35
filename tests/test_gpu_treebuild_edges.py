"""The GPU tree build at the edges of its tiles against the host build, bit
for bit: particle counts around the sort's and the level kernels' tiles,
buckets from 1 to more than all particles (and around the largest whose
windows are kept in shared memory), node counts beyond the first allocation
(chains of single-child nodes), coincident and massless particles."""
import numpy as np
import pytest

from changa_gb300 import tree
from changa_gb300.gputree import DeviceTree

pytestmark = pytest.mark.gpu


def particles(kind, n):
    rng = np.random.default_rng(n + len(kind))
    if kind == "uniform":
        pos = rng.uniform(-1, 1, (n, 3))
    elif kind == "pairs":  # each pair shares almost every key bit
        pos = np.repeat(rng.uniform(0, 1, ((n + 1) // 2, 3)), 2, axis=0)[:n]
        pos[1::2] += 1.5e-6
    elif kind == "coincident":
        pos = rng.uniform(-1, 1, (n, 3))
        pos[n // 4:n // 2] = pos[0]
    else:  # a clump far from the origin and one distant particle
        pos = 1e3 + rng.normal(0, 1e-3, (n, 3))
        pos[-1] = 2e3
    mass = np.full(n, 1.0 / n)
    if kind == "uniform" and n > 4:
        mass[rng.integers(0, n, n // 4)] = 0.0
    return pos, mass, rng.uniform(1e-3, 1e-2, n)


@pytest.mark.parametrize("kind", ["uniform", "pairs", "coincident", "clump"])
@pytest.mark.parametrize("n,n_bucket", [
    (1, 1), (2, 1), (3, 2), (31, 8), (255, 1), (256, 12), (1023, 16), (1024, 5), (1025, 32),
    (2047, 1), (2048, 16), (2049, 64), (4097, 512), (5000, 511), (5000, 513), (5000, 4999),
    (5000, 5000), (5000, 7000), (70001, 12), (70001, 1000)])
def test_treebuild_edges(cuda_ok, kind, n, n_bucket):
    import torch
    pos, mass, soft = particles(kind, n)
    L = tree.build_lists(pos, mass, soft, n_bucket=n_bucket, theta=0.9)
    T = DeviceTree(*(torch.from_numpy(a).cuda() for a in (pos, mass, soft)), n_bucket=n_bucket,
                   theta=0.9)
    try:
        assert T.n_nodes == L.moments.shape[0] and T.n_buckets == len(L.bucket_starts)
        for got, want in ((T.perm, L.perm), (T.parts, L.parts), (T.moments, L.moments),
                          *((T.meta[k], L.meta[k]) for k in ("node_info", "parent", "bucket_node",
                                                             "leaf", "node_bbox", "node_geom"))):
            np.testing.assert_array_equal(got.cpu().numpy(), want)
    finally:
        T.close()
