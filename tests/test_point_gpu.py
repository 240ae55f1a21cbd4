"""The one-warp-per-point search (calls of few points) against the packet traversal, which the
counters entry point always runs, and against the exhaustive FP64 restatement.

Sizes: the smallest mesh (its root is a leaf), leaves of 1 and of the largest size, a deep tree; 1 point,
partial blocks, and the two sizes on either side of the call limit."""
import numpy as np
import pytest
import torch

import oracle
from ebgeometry_b200 import MeshSDF, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu

LIMIT = 65536  # points of the largest call that takes the search (POINT_CALL)


def _mesh(name):
    if name == "tetra":
        v = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], np.float64) * 0.7
        return v, np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]], np.int32)
    return W.displaced_icosphere(int(name[1:]), 5)


@pytest.mark.parametrize("name,leaf,n", [("tetra", 8, 1), ("tetra", 1, 33), ("l2", 32, 5), ("l2", 1, 1000),
                                         ("l4", 8, 4099), ("l4", 8, LIMIT), ("l4", 8, LIMIT + 1), ("l7", 8, 2000)])
def test_search_equals_packets_and_brute_force(name, leaf, n):
    v, f = _mesh(name)
    m = TriMeshSDF(v, f, leaf_size=leaf)
    # everywhere, near the surface (the FP64 band), at vertices, at the centre (all triangles tie nearly)
    p = np.concatenate([W.uniform_points(n, n), W.band_points(v, f, n, n + 1), v[:n].astype(np.float32),
                        np.zeros((1, 3), np.float32)])
    p = p[np.random.default_rng(n).permutation(p.shape[0])[:n]]
    pd = torch.from_numpy(p).cuda()
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    d, _ = m.signed_distance(pd, closest_tri=tri)
    d_pk, _ = m.stats(pd)
    m.check_status()
    assert torch.equal(d, d_pk)
    # FP64 points: the same values as the exhaustive search, up to which of two tied triangles won
    k = min(n, 1500)
    p64 = p[:k].astype(np.float64) + 1e-9
    d_ref, _ = oracle.port().mesh_sdf_brute(v, f, p64)
    for cls in (TriMeshSDF, MeshSDF):
        mm = m if cls is TriMeshSDF else MeshSDF(v, f, leaf_size=leaf)
        d64 = mm.signed_distance(torch.from_numpy(p64).cuda()).cpu().numpy()
        mm.check_status()
        # (the DCEL face rounds differently from the triangle test the oracle runs)
        assert np.abs(d64 - d_ref).max() <= (1e-12 if cls is TriMeshSDF else 1e-11) * m.diagonal


def test_far_and_non_finite_points():
    v, f = _mesh("l3")
    m = TriMeshSDF(v, f)
    p = np.array([[1e25, 0, 0], [50.0, -70.0, 1e3], [0.2, 0.1, 0.0]], np.float32)
    d_pk, _ = m.stats(torch.from_numpy(p).cuda())
    assert torch.equal(m.signed_distance(torch.from_numpy(p).cuda()), d_pk)
    m.check_status()
    for bad in (np.nan, np.inf):
        q = p.copy()
        q[1, 2] = bad
        d = m.signed_distance(torch.from_numpy(q).cuda())
        assert torch.equal(d[[0, 2]], d_pk[[0, 2]])
        with pytest.raises(Exception):
            m.check_status()
