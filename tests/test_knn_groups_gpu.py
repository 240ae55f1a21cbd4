"""The two k-NN walks of the point cloud -- four lanes per query (calls of at most LANES queries, and every
k above 8) and one lane per query -- give the same neighbours: a large call against its pieces, and
a sample against brute force.  k at the edges of the lists kept per lane; clouds that are one leaf, one
node, duplicates; the piece sizes that end in the middle of a warp's run."""
import numpy as np
import pytest
import torch

import oracle
from ebgeometry_b200 import PointCloudBVH
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu

LANES = 262144


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("cloud", ["clustered", "leaf", "node", "copies"])
def test_large_call_equals_its_pieces_and_brute_force(cloud, k):
    pts = {"clustered": lambda: W.point_cloud(50000, 3), "leaf": lambda: W.point_cloud(5, 3),
           "node": lambda: W.point_cloud(33, 3), "copies": lambda: np.repeat(W.point_cloud(40, 3), 37, axis=0)}[cloud]()
    n = LANES + 1 + 32 * 3
    q = W.uniform_points(n, k, -0.1, 1.1)
    q[::97] = pts[np.arange(q[::97].shape[0]) % len(pts)]  # exact hits
    c = PointCloudBVH(pts)
    qd = torch.from_numpy(q).cuda()
    idx, d2 = c.knn(qd, k)
    for b, e in ((0, 1), (1, 8), (8, 2009), (2009, n - 123456), (n - 123456, n)):
        i, d = c.knn(qd[b:e].contiguous(), k)
        assert torch.equal(i, idx[b:e]) and torch.equal(d, d2[b:e])
    c.check_status()
    s = np.arange(0, n, 1009)
    ri, rd = oracle.port().knn_brute(pts, q[s], k)
    assert np.array_equal(idx.cpu().numpy()[s], ri) and np.array_equal(d2.cpu().numpy()[s], rd)


@pytest.mark.parametrize("k", [1, 4, 8, 12, 32])
def test_self_queries(k):
    pts = W.point_cloud(LANES + 3000, 5)
    c = PointCloudBVH(pts)
    idx, d2 = c.all_nearest_neighbors(k, device=True)
    ids = torch.arange(0, pts.shape[0], 17, device="cuda")
    i, d = c.nearest_neighbors(ids, k)
    c.check_status()
    assert torch.equal(i, idx[ids]) and torch.equal(d, d2[ids])
    small = PointCloudBVH(pts[:3000])
    i, d = small.all_nearest_neighbors(k)
    ri, rd = oracle.port().knn_brute_self(pts[:3000], k)
    assert np.array_equal(i, ri) and np.array_equal(d, rd)
