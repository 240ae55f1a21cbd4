"""The routes of the grid k-NN -- one launch or two (calls of SPLIT queries and more, and every k above 8),
queries in the caller's order or in Morton order (calls above ORDERED) -- give the same neighbours: a large
call against its pieces, and a sample against brute force.  Clouds whose cells hold a point, many points or
one point many times, flat and empty clouds; queries outside the cloud; k beyond the cloud's size."""
import numpy as np
import pytest
import torch

import oracle
from ebgeometry_b200 import PointCloudHashGrid
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu

SPLIT = 1 << 18
ORDERED = 1 << 20
CLOUDS = {"uniform": lambda: W.uniform_points(30000, 3, 0.0, 1.0), "clustered": lambda: W.point_cloud(30000, 3),
          "copies": lambda: np.repeat(W.point_cloud(40, 3), 37, axis=0), "few": lambda: W.point_cloud(5, 3),
          "flat": lambda: W.uniform_points(9000, 3, 0.0, 1.0) * np.array([1, 1, 0], np.float32)}


@pytest.mark.parametrize("k", [1, 2, 3, 4, 7, 8, 9, 16, 31, 32])
@pytest.mark.parametrize("cloud", list(CLOUDS))
def test_large_call_equals_its_pieces_and_brute_force(cloud, k):
    pts = CLOUDS[cloud]()
    n = SPLIT + 1 + 32 * 3
    q = W.uniform_points(n, k, -0.3, 1.3)
    q[::97] = pts[np.arange(q[::97].shape[0]) % len(pts)]  # exact hits
    q[5::3001] *= 1.0e4  # far outside
    g = PointCloudHashGrid(pts)
    qd = torch.from_numpy(q).cuda()
    idx, d2 = g.knn(qd, k)
    for b, e in ((0, 1), (1, 8), (8, 2009), (2009, n - 123456), (n - 123456, n)):
        i, d = g.knn(qd[b:e].contiguous(), k)
        assert torch.equal(i, idx[b:e]) and torch.equal(d, d2[b:e])
    g.check_status()
    s = np.arange(0, n, 1009)
    ri, rd = oracle.port().knn_brute(pts, q[s], k)
    assert np.array_equal(idx.cpu().numpy()[s], ri) and np.array_equal(d2.cpu().numpy()[s], rd)


@pytest.mark.parametrize("k", [1, 4, 12])
def test_ordered_call_and_self_queries(k):
    pts = W.uniform_points(SPLIT + 3000, 5, 0.0, 1.0)
    g = PointCloudHashGrid(pts)
    q = torch.from_numpy(W.uniform_points(ORDERED + 77, 7, -0.1, 1.1)).cuda()
    idx, d2 = g.knn(q, k)
    i, d = g.knn(q[-50000:].contiguous(), k)
    assert torch.equal(i, idx[-50000:]) and torch.equal(d, d2[-50000:])
    idx, d2 = g.all_nearest_neighbors(k, device=True)
    ids = np.arange(0, pts.shape[0], 17)
    i, d = g.nearest_neighbors(ids, k)
    g.check_status()
    assert np.array_equal(i, idx.cpu().numpy()[ids]) and np.array_equal(d, d2.cpu().numpy()[ids])
