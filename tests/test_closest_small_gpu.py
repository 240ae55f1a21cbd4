"""FP32 closest triangles of calls of every size are the packet walk's, tied triangles included: points at
vertices and edges (where several triangles are equally near) and far away (where FP32 cannot tell them apart).
node_width=4 asks for the walk itself."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1000, 20000, 65536, 65537])
@pytest.mark.parametrize("level,stretch", [(3, 1.0), (5, 1.0), (5, 1e-3)])
def test_same_triangle_as_the_walk(level, stretch, n):
    v, f = W.displaced_icosphere(level, 5)
    v = v * [1.0, stretch, stretch]
    m = TriMeshSDF(v, f)
    rng = np.random.default_rng(n)
    mid = 0.5 * (v[f[:, 0]] + v[f[:, 1]])
    far = W.uniform_points(n, 2) * 10.0 ** rng.uniform(0, 6, (n, 1))
    p = np.concatenate([v[rng.integers(0, len(v), n)], mid[rng.integers(0, len(mid), n)], far])
    pd = torch.from_numpy(p[rng.permutation(len(p))[:n]].astype(np.float32)).cuda()
    for band in (True, False):
        a, b = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
        d = m.signed_distance(pd, closest_tri=a, fp64_band=band)[0]
        e = m.signed_distance(pd, closest_tri=b, fp64_band=band, node_width=4)[0]
        m.check_status()
        assert torch.equal(a, b) and torch.equal(d, e)
        # and the host call
        t = np.empty(n, np.int32)
        h = m.signed_distance(pd.cpu().numpy(), closest_tri=t, fp64_band=band)[0]
        assert np.array_equal(t, a.cpu().numpy()) and np.array_equal(h, d.cpu().numpy())
