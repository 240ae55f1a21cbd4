"""The ways a union's mesh is searched -- for a packet together, or for one query after the other -- and the
packet sizes (1 to 32 queries, by the call's size) give the same values: a large call against its pieces
and against brute force.  Points packed around the meshes, far from them, inside them, and single points."""
import numpy as np
import pytest
import torch

import oracle
from ebgeometry_b200 import BVHUnion, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spheres", [0, 1, 400])
def test_large_call_equals_its_pieces_and_brute_force(spheres):
    sc = W.csg_scene(7, n_spheres=400, n_meshes=9, levels=(1, 5), mesh_radius=(0.02, 0.4))
    tms = [TriMeshSDF(v, f) for v, f in sc["meshes"]]
    sp = sc["spheres"][:spheres]
    u = BVHUnion(sp if spheres else None, tms, sc["poses"])
    p = np.concatenate([W.uniform_points(150000, 6, -1.3, 1.3), W.uniform_points(50000, 8, -30.0, 30.0)] +
                       [sc["poses"][i, 2:5].astype(np.float32) + W.uniform_points(12000, 9 + i, -0.1, 0.1)
                        for i in range(len(sc["poses"]))])
    q = torch.from_numpy(np.ascontiguousarray(p, np.float32)).cuda()
    d = u.values(q)
    n = q.shape[0]
    # (pieces of other sizes are other packets; the FP32 nearest triangle and the FP64 band are the same)
    for b, e in ((0, 1), (1, 34), (34, 5011), (5011, 60000), (150000, 180000), (n - 70000, n)):
        assert torch.equal(u.values(q[b:e].contiguous()), d[b:e])
    assert torch.equal(u.values(q[:9000].contiguous(), sort=False), d[:9000])
    u.check_status()
    s = np.concatenate([np.arange(0, n, 211), np.arange(n - 500, n)])
    ref = oracle.port().scene_brute(np.asarray(sp).reshape(-1, 4), sc["meshes"], sc["poses"], p[s].astype(np.float64))
    got = d.cpu().numpy()[s].astype(np.float64)
    # the scene's diagonal is about 5, the far points' about 104: 1e-6 of each
    assert np.all(np.abs(got - ref) <= 1e-6 * np.where(np.abs(p[s]).max(1) > 1.5, 104.0, 5.0))
    clear = np.abs(ref) > 1e-4 * 5.0
    assert np.all(np.sign(got[clear]) == np.sign(ref[clear]))
    assert spheres or np.any(got < 0)
