"""Meshes far from the origin, where the FP32 bounds of every search lean on their allowance for rounding: calls
that search point by point and in packets, FP32 and FP64, against the exhaustive FP64 search; and the union of
such meshes."""
import numpy as np
import pytest
import torch

import oracle
from ebgeometry_b200 import BVHUnion, FlatMeshSDF, MeshSDF, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 70001])
@pytest.mark.parametrize("offset", [[10.0, -20.0, 5.0], [1000.0, -500.0, 2000.0], [1e6, 0.0, -3e5]])
def test_distances_off_the_origin(offset, n):
    v, f = W.displaced_icosphere(5, 5)
    v = v + offset
    far = np.abs(v).max()
    p = np.concatenate([W.uniform_points(n, n), W.band_points(*W.displaced_icosphere(5, 5), n, n + 1)])
    p = (p.astype(np.float64) + offset)[np.random.default_rng(n).permutation(2 * n)[:n]]
    p64 = torch.from_numpy(p).cuda()
    ref = FlatMeshSDF(v, f).signed_distance(p64)
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    for cls in (TriMeshSDF, MeshSDF):
        m = cls(v, f)
        d, _ = m.signed_distance(p64, closest_tri=tri)
        m.check_status()
        # the same triangle's FP64 distance, its differences of coordinates rounded to eps of them
        assert ((d - ref).abs() <= 32 * 2.3e-16 * far).all() and (tri >= 0).all()
    m = TriMeshSDF(v, f)
    p32 = p64.float()
    ref = FlatMeshSDF(v, f).signed_distance(p32.double())
    d = m.signed_distance(p32)
    m.check_status()
    # the error scale of the FP32 pass is the larger of the diagonal and the coordinates; the library's
    # allowance is 2e-6 of it and a face distance takes the errors of three coordinates
    scale = max(m.diagonal, far)
    assert ((d.double() - ref).abs() <= 4e-6 * scale).all()
    clear = ref.abs() > 1e-4 * scale
    assert (torch.sign(d[clear]) == torch.sign(ref[clear])).all()


def test_union_off_the_origin():
    sc = W.csg_scene(7, n_spheres=20, n_meshes=6, levels=(2, 4), mesh_radius=(0.1, 0.4))
    off = np.array([300.0, -200.0, 100.0])
    sp = sc["spheres"].copy()
    sp[:, :3] += off
    poses = sc["poses"].copy()
    poses[:, 2:5] += off
    u = BVHUnion(sp, [TriMeshSDF(v, f) for v, f in sc["meshes"]], poses)
    p = (W.uniform_points(40000, 3, -1.3, 1.3).astype(np.float64) + off).astype(np.float32)
    d = u.values(torch.from_numpy(p).cuda()).cpu().numpy()
    u.check_status()
    ref = oracle.port().scene_brute(sp, sc["meshes"], poses, p[:3000].astype(np.float64))
    # FP32 coordinates of 300 round by 1.8e-5; the local point takes three of them and a rotation
    assert np.abs(d[:3000] - ref).max() <= 4e-6 * 600
