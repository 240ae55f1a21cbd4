"""Polygon-face distance of points whose squared distance overflows FP32 (|p| above 1.8e19): every face
counts there, so the magnitude and the tie rule are the exhaustive evaluation's.

Every face is then evaluated for every point, so the value is no farther than the exhaustive search's, and of
faces at the same distance the lowest in leaf order wins whatever other points share the packet."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import PolygonFlatMeshSDF, PolygonMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e15, 1e18])
@pytest.mark.parametrize("name", ["prism40", "quad24"])
def test_points_beyond_the_square_root_of_flt_max(name, scale):
    v, faces = W.polygon_prism(40, 0.8, 1.5) if name == "prism40" else W.displaced_quad_sphere(24, 7)
    m = PolygonMeshSDF(v * scale, faces)
    rng = np.random.default_rng(4)
    u = rng.normal(size=(3000, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    p = u * 10.0 ** rng.uniform(19.4, 25, (3000, 1))
    f = torch.empty(3000, dtype=torch.int32, device="cuda")
    d = m.signed_distance(torch.from_numpy(p).cuda(), closest_face=f)[0].cpu().numpy()
    m.check_status()
    ref = PolygonFlatMeshSDF(v * scale, faces).signed_distance(p)
    # faces off their plane by h return as much less than their distance (h below 2 % of the scale)
    off = 0.02 * scale if name == "quad24" else 0.0
    assert np.all(np.abs(d) <= np.abs(ref) * (1 + 1e-15) + off)
    perm = rng.permutation(3000)
    g = torch.empty(3000, dtype=torch.int32, device="cuda")
    e = m.signed_distance(torch.from_numpy(p[perm]).cuda(), closest_face=g)[0].cpu().numpy()
    assert np.array_equal(e, d[perm]) and np.array_equal(g.cpu().numpy(), f.cpu().numpy()[perm])
