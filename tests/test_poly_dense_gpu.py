"""Polygon leaves that most queries of a packet need: every lane evaluates its own faces, with the values and faces
of the search that takes four lanes a pair (which a point alone takes), and on planar faces of the exhaustive
search."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import PolygonFlatMeshSDF, PolygonMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [1, 4, 32])
@pytest.mark.parametrize("name", ["prism3", "prism40", "tris"])
def test_dense_packets(name, leaf):
    if name == "tris":
        v, f = W.displaced_icosphere(3, 4)
        faces = (np.arange(f.shape[0] + 1, dtype=np.int64) * 3, f.ravel())
    else:
        v, faces = W.polygon_prism(int(name[5:]), 0.8, 1.5)
    m = PolygonMeshSDF(v, faces, leaf_size=leaf)
    rng = np.random.default_rng(leaf)
    # packets of 32 points at one place, near the surface: all of them need the same leaves
    at = v[rng.integers(0, len(v), 300)]
    p = (np.repeat(at, 32, axis=0) + rng.normal(size=(9600, 3)) * 1e-4)
    pd = torch.from_numpy(p).cuda()
    f = torch.empty(9600, dtype=torch.int32, device="cuda")
    d = m.signed_distance(pd, closest_face=f)[0]
    m.check_status()
    ref = np.abs(PolygonFlatMeshSDF(v, faces).signed_distance(p))
    assert np.abs(np.abs(d.cpu().numpy()) - ref).max() <= 16 * 2.3e-16 * 4
    g = torch.empty(1, dtype=torch.int32, device="cuda")
    for i in range(0, 9600, 331):
        e = m.signed_distance(pd[i:i + 1].contiguous(), closest_face=g)[0]
        assert torch.equal(e.abs(), d[i:i + 1].abs())
