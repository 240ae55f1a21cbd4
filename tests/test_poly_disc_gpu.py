"""The disc bounds of the polygon-face search: with planar faces its result is the exhaustive search's,
bit for bit (no face returns less than the distance to its box); with faces off their plane by at
most h it is within 2 h of it.  Faces of 3 to 129 vertices, leaves of 1 to 32 faces, one point to several
packets, points near, far and inside."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import PolygonFlatMeshSDF, PolygonMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _mesh(name):
    if name.startswith("prism"):
        return W.polygon_prism(int(name[5:]), 0.8, 1.5)
    if name == "tris":
        v, f = W.displaced_icosphere(3, 4)
        return v, (np.arange(f.shape[0] + 1, dtype=np.int64) * 3, f.ravel())
    return W.displaced_quad_sphere(int(name[4:]), 7)


def _off_plane(m):
    """The largest distance of a corner from its face's plane."""
    v, (off, idx), obj = m
    fn, c, _, _ = obj.normals()
    face = np.repeat(np.arange(off.size - 1), np.diff(off))
    return np.abs(((v[idx] - c[face]) * fn[face]).sum(1)).max()


@pytest.mark.parametrize("name,leaf,n", [("prism3", 4, 1), ("prism40", 1, 3000), ("prism129", 32, 2049), ("tris", 4, 20001),
                                         ("tris", 32, 33), ("quad12", 4, 5000), ("quad24", 1, 4097)])
@pytest.mark.parametrize("build", ["SAH", "Morton"])
def test_search_against_exhaustive(name, leaf, n, build):
    v, faces = _mesh(name)
    m = PolygonMeshSDF(v, faces, build=build, leaf_size=leaf)
    rng = np.random.default_rng(n)
    p = np.concatenate([rng.uniform(-1.6, 1.6, (n, 3)), rng.normal(0, 40, (n, 3)), v[rng.integers(0, len(v), n)] +
                        rng.normal(0, 1e-4, (n, 3))])[rng.permutation(3 * n)[:n]]
    pd = torch.from_numpy(p).cuda()
    d = m.signed_distance(pd).cpu().numpy()
    m.check_status()
    ref = PolygonFlatMeshSDF(v, faces).signed_distance(p)
    if name.startswith("quad"):
        h = _off_plane((v, faces, m))
        assert np.abs(np.abs(d) - np.abs(ref)).max() <= 2 * h
    else:
        # a face value is the distance to the face up to its own rounding: 16 eps of the coordinates
        assert np.abs(np.abs(d) - np.abs(ref)).max() <= 16 * 2.3e-16 * (np.abs(p).max() + 2)
        assert np.mean(d == ref) > 0.999
