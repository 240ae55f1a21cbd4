"""FP64 distances to needle-like triangles and to very small meshes, whose FP32 distances and squares are
poor: the search's FP32 radius and candidate tests must not decide the result.  Calls that search point by
point and calls that search in packets, against the exhaustive FP64 search of the same faces."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import FlatMeshSDF, MeshSDF, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _needles(width, offset, n=6000):
    rng = np.random.default_rng(0)

    def unit(x):
        return x / np.linalg.norm(x, axis=1, keepdims=True)

    c = rng.uniform(-1, 1, (n, 3))
    d = unit(rng.normal(size=(n, 3)))
    e = unit(np.cross(d, rng.normal(size=(n, 3))))
    t = rng.uniform(0, 1, (n, 1))
    x = np.stack([c - d * 0.5, c + d * 0.5, c + d * (t - 0.5) + e * width], 1) + offset
    return x.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


@pytest.mark.parametrize("n", [3000, 70001])
@pytest.mark.parametrize("name", ["needle1e-5", "needle1e-7", "needle1e-7 off", "needle1e-9", "tiny1e-20", "tiny1e-25"])
def test_fp64_against_exhaustive(name, n):
    if name.startswith("needle"):
        v, f = _needles(float(name[6:10]), 100.0 if name.endswith("off") else 0.0)
    else:
        v, f = W.displaced_icosphere(4, 5)
        v = v * float(name[4:])
    lo, hi = v.min(0), v.max(0)
    size = (hi - lo).max()
    rng = np.random.default_rng(n)
    p = (lo + hi) / 2 + rng.uniform(-1, 1, (n, 3)) * size
    p[::7] = v[rng.integers(0, len(v), p[::7].shape[0])] + rng.normal(size=p[::7].shape) * 1e-4 * size
    pd = torch.from_numpy(p).cuda()
    ref = FlatMeshSDF(v, f).signed_distance(pd).abs()
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    d = MeshSDF(v, f).signed_distance(pd, closest_tri=tri)[0].abs()
    # the same faces by the same function: the least of the same values, up to the rounding of the squares
    # by which the exhaustive search compares them (a few eps of the coordinates)
    assert ((d - ref).abs() <= 1e-14 * (np.abs(v).max() + size) + 1e-13 * ref).all()
    assert (tri >= 0).all()
    # (the triangle test rounds the in-plane offsets of a needle by eps / width)
    width = float(name[6:10]) if name.startswith("needle") else 1.0
    t = TriMeshSDF(v, f).signed_distance(pd).abs()
    assert ((t - ref).abs() <= (np.abs(v).max() + size) * 1e-14 / width).all()


@pytest.mark.parametrize("n", [3000, 70001])
@pytest.mark.parametrize("scale", [1e-20, 1e-25])
def test_fp32_of_tiny_meshes_finds_a_triangle(scale, n):
    """FP32 squares of these distances underflow: every point still gets the distance of some triangle near
    it, within the distance to the farthest corner of the mesh's box."""
    v, f = W.displaced_icosphere(5, 5)
    m = TriMeshSDF(v * scale, f)
    for reach in (1.5, 1e4):
        p = torch.from_numpy((W.uniform_points(n, n, -reach, reach) * np.float32(scale)).astype(np.float32)).cuda()
        d = m.signed_distance(p)
        m.check_status()
        assert (d.abs() <= 1.001 * (p.double().norm(dim=1) + 2.0 * scale) + 2e-23).all()


@pytest.mark.parametrize("n", [3000, 70001])
def test_fp64_of_a_tiny_mesh_from_afar(n):
    """Squared distances of 1e-44 have one digit in FP32: the FP64 result must not depend on them."""
    v, f = W.displaced_icosphere(4, 5)
    v = v * 1e-25
    rng = np.random.default_rng(n)
    u = rng.normal(size=(n, 3))
    p = torch.from_numpy(u / np.linalg.norm(u, axis=1, keepdims=True) * 10.0 ** rng.uniform(-25, -19, (n, 1))).cuda()
    ref = FlatMeshSDF(v, f).signed_distance(p).abs()
    for cls in (MeshSDF, TriMeshSDF):
        d = cls(v, f).signed_distance(p).abs()
        assert ((d - ref).abs() <= 1e-14 * (1e-25 + ref)).all()
