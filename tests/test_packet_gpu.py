"""The FP32 search by packet boxes against the packet walk, which the counters entry point always runs:
the same distances bit for bit, for dense, sparse and clustered points, ragged sizes, unordered calls,
points far away or not finite inside a packet, leaves of any size, and an attached model."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import EbgError, MeshSDF, SeedModel, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu

LIMIT = 65536  # larger calls take packets


def _points(kind, v, f, n):
    if kind == "grid":
        return W.grid_points(round(n ** (1 / 3)) + 1)[:n]
    if kind == "near":
        return W.band_points(v, f, n, 3)
    if kind == "centre":  # near the medial axis: everything is about equally far
        return W.uniform_points(n, 4, -0.05, 0.05)
    if kind == "pairs":  # runs of neighbours that jump between far places inside a packet
        p = np.repeat(W.uniform_points(n // 5 + 1, 5), 5, axis=0)[:n]
        return (p + W.uniform_points(n, 6, -1e-3, 1e-3)).astype(np.float32)
    if kind == "same":
        return np.full((n, 3), 0.3, np.float32)
    return W.uniform_points(n, 7)


@pytest.mark.parametrize("level,leaf,kind,n", [
    (5, 8, "uniform", LIMIT + 1), (5, 8, "grid", 300007), (5, 1, "near", 100031), (5, 32, "uniform", 70001),
    (5, 8, "centre", 70003), (6, 8, "pairs", 200001), (5, 8, "same", 66000), (7, 8, "uniform", 150001),
    (7, 12, "grid", 1000003)])
def test_packet_boxes_equal_the_walk(level, leaf, kind, n):
    v, f = W.displaced_icosphere(level, 9)
    m = TriMeshSDF(v, f, leaf_size=leaf, build="Morton" if level == 7 else "SAH", on_device=level == 7)
    p = torch.from_numpy(np.ascontiguousarray(_points(kind, v, f, n))).cuda()
    d_walk, _ = m.stats(p)
    for sort in (True, False) if n < 100000 and kind != "centre" else (True,):
        d = m.signed_distance(p, sort=sort)
        m.check_status()
        assert torch.equal(d, d_walk), (kind, sort)


def test_far_and_non_finite_points_in_packets():
    v, f = W.displaced_icosphere(5, 9)
    m = TriMeshSDF(v, f)
    p = W.uniform_points(80000, 2)
    rng = np.random.default_rng(1)
    far = rng.choice(80000, 300, replace=False)
    p[far] *= rng.choice([1e3, 1e13, 1e25], 300)[:, None].astype(np.float32)
    pd = torch.from_numpy(p).cuda()
    d_walk, _ = m.stats(pd)
    assert torch.equal(m.signed_distance(pd), d_walk)
    m.check_status()
    bad = rng.choice(80000, 50, replace=False)
    p[bad, 1] = np.where(np.arange(50) % 2, np.nan, np.inf)
    pd = torch.from_numpy(p).cuda()
    d = m.signed_distance(pd).cpu().numpy()
    with pytest.raises(EbgError):
        m.check_status()
    ok = np.ones(80000, bool)
    ok[bad] = False
    assert np.array_equal(d[ok], d_walk.cpu().numpy()[ok])


def test_attached_model_and_refit():
    v, f = W.displaced_icosphere(5, 9)
    m = TriMeshSDF(v, f)
    seed = SeedModel.create(lo=[-1.2] * 3, hi=[1.2] * 3, log2_table=12)
    m.attach_seed(seed, cells_per_axis=24, radius_mode=1)
    p = torch.from_numpy(np.concatenate([W.uniform_points(60000, 3), W.grid_points(50)])).cuda()  # some outside the cells
    d_walk, _ = m.stats(p)
    assert torch.equal(m.signed_distance(p, seed=seed), d_walk)
    m.refit(W.displaced_icosphere(5, 10)[0])
    d_walk, _ = m.stats(p)
    assert torch.equal(m.signed_distance(p), d_walk)
    m.check_status()


@pytest.mark.parametrize("cls", [TriMeshSDF, MeshSDF])
@pytest.mark.parametrize("level,leaf,kind,n", [(5, 8, "uniform", 70001), (5, 32, "near", 131073), (6, 1, "grid", 100033),
                                               (5, 8, "centre", 66001), (3, 8, "pairs", 65537), (5, 8, "same", 65568)])
def test_fp64_pass_in_packets_equals_point_by_point(cls, level, leaf, kind, n):
    """Calls of at most LIMIT points search point by point (tested against the exhaustive oracle);
    a larger one takes the packets of the FP64 pass and the groups that they leave points to."""
    v, f = W.displaced_icosphere(level, 9)
    m = cls(v, f, leaf_size=leaf)
    p = torch.from_numpy(_points(kind, v, f, n).astype(np.float64) + 1e-9).cuda()
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    d = m.signed_distance(p, closest_tri=tri)[0].clone()
    m.check_status()
    for b in range(0, n, LIMIT):
        t = torch.empty(min(LIMIT, n - b), dtype=torch.int32, device="cuda")
        part = m.signed_distance(p[b:b + LIMIT].contiguous(), closest_tri=t)[0]
        assert torch.equal(d[b:b + LIMIT], part) and torch.equal(tri[b:b + LIMIT], t)
