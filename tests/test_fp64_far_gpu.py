"""FP64 calls write every result: a point that is not finite, or so far that its squared distance overflows
FP32, gets FLT_MAX and triangle -1 in calls of every size (large calls left its place as it was)."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import EbgError, MeshSDF, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cls", [TriMeshSDF, MeshSDF])
@pytest.mark.parametrize("level,n", [(3, 1000), (3, 70001), (5, 1000), (5, 70001)])
def test_every_result_is_written(cls, level, n):
    v, f = W.displaced_icosphere(level, 5)
    m = cls(v, f)
    p = W.uniform_points(n, 3).astype(np.float64)
    rng = np.random.default_rng(n)
    far = rng.choice(n, 60, replace=False)
    p[far[:30]] *= 1e25
    p[far[30:], 1] = np.where(np.arange(30) % 2, np.nan, np.inf)
    pd = torch.from_numpy(p).cuda()
    # what the results' memory held before must not show: fill it, free it, and let the call take it
    junk = [torch.full((n,), 7.5, dtype=torch.float64, device="cuda") for _ in range(8)]
    del junk
    tri = torch.full((n,), 12345, dtype=torch.int32, device="cuda")
    d, _ = m.signed_distance(pd, closest_tri=tri)
    with pytest.raises(EbgError):
        m.check_status()
    d, tri = d.cpu().numpy(), tri.cpu().numpy()
    assert np.all(d[far] == np.finfo(np.float32).max) and np.all(tri[far] == -1)
    near = np.ones(n, bool)
    near[far] = False
    assert np.all(np.abs(d[near]) < 10) and np.all(tri[near] >= 0)
