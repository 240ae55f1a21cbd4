"""The autotuner's launch shape is the packet walk's: on a mesh whose plain calls do not take the walk, calls that
do (FP32 closest triangles) are as fast with the tuned defaults as with the best shape given by hand."""
import pytest
import torch

from ebgeometry_b200 import TriMeshSDF, _capi
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_tuned_shape_is_the_walks():
    v, f = W.displaced_icosphere(6, 8)
    m = TriMeshSDF(v, f)
    p = torch.from_numpy(W.uniform_points(400000, 9)).cuda()
    tri = torch.empty(400000, dtype=torch.int32, device="cuda")
    plain = m.signed_distance(p).clone()

    def ms(**kw):
        best = 1e9
        for _ in range(4):
            t = _capi.PhaseTimings()
            m.signed_distance(p, closest_tri=tri, fp64_band=False, timings=t, **kw)
            best = min(best, t.traverse_ms)
        return best

    shapes = [(o, w) for o in (1, 2, 4) for w in (2, 4, 8) if o == 4 or w <= 4]
    times = {s: ms(occupancy=s[0], warps_per_block=s[1], queue_chunk=1) for s in shapes}
    r = m.autotune(p)
    chosen = times[r["occupancy"], r["warps_per_block"]]
    # (other shapes are 1.18 times and more; the clocks of a shared machine may move by a few per cent)
    assert chosen <= 1.12 * min(times.values()), (r, times)
    assert ms() <= 1.2 * min(times.values())
    t = _capi.PhaseTimings()
    m.signed_distance(p, fp64_band=False, timings=t)
    assert t.traverse_ms <= 2.0 * r["ms"]  # the reported time is a plain call's
    assert torch.equal(m.signed_distance(p), plain)
