"""The discs of the polygon-face search leave out only evaluations that cannot lower a query's minimum: with discs
that every query reaches, the same kernel returns the same values and faces bit for bit -- on faces off their
plane as well, whose results depend on which boxes were open when."""
import ctypes as C

import numpy as np
import pytest
import torch

from ebgeometry_b200 import PolygonMeshSDF, _capi
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu

_capi.lib.ebg_polymesh_open_discs.argtypes = [C.c_void_p]
_capi.lib.ebg_polymesh_open_discs.restype = C.c_int


@pytest.mark.parametrize("name,warp", [("quad24", 0.0), ("quad24", 0.01), ("quad12", 0.1), ("mixed16", 0.03), ("prism129", 0.0),
                                       ("prism40", 0.05)])
@pytest.mark.parametrize("leaf", [1, 4, 32])
def test_open_discs_change_nothing(name, warp, leaf):
    kind, size = name.rstrip("0123456789"), int("".join(c for c in name if c.isdigit()))
    v, faces = {"quad": lambda: W.displaced_quad_sphere(size, 7), "mixed": lambda: W.mixed_polygon_sphere(size, 3),
                "prism": lambda: W.polygon_prism(size, 0.8, 1.5)}[kind]()
    rng = np.random.default_rng(leaf)
    v = v + rng.normal(size=v.shape) * warp
    m = PolygonMeshSDF(v, faces, leaf_size=leaf)
    p = np.concatenate([rng.uniform(-1.6, 1.6, (9001, 3)), rng.normal(0, 40, (3000, 3)), rng.normal(0, 1e6, (500, 3)),
                        v[rng.integers(0, len(v), 4000)] + rng.normal(0, 1e-3, (4000, 3))])
    p = torch.from_numpy(p[rng.permutation(len(p))]).cuda()
    a, b = (torch.empty(len(p), dtype=torch.int32, device="cuda") for _ in range(2))
    d = m.signed_distance(p, closest_face=a)[0].clone()
    assert _capi.lib.ebg_polymesh_open_discs(m._h) == 0
    e = m.signed_distance(p, closest_face=b)[0]
    m.check_status()
    assert torch.equal(d, e) and torch.equal(a, b)
