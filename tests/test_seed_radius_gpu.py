"""Queries that pass an attached model, with and without anchors, give the plain distances whatever the model's
radii are: a trained model's, none, exact ones, and an untrained model's, which leave most queries far from
the surface without a triangle in reach (these are searched again without a bound)."""
import numpy as np
import pytest
import torch

from ebgeometry_b200 import SeedModel, TriMeshSDF
from ebgeometry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mesh_and_models():
    v, f = W.displaced_icosphere(5, 9)
    m = TriMeshSDF(v, f)
    box = dict(lo=[-1.2] * 3, hi=[1.2] * 3)
    return m, {"trained": SeedModel.train(m, attach=False, num_samples=1 << 18, steps=200, batch=1 << 14, rng_seed=5, **box),
               "untrained": SeedModel.create(log2_table=12, **box)}


@pytest.mark.parametrize("model,mode", [("trained", 0), ("untrained", 0), ("untrained", 1), ("untrained", 2)])
@pytest.mark.parametrize("anchors", [True, False])
def test_plain_distances_for_any_radius(mesh_and_models, model, mode, anchors):
    m, models = mesh_and_models
    # inside the cells, outside of them (where the model says nothing), and on the grid's faces
    p = torch.from_numpy(np.concatenate([W.uniform_points(90001, 3), W.grid_points(50), W.uniform_points(5000, 4, -9, 9),
                                         np.array([[1.2, 0, 0], [-1.2, -1.2, -1.2]], np.float32)])).cuda()
    plain = m.signed_distance(p).clone()
    m.attach_seed(models[model], cells_per_axis=24, radius_mode=mode, anchors=anchors)
    try:
        for kw in ({}, {"fp64_band": False}, {"sort": False}):
            ref = m.signed_distance(p, **kw)
            assert torch.equal(m.signed_distance(p, seed=models[model], **kw), ref), kw
        assert torch.equal(m.signed_distance(p, seed=models[model]), plain)
        m.check_status()
    finally:
        m.detach_seed()
