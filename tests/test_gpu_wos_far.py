"""Walks on spheres that leave the float range: from points outside the boundary one walk in some thirty
jumps past 1.8e19, where squared distances overflow. Such a walk ends without a value (0), as in the
oracle, and not at the step limit."""
from __future__ import annotations

import numpy as np
import pytest

from wobtoolbox_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("n_seg", [5, 300])
def test_walks_that_overflow_end_without_a_value(engine, oracle, cuda, n_seg):
    torch = cuda
    verts, normals = W.star_polygon(n_seg, 3, 0.2)
    data = (2.0 + W.exp_cos(verts.reshape(-1, 2))[:, 0]).reshape(-1, 2).astype(F32)
    scene = engine.SceneHost(verts, normals, data, np.zeros(n_seg, np.int32))
    pts = np.array([[2.0, 0.5], [-3.0, 4.0], [50.0, 1.0], [3e18, -1e18], [3e30, 0.0], [np.inf, 0.0], [np.nan, 0.0]], F32)
    paths = 256
    p = engine.EstimatorParams(num_sample_paths=paths, eps=1e-3, seed=8)
    per = torch.full((len(pts), paths), -1.0, device="cuda")
    q = torch.zeros(1, dtype=torch.int64, device="cuda")
    scene.solve_wos(p, torch.from_numpy(pts).cuda(), len(pts), None, None, q, per)
    torch.cuda.synchronize()
    _, ref, queries = oracle.wos(oracle.Elements(*scene.stored_arrays()), p, pts, per_path=True)
    assert (ref == 0.0).any() and (ref[:3] > 0.0).any()
    assert scene.poll_error() == 0
    assert np.array_equal(per.cpu().numpy(), ref) and int(q.item()) == queries
    scene.close()
