"""An infinite density on one triangle in the control-variate sums (every triangle taken, theta = 0): the
potential is infinite at every point, also where the triangle is near enough for the closed form, and
the residual data away from it is that of the far rule."""
from __future__ import annotations

import numpy as np
import pytest

from wobtoolbox_gb300 import cv
from wobtoolbox_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("subdiv", [1, 3])
def test_infinite_density(engine, cuda, subdiv):
    torch = cuda
    V, F, _ = W.displaced_icosphere(subdiv, 0.1, 4, 2)
    verts, normals = W.mesh_elements(V, F)
    scene = engine.SceneHost(verts, normals, np.ones((len(F), 3), F32), np.ones(len(F), np.int32))
    v, n = scene.stored_arrays()[:2]
    k = len(F) // 3
    sigma = np.full(len(F), 0.25, F32)
    sigma[k] = np.inf
    cen = v.astype(np.float64).mean(1)
    # above the triangle (closed form), above its neighbours, and far from all
    d2 = ((cen - cen[k]) ** 2).sum(1)
    order = np.argsort(d2)
    pts = np.concatenate([cen[order[:40]] + 0.01 * n[order[:40]].astype(np.float64), [[0, 0, 2.5], [-2, 1, 0.3]]]).astype(F32)
    d_sigma = torch.from_numpy(sigma).cuda()
    got = cv.control_variate_potential(scene, d_sigma, torch.from_numpy(pts).cuda(), len(pts), near_factor=3.0, theta=0.0)
    delta = torch.zeros(len(F), device="cuda")
    engine.check(engine.load().wob_cv_residual_data(scene.handle, d_sigma.data_ptr(), 1, 3.0, 0.0, delta.data_ptr(), None))
    torch.cuda.synchronize()
    assert (got[:, 0] == float("inf")).all()
    # grad u of one infinite charge: infinite along every axis on which the point is off its centroid
    # and its field does not vanish
    assert not torch.isnan(got[:, 1:]).any()
    # -inf or inf with the sign of the normal derivative; the triangle itself has -sigma / c = inf / 2
    assert torch.isinf(delta).all() and not torch.isnan(delta).any()
    scene.close()
