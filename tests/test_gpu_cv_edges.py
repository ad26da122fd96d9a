"""The closed form near triangles' edges against 64 bits. The potential's gradient there is a logarithm of the
distance d to the edge and the solid angle of the triangle.

Bound: a coordinate along a unit vector (distance to the plane, to the edge's line) carries some 8 roundings of
|v| <= L, so d is off by 8 u L, the logarithm of d^2 by 16 u L / d and the solid angle by about 10 u L / d; up to
six triangles meet near a point of an edge, each with density at most smax: 6 (16 + 10) u L / d smax / (4 pi), beside
1e-6 of the largest gradient for everything farther away."""
from __future__ import annotations

import numpy as np
import pytest

from wobtoolbox_gb300 import cv
from wobtoolbox_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("subdiv", [1, 2, 3])
@pytest.mark.parametrize("scale", [1.0, 1e-3])
def test_gradient_near_edges(engine, cuda, subdiv, scale):
    from oracle import cv_tables as T
    torch = cuda
    V, F, _ = W.displaced_icosphere(subdiv, 0.15, 4, 0)
    verts, normals = W.mesh_elements(V * scale, F)
    scene = engine.SceneHost(verts, normals, np.ones((len(F), 3), F32), np.ones(len(F), np.int32))
    v = scene.stored_arrays()[0].astype(np.float64)
    rng = np.random.default_rng(subdiv)
    sigma = rng.uniform(0.5, 1.0, len(F)).astype(F32)
    n = 3000
    t, e = rng.integers(0, len(F), n), rng.integers(0, 3, n)
    a, b = v[t, e], v[t, (e + 1) % 3]
    s = (b - a) / np.linalg.norm(b - a, axis=1, keepdims=True)
    r = np.cross(s, rng.standard_normal((n, 3)))
    d = np.exp(rng.uniform(np.log(1e-4), np.log(1e-2), (n, 1))) * scale
    x = (a + (b - a) * rng.uniform(0.15, 0.85, (n, 1)) + d * r / np.linalg.norm(r, axis=1, keepdims=True)).astype(F32)
    got = cv.control_variate_potential(scene, torch.from_numpy(sigma).cuda(), torch.from_numpy(x).cuda(), n,
                                       near_factor=3.0, theta=0.0)
    torch.cuda.synchronize()
    ref = T.potential(v, sigma, x, 3.0)
    w = x.astype(np.float64) - a
    dist = np.linalg.norm(w - (w * s).sum(1, keepdims=True) * s, axis=1)
    L = 2 * np.linalg.norm(b - a, axis=1).max()
    bound = 6 * 26 * 2.0 ** -24 * L / dist * float(sigma.max()) / (4 * np.pi) + 1e-6 * np.abs(ref[:, 1:]).max()
    err = np.linalg.norm(got.cpu().numpy()[:, 1:] - ref[:, 1:], axis=1)
    assert (err <= bound).all(), (np.max(err / bound), np.quantile(err / bound, [0.5, 0.99]))
    scene.close()
