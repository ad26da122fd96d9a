"""Batched scenes of the direct model, with and without a source term, and of the forward estimator, among others: every scene's sums are
those of its own solve (the same paths, whose values the oracle tests cover, in another order)."""
from __future__ import annotations

import numpy as np
import pytest

from tests import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("points,paths", [(1, 1), (7, 33), (90, 64)])
def test_direct_scenes_in_a_batch(engine, oracle, cuda, dim, points, paths):
    torch = cuda
    make = (lambda problem, k: S.scene2d(problem, False, n_seg=30 + 7 * k)) if dim == 2 else \
        (lambda problem, k: S.scene3d(problem, False, subdiv=1 + k % 2, seed=k))
    scenes, params = [], []
    rng = np.random.default_rng(dim)
    # (model, problem, source, estimator): uniform samples (problems 0, 2, 3), line queries (1), other models and
    # the forward estimator between them
    for k, (bie, problem, vol, est) in enumerate([(2, 0, 0, 0), (2, 2, 1, 0), (0, 2, 0, 0), (2, 3, 0, 0), (2, 1, 0, 1),
                                                  (2, 1, 0, 0), (1, 0, 0, 0), (2, 3, 1, 0), (2, 3, 1, 1), (2, 0, 1, 0),
                                                  (0, 0, 1, 1), (1, 0, 0, 1), (0, 1, 0, 1)]):
        sc = make(problem, k)
        h = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"], sc["alphas"])
        if vol:
            h.set_volume_cache(8, 2.6, rng.standard_normal(8 ** dim).astype(np.float32))
        scenes.append(h)
        params.append(engine.EstimatorParams(bie_model=bie, problem=problem, estimator=est, path_length=4, num_sample_paths=paths, seed=k,
                                             num_volume_samples=vol, num_resampling_candidates=4, eps=1e-5))
    n = len(scenes)
    pts = torch.from_numpy(rng.uniform(-0.3, 0.3, (n * points, dim)).astype(np.float32)).cuda()
    s, q = (torch.zeros(n * points, dim + 1, dtype=torch.float64, device="cuda") for _ in range(2))
    engine.SceneBatch(scenes, params, [points] * n).solve(pts, s, q)
    for i, (h, p) in enumerate(zip(scenes, params)):
        k = slice(points * i, points * (i + 1))
        per = torch.zeros(points, paths, dim + 1, device="cuda")
        h.debug_domain_paths(p, pts[k].contiguous(), points, per)
        torch.cuda.synchronize()
        exact = per.double()
        bound = paths * 2.0 ** -52 * exact.abs().sum(1) + 1e-300
        assert (torch.abs(s[k] - exact.sum(1)) <= bound).all(), i
        assert (torch.abs(q[k] - (exact ** 2).sum(1)) <= paths * 2.0 ** -52 * (exact ** 2).sum(1) + 1e-300).all(), i
