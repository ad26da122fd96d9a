"""The walk kernels' variants at the sizes where they can go wrong, path for path (or sum for sum)
against the oracle: resampling windows, shared line lists and their limit, walk-on-spheres scheduling,
batched scenes with sources, the wavefront's merged leaves, packed VPL sums, one-kernel inference.
Comparisons are exact where the arithmetic is (path values, VPL sums, the network's bits)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tests import scenes as S
from wobtoolbox_gb300 import workloads as W

pytestmark = pytest.mark.gpu
F32 = np.float32


def _elems(oracle, scene):
    return oracle.Elements(*scene.stored_arrays())


def _same_paths(engine, oracle, torch, scene, params, pts):
    vals = torch.zeros(len(pts), params.num_sample_paths, scene.dim + 1, dtype=torch.float32, device="cuda")
    scene.debug_domain_paths(params, torch.from_numpy(np.ascontiguousarray(pts, dtype=F32)).cuda(), len(pts), vals)
    torch.cuda.synchronize()
    ref = oracle.solve_domain(_elems(oracle, scene), params, pts, per_path=True)[3]
    got = vals.cpu().numpy()
    assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()


@pytest.mark.parametrize("dim,problem,bounces", [(2, 1, 3), (2, 3, 4), (3, 2, 3), (3, 3, 4)])
@pytest.mark.parametrize("candidates", [2, 3, 5, 64])
def test_resampling_windows(engine, oracle, cuda, dim, problem, bounces, candidates):
    sc = S.scene2d(problem, False) if dim == 2 else S.scene3d(problem, False)
    scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"], sc["alphas"])
    p = engine.EstimatorParams(bie_model=0, problem=problem, path_length=bounces, num_sample_paths=33, seed=4,
                               num_resampling_candidates=candidates, eps=1e-5,
                               first_kind_equation_scaling_constant=2.0)
    _same_paths(engine, oracle, cuda, scene, p, sc["points"][:4])
    scene.close()


def _comb(n, spread):
    """n vertical segments side by side: a horizontal line meets all of them."""
    x = np.linspace(-spread, spread, n)
    verts = np.stack([np.stack([x, np.full(n, 0.5)], 1), np.stack([x, np.full(n, -0.5)], 1)], 1).astype(F32)
    normals = np.tile(np.array([[1.0, 0.0]], F32), (n, 1))
    return verts, normals, np.cos(verts[..., 0]).astype(F32), np.zeros(n, np.int32)


@pytest.mark.parametrize("n,paths,bounces", [(1, 1, 1), (7, 31, 2), (40, 33, 3), (80, 64, 3), (110, 32, 4), (300, 40, 2)])
def test_shared_line_lists(engine, oracle, cuda, n, paths, bounces):
    """Totals of a warp from none to past the shared limit (3072 candidates), hits past the 64-hit cap."""
    verts, normals, data, types = _comb(n, 0.4)
    scene = engine.SceneHost(verts, normals, data, types)
    p = engine.EstimatorParams(bie_model=1, path_length=bounces, num_sample_paths=paths, seed=9)
    _same_paths(engine, oracle, cuda, scene, p, np.array([[-0.45, 0.1], [0.013, 0.02], [0.9, 0.4]], F32))
    scene.close()


@pytest.mark.parametrize("n_seg,paths,eps", [(3, 1, 1e-2), (5, 33, 1e-3), (64, 257, 1e-4), (1000, 300, 1e-4)])
def test_walk_on_spheres_sizes(engine, oracle, cuda, n_seg, paths, eps):
    torch = cuda
    verts, normals = W.star_polygon(n_seg, 3, 0.2)
    data = W.exp_cos(verts.reshape(-1, 2))[:, 0].reshape(-1, 2).astype(F32)
    scene = engine.SceneHost(verts, normals, data, np.zeros(n_seg, np.int32))
    pts = np.array([[0.05, 0.02], [0.1, -0.3], [verts[0, 0, 0], verts[0, 0, 1]]], F32)
    p = engine.EstimatorParams(num_sample_paths=paths, eps=eps, seed=2)
    per = torch.zeros(len(pts), paths, device="cuda")
    q = torch.zeros(1, dtype=torch.int64, device="cuda")
    scene.solve_wos(p, torch.from_numpy(pts).cuda(), len(pts), None, None, q, per)
    torch.cuda.synchronize()
    _, ref, queries = oracle.wos(_elems(oracle, scene), p, pts, per_path=True)
    assert np.array_equal(per.cpu().numpy(), ref) and int(q.item()) == queries
    scene.close()


def test_batched_sources_match_single_solves(engine, cuda):
    torch = cuda
    scs = W.batch_scenes(8, 3, 48, 4, (40, 40))
    scenes, params = [], []
    for sc in scs:
        h = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"], sc["alphas"])
        if sc["volume"] is not None:
            h.set_volume_cache(*sc["volume"])
        scenes.append(h)
        params.append(engine.EstimatorParams(**sc["params"], seed=6))
    pts = torch.from_numpy(np.concatenate([sc["points"] for sc in scs])).cuda()
    s, q = (torch.zeros(len(pts), 3, dtype=torch.float64, device="cuda") for _ in range(2))
    engine.SceneBatch(scenes, params, [40] * 8).solve(pts, s, q)
    ref, rq = torch.zeros_like(s), torch.zeros_like(q)
    for i, (h, p) in enumerate(zip(scenes, params)):
        k = slice(40 * i, 40 * i + 40)
        h.solve_domain(p, pts[k].contiguous(), 40, ref[k], rq[k])
    torch.cuda.synchronize()
    # the same paths, added in another order: FP64 rounding of 48 addends against their magnitude
    bound = 48 * 2.0 ** -52 * torch.sqrt(48 * rq) + 1e-300
    assert (torch.abs(s - ref) <= bound).all()


@pytest.mark.parametrize("n", [1, 3, 5, 13, 21, 80])
def test_wavefront_on_small_trees(engine, oracle, cuda, n):
    """Roots of one leaf, two-leaf nodes merged into leaves, odd counts: every wavefront shape."""
    V, F, _ = W.displaced_icosphere(1, 0.1, 4, 2)
    verts, normals = W.mesh_elements(V, F)
    verts, normals = verts[:n], normals[:n]
    scene = engine.SceneHost(verts, normals, np.ones((n, 3), F32), np.ones(n, np.int32))
    p = engine.EstimatorParams(bie_model=0, domain=1, estimator=1, problem=1, path_length=3, num_sample_paths=70, seed=1)
    lib, old = engine.load(), C.c_int32(0)
    engine.check(lib.wob_get_domain_config(3, C.byref(old)))
    try:
        for config in (0, 1, 2, 3):
            engine.check(lib.wob_set_domain_config(3, config))
            _same_paths(engine, oracle, cuda, scene, p, np.array([[1.5, 0.2, 0.1], [0.0, -1.9, 0.3]], F32))
    finally:
        lib.wob_set_domain_config(3, old.value)
    scene.close()


@pytest.mark.parametrize("n_vpl", [1, 127, 128, 129, 256, 2047, 2049, 4095, 4100])
def test_packed_vpl_sums(engine, oracle, cuda, n_vpl):
    """Tile and stage edges; points on a VPL (distance 0), within eps of one, and with zero weights."""
    torch = cuda
    verts, nrm, data, ty, _ = W.vpl_flow_scene()
    scene = engine.SceneHost(verts, nrm, data, ty)
    rng = np.random.default_rng(n_vpl)
    vp = rng.uniform(-0.5, 0.5, (n_vpl, 2)).astype(F32)
    mu = (rng.standard_normal(n_vpl) * (rng.random(n_vpl) < 0.9)).astype(F32)
    mu[n_vpl // 2] = F32(1e-25)
    pts = rng.uniform(-0.5, 0.5, (37, 2)).astype(F32)
    pts[0] = vp[0]
    pts[1] = vp[-1] + F32(3e-5)
    s = torch.zeros(len(pts), 3, dtype=torch.float64, device="cuda")
    scene.vpl_aggregate(1e-4, torch.from_numpy(vp).cuda(), torch.from_numpy(mu).cuda(), n_vpl,
                        torch.from_numpy(pts).cuda(), len(pts), s)
    torch.cuda.synchronize()
    assert np.array_equal(s.cpu().numpy(), oracle.vpl_aggregate(2, scene.info()["total_area"], 1e-4, vp, mu, pts))
    scene.close()


@pytest.mark.parametrize("eps", [1e-30, float("inf")])
@pytest.mark.parametrize("n_vpl", [130, 2100, 4100])
def test_packed_vpl_sums_infinite(engine, oracle, cuda, n_vpl, eps):
    """Infinite logarithms (a point on a VPL with eps^2 = 0, eps = inf) of one sign, the second tile of a
    pair shorter than the first or missing: infinities stay infinities."""
    torch = cuda
    verts, nrm, data, ty, _ = W.vpl_flow_scene()
    scene = engine.SceneHost(verts, nrm, data, ty)
    rng = np.random.default_rng(n_vpl)
    vp = rng.uniform(-0.5, 0.5, (n_vpl, 2)).astype(F32)
    mu = rng.uniform(0.5, 1.0, n_vpl).astype(F32)
    pts = vp[[0, 51, 100, n_vpl - 1]].copy()
    s = torch.zeros(len(pts), 3, dtype=torch.float64, device="cuda")
    scene.vpl_aggregate(eps, torch.from_numpy(vp).cuda(), torch.from_numpy(mu).cuda(), n_vpl,
                        torch.from_numpy(pts).cuda(), len(pts), s)
    torch.cuda.synchronize()
    want = oracle.vpl_aggregate(2, scene.info()["total_area"], eps, vp, mu, pts)
    assert np.isinf(want[:, 0]).all()
    assert np.array_equal(s.cpu().numpy(), want, equal_nan=True)
    scene.close()


@pytest.mark.parametrize("at", [5, 2055])
def test_packed_vpl_sums_nan(engine, oracle, cuda, at):
    """A VPL without a coordinate in one half of a pair only: as in the scalar sums, not a finite value."""
    torch = cuda
    verts, nrm, data, ty, _ = W.vpl_flow_scene()
    scene = engine.SceneHost(verts, nrm, data, ty)
    rng = np.random.default_rng(at)
    vp = rng.uniform(-0.5, 0.5, (2100, 2)).astype(F32)
    vp[at, 0] = np.nan
    mu = rng.uniform(0.5, 1.0, len(vp)).astype(F32)
    pts = rng.uniform(-0.5, 0.5, (5, 2)).astype(F32)
    s = torch.zeros(len(pts), 3, dtype=torch.float64, device="cuda")
    scene.vpl_aggregate(1e-4, torch.from_numpy(vp).cuda(), torch.from_numpy(mu).cuda(), len(vp),
                        torch.from_numpy(pts).cuda(), len(pts), s)
    torch.cuda.synchronize()
    want = oracle.vpl_aggregate(2, scene.info()["total_area"], 1e-4, vp, mu, pts)
    assert np.array_equal(s.cpu().numpy(), want, equal_nan=True)
    scene.close()


@pytest.mark.parametrize("n,hidden,out_dim", [(1, 4, 1), (15, 1, 3), (16, 4, 64), (17, 16, 1), (129, 4, 9), (5000, 2, 8)])
def test_inference_is_the_layerwise_network(engine, cuda, n, hidden, out_dim):
    """The gradient's layer-by-layer forward pass against the one-kernel inference: with its outputs as
    targets the loss is zero only if every output has the same bits."""
    torch = cuda
    from wobtoolbox_gb300 import cv
    mlp = cv.MLP(32, hidden, out_dim, 1.0, n)
    g = torch.Generator().manual_seed(n)
    x = torch.randn(n, 6, generator=g).cuda()
    y = torch.full((n, out_dim), float("nan"), device="cuda")
    mlp.forward(x, n, y)
    loss = torch.ones(1, device="cuda")
    grad = torch.empty(mlp.n_params, device="cuda")
    mlp.gradient(x, y, n, grad, loss)
    torch.cuda.synchronize()
    assert torch.isfinite(y).all() and float(y.abs().max()) > 0.0
    assert float(loss.item()) == 0.0 and not bool(grad.any())
    mlp.close()


@pytest.mark.parametrize("on_device", [False, True])
def test_offsets_keep_the_scene_where_refused(engine, oracle, cuda, on_device):
    torch = cuda
    sc = S.scene3d(1, True, subdiv=3)
    scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"])
    n = scene.n_elems
    delta = np.linspace(-0.5, 0.5, n).astype(F32)
    give = lambda a: torch.from_numpy(a).cuda() if on_device else a
    clone = scene.clone_with_offsets(give(delta))
    _, _, totals = oracle.scene_cdfs(_elems(oracle, clone))
    assert F32(clone.info()["total_boundary_value"]) == F32(totals[1])
    bad = delta.copy()
    bad[n // 2] = np.inf
    d = give(bad)
    status = engine.load().wob_scene_add_boundary_offsets(clone.handle, d.data_ptr() if on_device else d.ctypes.data, n,
                                                          int(on_device), None)
    assert status != 0 and F32(clone.info()["total_boundary_value"]) == F32(totals[1])
    p = engine.EstimatorParams(bie_model=0, domain=1, estimator=1, problem=1, path_length=3, num_sample_paths=40, seed=3)
    _same_paths(engine, oracle, cuda, clone, p, sc["points"][:3])
    clone.close()
    scene.close()
