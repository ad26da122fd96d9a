"""The work a user of the engine has it do, as measurable cases through the public Python API.

Families (`kind`), over the ranges `draw` spreads:

* walk: per-point walks on one scene, accumulated into FP64 sums with the path offset advanced from
  pass to pass (the apps' iteration loop). 2D double-layer Dirichlet, 3D direct Robin and 3D forward
  single-layer Neumann, from a handful of points to whole slices; `host` cases go through the
  host-buffer call.
* batch: several 2D scenes with their own parameters (Neumann forward with and without a source
  term, Robin with resampling) solved in one call.
* multi: many right-hand sides sharing one set of walks (mixed problem, resampling).
* build: a scene built on the device from device arrays.
* vpl: one iteration of the virtual-point-light potential flow (walks, then the dense aggregation).
* wos: walk on spheres on a star.
* tables: the learned control variate's evaluation (network at the centroids, residual data,
  residual scene, potential at the points).
* train: optimisation steps of the control variate's network.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

import wobtoolbox_gb300 as wob
from wobtoolbox_gb300 import cv
from wobtoolbox_gb300 import workloads as W

F32 = np.float32


def listed():
    return [
        # an interactive probe: a few points on a small 2D scene, bound by launches and latency
        dict(name="star2d_probe", kind="walk", problem="dirichlet2d", elems=256, points=64, paths=64, bounces=6,
             host=False),
        # the 2D field of a general_2d configuration: the 1024-segment star on a 128^2 grid
        dict(name="star2d_dirichlet", kind="walk", problem="dirichlet2d", elems=1024, points=7960, paths=1024,
             bounces=8, host=False),
        # the 3D interior Robin slice on 81,920 triangles, a share of its paths
        dict(name="sphere3d_robin", kind="walk", problem="robin3d", elems=81920, points=109062, paths=512, bounces=16,
             host=False),
        # one host-buffer call of a medium 3D scene (copies in, walks, copies out)
        dict(name="sphere3d_robin_host", kind="walk", problem="robin3d", elems=20480, points=4099, paths=96, bounces=8,
             host=True),
        # the exterior Neumann slice on 327,680 triangles by the forward estimator
        dict(name="sphere3d_neumann", kind="walk", problem="neumann3d", elems=327680, points=54025, paths=64,
             bounces=4, host=False),
        # several 2D problems with their own meshes, sources and parameters in one call
        dict(name="star2d_batch", kind="batch", scenes=24, points=4000, paths=64, bounces=8),
        # the mixed 3D problem for 64 right-hand sides at once
        dict(name="sphere3d_mixed_64rhs", kind="multi", elems=81920, points=20011, paths=32, bounces=4, rhs=64,
             candidates=64),
        # a scene built on the device from a mesh of 327,680 triangles
        dict(name="sphere3d_build", kind="build", mesh="ico", elems=327680, robin=False),
        # one iteration of the potential-flow app's configuration
        dict(name="flow2d_vpl", kind="vpl", paths=100000, points=39280, bounces=4, candidates=1024),
        # walk on spheres for the star's field
        dict(name="star2d_spheres", kind="wos", elems=1024, points=7960, paths=256, eps=1e-4),
        # the learned control variate evaluated on 327,680 triangles and a slice of points
        dict(name="sphere3d_cv_tables", kind="tables", elems=327680, points=54025),
        # the control variate's network: optimisation steps on 65,536 boundary samples
        dict(name="network_train", kind="train", rows=65536, batch=8192, steps=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "walk", "walk", "batch", "multi", "build", "vpl", "wos", "tables", "train"])
    ico = lambda lo, hi: 20 * 4 ** rng.randint(lo, hi)  # icosphere sizes  # noqa: E731
    if kind == "walk":
        problem = rng.choice(["dirichlet2d", "robin3d", "neumann3d"])
        elems = _log(rng, 64, 8192) if problem == "dirichlet2d" else ico(3, 6) if problem == "robin3d" else ico(3, 7)
        host = problem != "neumann3d" and rng.random() < 0.3
        points = _log(rng, 16, 8192 if host else 40000)
        paths = _log(rng, 16, 512 if problem != "neumann3d" else 64)
        return dict(kind=kind, problem=problem, elems=elems, points=points, paths=paths, bounces=rng.randint(3, 12) if problem != "neumann3d" else rng.randint(2, 4),
                    host=host)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 24), points=_log(rng, 100, 4000), paths=_log(rng, 16, 64),
                    bounces=rng.randint(3, 8))
    if kind == "multi":
        return dict(kind=kind, elems=ico(3, 6), points=_log(rng, 64, 20000), paths=_log(rng, 8, 32),
                    bounces=rng.randint(2, 4), rhs=rng.randint(3, 64), candidates=rng.choice([1, 8, 64]))
    if kind == "build":
        return dict(kind=kind, mesh=rng.choice(["ico", "uv"]), elems=ico(3, 7) if rng.random() < 0.4 else _log(rng, 300, 327680),
                    robin=rng.random() < 0.5)
    if kind == "vpl":
        return dict(kind=kind, paths=_log(rng, 1000, 100000), points=_log(rng, 256, 39280), bounces=rng.randint(2, 4),
                    candidates=rng.choice([1, 16, 256, 1024]))
    if kind == "wos":
        return dict(kind=kind, elems=_log(rng, 64, 8192), points=_log(rng, 64, 7960), paths=_log(rng, 16, 256),
                    eps=rng.choice([1e-3, 1e-4]))
    if kind == "tables":
        return dict(kind=kind, elems=ico(3, 7), points=_log(rng, 64, 54025))
    return dict(kind=kind, rows=_log(rng, 1000, 65536), batch=_log(rng, 64, 8192), steps=rng.randint(5, 128))


# ------------------------------------------------------------------ meshes and points
@functools.lru_cache(maxsize=None)
def _unit_icosphere(subdiv):
    V, F = W.icosphere(subdiv)
    return V, F, W.real_sph_harm(4, V)


def _uv_sphere(n):
    """A latitude-longitude sphere with about n triangles (an odd number of segments)."""
    seg = max(3, int(math.sqrt(n))) | 1
    ring = max(2, int(round(n / (2 * seg))) + 1)
    t = np.pi * np.arange(1, ring) / ring
    p = 2 * np.pi * np.arange(seg) / seg
    V = np.stack([np.outer(np.sin(t), np.cos(p)), np.outer(np.sin(t), np.sin(p)),
                  np.outer(np.cos(t), np.ones(seg))], -1).reshape(-1, 3)
    V = np.concatenate([V, [[0.0, 0.0, 1.0], [0.0, 0.0, -1.0]]])
    top, bot = len(V) - 2, len(V) - 1
    j = np.arange(seg)
    k = (j + 1) % seg
    faces = [np.stack([np.full(seg, top), j, k], 1), np.stack([np.full(seg, bot), (ring - 2) * seg + k,
                                                               (ring - 2) * seg + j], 1)]
    for r in range(ring - 2):
        a, b = r * seg + j, r * seg + k
        faces += [np.stack([a, a + seg, b], 1), np.stack([b, a + seg, b + seg], 1)]
    F = np.concatenate(faces)
    return V, F, W.real_sph_harm(4, V)


def _subdiv(elems):
    s = int(round(math.log(elems / 20, 4)))
    if 20 * 4 ** s != elems:
        raise ValueError("an icosphere has 20 * 4^s triangles")
    return s


def _coefficients(rng, Y):
    """Seeded radial displacement 0.15 sum c_lm Y_lm (l <= 4), at most 0.4 of the radius."""
    c = 0.15 * rng.standard_normal(Y.shape[1])
    c[0] = 0.0
    return c * min(1.0, 0.4 / np.abs(Y @ c).max())


def _surface(elems, rng, mesh="ico"):
    V, F, Y = _unit_icosphere(_subdiv(elems)) if mesh == "ico" and elems in {20 * 4 ** s for s in range(3, 8)} \
        else _uv_sphere(elems)
    c = _coefficients(rng, Y)
    V = V * (1.0 + Y @ c)[:, None]
    verts, normals = W.mesh_elements(V, F)
    return verts, normals, c


def _sources(rng, exterior):
    d = rng.standard_normal((3, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return d * (rng.uniform(0.0, 0.3, (3, 1)) if exterior else rng.uniform(2.0, 4.0, (3, 1))), rng.uniform(-1, 1, 3)


def _field(verts, src, q):
    """u and grad u of point sources at every element vertex, float64 on the GPU: [n, D, 4]."""
    p = torch.from_numpy(verts.reshape(-1, 3)).cuda().double()
    u = torch.zeros(len(p), 4, dtype=torch.float64, device="cuda")
    for s, a in zip(src, q):
        d = p - torch.from_numpy(s).cuda()
        r = torch.linalg.norm(d, dim=1, keepdim=True)
        u[:, :1] += a / (4 * math.pi * r)
        u[:, 1:] += -a * d / (4 * math.pi * r ** 3)
    return u.reshape(len(verts), 3, 4)


def _dudn(u, normals):
    return (u[..., 1:] * torch.from_numpy(normals).cuda().double()[:, None, :]).sum(-1)


def _pick(cand, n):
    return np.ascontiguousarray(cand[np.linspace(0, len(cand) - 1, n).astype(np.int64)])


def _slice_points(c, n, exterior):
    """n points of a z = 0 slice inside (or outside) the displaced sphere, in grid order."""
    size = 4.0 if exterior else 2.8
    res = max(8, int(math.sqrt(6.0 * n)) + 1)
    g = W.slice_points_z0(res, size)
    r = np.linalg.norm(g.astype(np.float64), axis=1)
    surf = 1.0 + W.real_sph_harm(4, g / np.maximum(r, 1e-12)[:, None]) @ c
    return _pick(g[r > 1.04 * surf] if exterior else g[(r < 0.96 * surf)], n)


def _star(elems, rng):
    lobes, amp = int(rng.integers(3, 10)), float(rng.uniform(0.1, 0.35))
    verts, normals = W.star_polygon(elems, lobes, amp)
    g = W.exp_cos(verts.reshape(-1, 2))[:, 0].reshape(-1, 2).astype(F32)
    return verts, normals, g, lobes, amp


def _star_points(n, lobes, amp):
    g = W.idx_to_domain_point(max(8, int(math.sqrt(4.0 * n)) + 1), 2.0 * (1.0 + amp), 2)
    r = np.linalg.norm(g.astype(np.float64), axis=1)
    return _pick(g[r < 0.97 * (1.0 + amp * np.cos(lobes * np.arctan2(g[:, 1], g[:, 0])))], n)


def _sums(points, width):
    z = lambda: torch.zeros(points, width, dtype=torch.float64, device="cuda")  # noqa: E731
    return dict(sum=z(), sumsq=z(), bounces=torch.zeros(1, dtype=torch.int64, device="cuda"))


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    rng = np.random.default_rng([seed, 20250])
    kind = case["kind"]
    s = dict(case=dict(case), kind=kind, done=0, seed=seed)
    if kind == "walk":
        if case["problem"] == "dirichlet2d":
            verts, normals, g, lobes, amp = _star(case["elems"], rng)
            s["scene"] = wob.SceneHost(verts, normals, g, np.zeros(len(verts), np.int32))
            pts = _star_points(case["points"], lobes, amp)
            s["params"] = wob.EstimatorParams(bie_model=wob.IndirectDoubleLayer)
        else:
            exterior = case["problem"] == "neumann3d"
            verts, normals, c = _surface(case["elems"], rng)
            u = _field(verts, *_sources(rng, exterior))
            if exterior:
                s["scene"] = wob.SceneHost(verts, normals, _dudn(u, normals).float().cpu().numpy(),
                                           np.ones(len(verts), np.int32))
                s["params"] = wob.EstimatorParams(bie_model=wob.IndirectSingleLayer, domain=wob.ExteriorDomain,
                                                  estimator=wob.ForwardEstimator, problem=wob.NeumannProblem)
            else:
                h = (_dudn(u, normals) + 2.0 * u[..., 0]).float().cpu().numpy()
                s["scene"] = wob.SceneHost(verts, normals, h, np.full(len(verts), 2, np.int32),
                                           np.full((len(verts), 3), 2.0, F32))
                s["params"] = wob.EstimatorParams(bie_model=wob.Direct, problem=wob.RobinProblem)
            pts = _slice_points(c, case["points"], exterior)
        s["params"] = dataclasses.replace(s["params"], path_length=case["bounces"], num_sample_paths=case["paths"],
                                          seed=seed)
        if case["host"]:
            s["points"] = pts
            s["sum"], s["sumsq"] = (np.zeros((len(pts), pts.shape[1] + 1)) for _ in range(2))
        else:
            s["points"] = torch.from_numpy(pts).cuda()
            s.update(_sums(len(pts), pts.shape[1] + 1))
    elif kind == "batch":
        scs = W.batch_scenes(case["scenes"], seed, case["paths"], case["bounces"], (case["points"], case["points"]))
        for i, sc in enumerate(scs):  # point counts spread from an eighth of `points` to all of them
            sc["points"] = sc["points"][:max(1, case["points"] * (8 - 3 * i % 8) // 8)]
        scenes = []
        for sc in scs:
            h = wob.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"], sc["alphas"])
            if sc["volume"] is not None:
                h.set_volume_cache(*sc["volume"])
            scenes.append(h)
        n = [len(sc["points"]) for sc in scs]
        s["batch"] = wob.SceneBatch(scenes, [wob.EstimatorParams(**sc["params"], seed=seed) for sc in scs], n)
        s["points"] = torch.from_numpy(np.concatenate([sc["points"] for sc in scs])).cuda()
        s.update(_sums(sum(n), 3))
    elif kind == "multi":
        verts, normals, c = _surface(case["elems"], rng)
        dirichlet = torch.from_numpy(verts[:, :, 2].astype(np.float64).mean(1) > 0).cuda()
        table = torch.empty(len(verts), 3, case["rhs"], device="cuda")
        for r in range(case["rhs"]):
            u = _field(verts, *_sources(rng, False))
            table[:, :, r] = torch.where(dirichlet[:, None], u[..., 0], _dudn(u, normals)).float()
        table = table.cpu().numpy()
        s["scene"] = wob.SceneHost(verts, normals, table[:, :, 0], np.where(dirichlet.cpu().numpy(), 0, 1))
        s["scene"].set_rhs(table)
        s["params"] = wob.EstimatorParams(bie_model=wob.IndirectSingleLayer, problem=wob.MixedProblem,
                                          path_length=case["bounces"], num_sample_paths=case["paths"],
                                          num_resampling_candidates=case["candidates"], eps=float(F32(1e-5)),
                                          first_kind_equation_scaling_constant=2.0, seed=seed)
        s["points"] = torch.from_numpy(_slice_points(c, case["points"], False)).cuda()
        s.update(_sums(case["points"], case["rhs"]))
    elif kind == "build":
        verts, normals, _ = _surface(case["elems"], rng, case["mesh"])
        u = _field(verts, *_sources(rng, False))
        alphas = rng.uniform(0.5, 2.0, (len(verts), 3)).astype(F32) if case["robin"] else None
        g = _dudn(u, normals).float()
        order = rng.permutation(len(verts))  # a mesh file's faces come in no spatial order
        s["mesh"] = [torch.from_numpy(np.ascontiguousarray(verts[order])).cuda(),
                     torch.from_numpy(np.ascontiguousarray(normals[order])).cuda(),
                     g[torch.from_numpy(order).cuda()].contiguous(),
                     torch.full((len(verts),), 2 if case["robin"] else 1, dtype=torch.int32, device="cuda"),
                     None if alphas is None else torch.from_numpy(alphas).cuda()]
    elif kind == "vpl":
        verts, normals, data, types, circles = W.vpl_flow_scene()
        data = data * F32(rng.uniform(0.5, 2.0))
        s["scene"] = wob.SceneHost(verts, normals, data, types)
        g, keep = W.vpl_flow_points(max(24, int(math.sqrt(2.0 * case["points"])) + 1), circles)
        s["points"] = torch.from_numpy(_pick(g[keep], case["points"])).cuda()
        s["params"] = wob.EstimatorParams(bie_model=wob.IndirectSingleLayer, problem=wob.NeumannProblem,
                                          path_length=case["bounces"], num_resampling_candidates=case["candidates"],
                                          eps=1e-4, seed=seed)
        s["vpl"] = (torch.empty(case["paths"], 2, device="cuda"), torch.empty(case["paths"], device="cuda"))
        s["sum"] = torch.zeros(case["points"], 3, dtype=torch.float64, device="cuda")
        s["bounces"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    elif kind == "wos":
        verts, normals, g, lobes, amp = _star(case["elems"], rng)
        s["scene"] = wob.SceneHost(verts, normals, g, np.zeros(len(verts), np.int32))
        s["points"] = torch.from_numpy(_star_points(case["points"], lobes, amp)).cuda()
        s["params"] = wob.EstimatorParams(num_sample_paths=case["paths"], eps=case["eps"], seed=seed)
        s.update(_sums(case["points"], 1))
    elif kind == "tables":
        verts, normals, c = _surface(case["elems"], rng)
        u = _field(verts, *_sources(rng, True))
        s["scene"] = wob.SceneHost(verts, normals, _dudn(u, normals).float().cpu().numpy(),
                                   np.ones(len(verts), np.int32))
        s["mlp"] = cv.MLP(32, 4, 1, 1.0, seed)
        s["order"] = torch.from_numpy(s["scene"].element_order.astype(np.int64)).cuda()
        s["points"] = torch.from_numpy(_slice_points(c, case["points"], True)).cuda()
    else:
        s["inputs"], s["targets"] = _rows(case, seed)
        s["mlp"] = cv.MLP(32, 4, 1, 1.0, seed)
        s["loss"] = torch.zeros(case["steps"], device="cuda")
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "walk":
        p = dataclasses.replace(s["params"], path_offset=s["done"] * case["paths"])
        s["done"] += 1
        if case["host"]:
            return s["scene"].solve_domain_host(p, s["points"], s["sum"], s["sumsq"])
        s["scene"].solve_domain(p, s["points"], case["points"], s["sum"], s["sumsq"], s["bounces"])
        return s["sum"], s["sumsq"], s["bounces"]
    if kind == "batch":
        s["batch"].solve(s["points"], s["sum"], s["sumsq"], s["bounces"], s["done"] * case["paths"])
        s["done"] += 1
        return s["sum"], s["sumsq"], s["bounces"]
    if kind == "multi":
        p = dataclasses.replace(s["params"], path_offset=s["done"] * case["paths"])
        s["done"] += 1
        s["scene"].solve_domain_multi(p, s["points"], case["points"], s["sum"], s["sumsq"], s["bounces"])
        return s["sum"], s["sumsq"], s["bounces"]
    if kind == "build":
        scene = wob.SceneHost.build_on_device(*s["mesh"])
        info = scene.info()
        order = scene.element_order.astype(np.int64)
        scene.close()
        return dict(order=order, nodes=info["n_nodes"], depth=info["bvh_depth"], area=info["total_area"],
                    boundary=info["total_boundary_value"])
    if kind == "vpl":
        p = dataclasses.replace(s["params"], path_offset=s["done"] * case["paths"])
        s["done"] += 1
        pos, mu = s["vpl"]
        s["scene"].vpl_paths(p, case["paths"], pos, mu, s["bounces"])
        s["scene"].vpl_aggregate(p.eps, pos, mu, case["paths"], s["points"], case["points"], s["sum"])
        return pos, mu, s["sum"], s["bounces"]
    if kind == "wos":
        p = dataclasses.replace(s["params"], path_offset=s["done"] * case["paths"])
        s["done"] += 1
        s["scene"].solve_wos(p, s["points"], case["points"], s["sum"], s["sumsq"], s["bounces"])
        return s["sum"], s["sumsq"], s["bounces"]
    if kind == "tables":
        scene, n = s["scene"], s["scene"].n_elems
        x = cv.centroid_inputs(scene)
        sigma = torch.empty(n, 1, device="cuda")
        s["mlp"].forward(x, n, sigma)
        delta = torch.empty(n, device="cuda")
        wob._capi.check(wob.load().wob_cv_residual_data(scene.handle, sigma.data_ptr(), wob.ExteriorDomain, 3.0, 0.3,
                                                        delta.data_ptr(), None))
        residual = scene.clone_with_offsets(delta)
        total = residual.info()["total_boundary_value"]
        potential = cv.control_variate_potential(scene, sigma, s["points"], case["points"])
        residual.close()
        by_face = torch.empty(n, device="cuda")
        by_face[s["order"]] = sigma[:, 0]  # the density in the mesh's own order
        return dict(sigma=by_face, delta=delta, boundary=total, potential=potential)
    s["mlp"].train(s["inputs"], s["targets"], case["rows"], case["steps"], case["batch"], 2e-3, seed=s["seed"],
                   loss_history=s["loss"])
    return s["loss"], s["mlp"].params()[0]


# ------------------------------------------------------------------ network inputs and 64-bit values
def _rows(case, seed):
    """Boundary samples (point, normal) of a unit sphere with a smooth density and walk-like noise."""
    g = torch.Generator().manual_seed(seed)
    d = torch.randn(case["rows"], 3, generator=g)
    d = d / d.norm(dim=1, keepdim=True)
    a = torch.randn(4, generator=g)
    t = a[0] * d[:, 0] + a[1] * d[:, 1] * d[:, 2] + a[2] * torch.sin(3.0 * d[:, 2]) + 0.1 * a[3]
    t = t + 0.05 * torch.randn(case["rows"], generator=g)
    return torch.cat([d, d], 1).contiguous().cuda(), t.contiguous().cuda()


def _network(seed):
    """The network's seeded start in float64: parameters per layer and frequencies (splitmix64)."""
    mask = (1 << 64) - 1
    st = (seed * 0x9E3779B97F4A7C15 + 0x632BE59BD9B4E019) & mask

    def nxt():
        nonlocal st
        st = (st + 0x9E3779B97F4A7C15) & mask
        z = st
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return ((z ^ (z >> 31)) >> 11) * 2.0 ** -53

    layers = []
    for out in (64, 64, 64, 64, 1):
        w = np.array([(2.0 * nxt() - 1.0) / 8.0 for _ in range(64 * out)]).astype(F32)
        layers.append([torch.from_numpy(w.reshape(out, 64)).double().cuda(),
                       torch.zeros(out, dtype=torch.float64, device="cuda")])
    fr = []
    for _ in range(32 * 6):
        u1, u2 = nxt() + 1e-300, nxt()
        fr.append(math.sqrt(-2.0 * math.log(u1)) * math.cos(2.0 * math.pi * u2))
    return layers, torch.from_numpy(np.array(fr, F32).reshape(32, 6)).double().cuda()


def _forward(layers, freqs, x):
    t = 2.0 * math.pi * (x.double() @ freqs.T)
    h = torch.cat([torch.sin(t), torch.cos(t)], 1)
    for i, (w, b) in enumerate(layers):
        h = h @ w.T + b
        if i + 1 < len(layers):
            h = torch.nn.functional.silu(h)
    return h


def _exact_train(case, seed):
    layers, freqs = _network(seed)
    x, t = _rows(case, seed)
    t = t.double()[:, None]
    flat = [p.requires_grad_() for wb in layers for p in wb]
    m = [torch.zeros_like(p) for p in flat]
    v = [torch.zeros_like(p) for p in flat]
    rows = np.arange(case["batch"], dtype=np.uint64)
    losses = []
    for step in range(case["steps"]):
        with np.errstate(over="ignore"):
            c = [rows.copy(), np.full_like(rows, step), np.zeros_like(rows), np.full_like(rows, 0x7472616E)]
            k0, k1 = np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)
            f = np.uint64(0xFFFFFFFF)
            for _ in range(10):
                p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
                c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & f, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & f]
                k0, k1 = (k0 + np.uint64(0x9E3779B9)) & f, (k1 + np.uint64(0xBB67AE85)) & f
            idx = torch.from_numpy(((c[0] * np.uint64(case["rows"])) >> np.uint64(32)).astype(np.int64)).cuda()
        loss = ((_forward(layers, freqs, x[idx]) - t[idx]) ** 2).mean()
        losses.append(float(loss))
        grads = torch.autograd.grad(loss, flat)
        lr = 2e-3 * 0.5 * (1.0 + math.cos(math.pi * step / case["steps"]))
        with torch.no_grad():
            for p, g, a, b in zip(flat, grads, m, v):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).addcmul_(g, g, value=0.001)
                p -= lr * (a / (1 - 0.9 ** (step + 1))) / ((b / (1 - 0.999 ** (step + 1))).sqrt() + 1e-8)
    return torch.tensor(losses, dtype=torch.float64), torch.cat([p.detach().reshape(-1) for p in flat])


def exact(case, seed):
    """Walk estimates (FP32 random walks) have no 64-bit counterpart; a build's totals, the network's
    values and its training do."""
    rng = np.random.default_rng([seed, 20250])
    if case["kind"] == "build":
        verts, normals, _ = _surface(case["elems"], rng, case["mesh"])
        g = _dudn(_field(verts, *_sources(rng, False)), normals).float().double()
        v = torch.from_numpy(verts).cuda().double()
        area = torch.linalg.norm(torch.linalg.cross(v[:, 2] - v[:, 0], v[:, 1] - v[:, 0]), dim=1) / 2
        f64 = lambda x: x.sum().cpu()  # noqa: E731
        return dict(order=None, nodes=None, depth=None, area=f64(area), boundary=f64(area * g.abs().mean(1)))
    if case["kind"] == "tables":
        verts, normals, _ = _surface(case["elems"], rng)
        x = torch.from_numpy(np.concatenate([verts.astype(np.float64).mean(1), normals], 1)).cuda()
        return dict(sigma=_forward(*_network(seed), x)[:, 0], delta=None, boundary=None, potential=None)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None


# ------------------------------------------------------------------ work a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "walk":
        D = 2 if case["problem"] == "dirichlet2d" else 3
        bounces = case["points"] * case["paths"] * case["bounces"]
        # per bounce: a line query and its segment tests (2D), two uniform samples and their kernels
        # (Robin), a line query over the triangles' hierarchy (Neumann)
        per = {"dirichlet2d": 345, "robin3d": 160, "neumann3d": 2535}[case["problem"]]
        return dict(bytes=case["elems"] * 4 * (D * D + 3 * D) + case["points"] * (4 * D + 32 * (D + 1)), flops=bounces * per)
    if kind == "batch":
        bounces = case["scenes"] * 0.5625 * case["points"] * case["paths"] * case["bounces"]
        return dict(bytes=case["scenes"] * (1024 * 40 + 0.5625 * case["points"] * 104), flops=bounces * (345 + 64 * 40) / 2)
    if kind == "multi":
        bounces = case["points"] * case["paths"] * case["bounces"]
        return dict(bytes=case["elems"] * 12 * (6 + case["rhs"]) + case["points"] * (12 + 32 * case["rhs"]),
                    flops=bounces * (case["candidates"] * 60 + case["rhs"] * 8))
    if kind == "build":
        n = case["elems"]
        # vertices, normals, data and types in; records, nodes, tables and the order out
        return dict(bytes=n * (36 + 12 + 12 + 4 + (12 if case["robin"] else 0) + 64 + 16 + 64 + 48 + 8 + 32 + 4), flops=0)
    if kind == "vpl":
        return dict(bytes=case["paths"] * 12 + case["points"] * 56,
                    flops=case["paths"] * (case["points"] * 60 + case["bounces"] * case["candidates"] * 40))
    if kind == "wos":
        jumps = 20 * case["points"] * case["paths"]  # about twenty closest-point queries a walk
        return dict(bytes=case["elems"] * 40 + case["points"] * 40, flops=jumps * 20 * math.log2(case["elems"]))
    if kind == "tables":
        n, m = case["elems"], case["points"]
        # per target some hundreds of expansions and near triangles, and the network's products
        return dict(bytes=n * (36 + 12 + 24 + 4 + 4 + 64) + m * 28, flops=n * 2 * 16448 + (n + m) * 2000 * 40)
    return dict(bytes=case["rows"] * 28, flops=case["steps"] * case["batch"] * 6 * 16448)
