"""The kernels behind the tunable variants' configurations (include/wob_capi.h, wob_autotune_domain), read
from the launches of captured solves, and path for path against the oracle."""
from __future__ import annotations

import ctypes as C
import re

import numpy as np
import pytest

from tests import scenes as S

pytestmark = pytest.mark.gpu


def _cudart():
    paths = {line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line}
    return C.CDLL(sorted(paths)[0])


def launches(torch, tmp_path, scene, params, pts):
    """The kernels a domain solve launches: [(name, minimum blocks per SM or None)]."""
    rt = _cudart()
    d = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    s = torch.zeros(len(pts), scene.dim + 1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), C.c_void_p()
    assert rt.cudaStreamBeginCapture(C.c_void_p(stream.cuda_stream), 2) == 0
    scene.solve_domain(params, d, len(pts), s, None, None, stream)
    assert rt.cudaStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph)) == 0
    dot = tmp_path / "graph.dot"
    assert rt.cudaGraphDebugDotPrint(graph, str(dot).encode(), 1) == 0
    rt.cudaGraphDestroy(graph)
    # mangled names: <length><identifier>_kernelI...Li<minimum blocks>EEE (the trace kernel's comes first)
    out = []
    for name, args in re.findall(r"\d((?:domain|dl2d|wave_\w+?|compress_nodes)_kernel)(I\w*?EEE?v)?", dot.read_text()):
        nums = re.findall(r"Li(\d+)E", args)
        out.append((name, int(nums[0 if "trace" in name else -1]) if nums else None))
    return out


@pytest.fixture
def configure(engine):
    """Sets configurations; the ones that were set before come back at the end."""
    lib, saved = engine.load(), {}

    def set_(variant, config):
        if variant not in saved:
            old = C.c_int32(0)
            engine.check(lib.wob_get_domain_config(variant, C.byref(old)))
            saved[variant] = old.value
        engine.check(lib.wob_set_domain_config(variant, config))

    yield set_
    for variant, config in saved.items():
        engine.check(lib.wob_set_domain_config(variant, config))


def _variant_case(engine, variant):
    dim, problem, bie, est, exterior = [(3, 2, 2, 0, False), (2, 0, 1, 0, False), (3, 1, 2, 0, False), (3, 1, 0, 1, True)][variant]
    sc = S.scene2d(problem, exterior) if dim == 2 else S.scene3d(problem, exterior)
    scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"], sc["alphas"])
    p = engine.EstimatorParams(bie_model=bie, problem=problem, estimator=est, domain=int(exterior), path_length=3,
                               num_sample_paths=33, seed=2)
    return scene, p, sc["points"]


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_published_occupancies(engine, cuda, tmp_path, configure, variant):
    """Configuration c of the walk kernels: the (c mod 4)-th of 1, 5, 6 resident blocks per SM and the one by
    size; a launch past every line takes 8 (12 for the double layer)."""
    import dataclasses
    scene, p, pts = _variant_case(engine, variant)
    large = dataclasses.replace(p, num_sample_paths=30000)
    for config in range(16):
        configure(variant, config)
        name = "dl2d_kernel" if variant == 1 else "domain_kernel"
        assert launches(cuda, tmp_path, scene, p, pts) == [(name, (1, 5, 6, 8 if variant == 1 else 1)[config % 4])]
        assert launches(cuda, tmp_path, scene, large, pts) == [(name, (1, 5, 6, 12 if variant == 1 else 8)[config % 4])]
    scene.close()


@pytest.mark.parametrize("problem", [1, 3])
@pytest.mark.parametrize("points,paths", [(456, 128), (457, 128), (760, 128), (761, 128)])
def test_direct_walks_on_both_sides_of_their_size_rules(engine, oracle, cuda, tmp_path, configure, problem, points, paths):
    """No cap, 5 and 8 blocks per SM by the launch's size: the oracle's path values, and sums, of each."""
    torch = cuda
    sc = S.scene3d(problem, False, subdiv=1)
    scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"], sc["alphas"])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pts = np.random.default_rng(points).uniform(-0.3, 0.3, (points, 3)).astype(np.float32)
    p = engine.EstimatorParams(bie_model=2, problem=problem, path_length=3, num_sample_paths=paths, seed=5)
    warps = points * -(-paths // 32)
    variant = 2 if problem == 1 else 0
    configure(variant, 3)
    want = 1 if warps <= 12 * sms else 5 if warps <= 20 * sms else 8
    assert launches(torch, tmp_path, scene, p, pts) == [("domain_kernel", want)]
    ref = oracle.solve_domain(oracle.Elements(*scene.stored_arrays()), p, pts, per_path=True)[3]
    d = torch.from_numpy(pts).cuda()
    for config in (3, 2):
        configure(variant, config)
        got = _paths(engine, torch, scene, p, d, points)
        assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()
    scene.close()


@pytest.mark.parametrize("n_seg,points,paths", [(40, 3, 33), (300, 304, 256), (300, 305, 256)])
def test_double_layer_without_a_line_grid(engine, oracle, cuda, tmp_path, configure, n_seg, points, paths):
    """Device-built scenes, which have no line grid: each configuration runs its own occupancy (no limit:
    4), the last one 4 or 8 by size, with the oracle's path values."""
    torch = cuda
    sc = S.scene2d(0, False, n_seg=n_seg)
    t = lambda a, dt=torch.float32: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dt)  # noqa: E731
    scene = engine.SceneHost.build_on_device(t(sc["verts"]), t(sc["normals"]), t(sc["bvals"]), t(sc["types"], torch.int32))
    pts = np.random.default_rng(points).uniform(-0.4, 0.4, (points, 2)).astype(np.float32)
    p = engine.EstimatorParams(bie_model=1, path_length=3, num_sample_paths=paths, seed=11)
    small = points * -(-paths // 32) <= 16 * torch.cuda.get_device_properties(0).multi_processor_count
    ref = oracle.solve_domain(oracle.Elements(*scene.stored_arrays()), p, pts, per_path=True)[3]
    d = torch.from_numpy(pts).cuda()
    for config in range(4):
        configure(1, config)
        assert launches(torch, tmp_path, scene, p, pts) == [("domain_kernel", (4, 5, 6, 4 if small else 8)[config])]
        got = _paths(engine, torch, scene, p, d, points)
        assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()
    scene.close()


def test_every_variant_starts_with_configuration_3_and_gets_it_back(engine, cuda, tmp_path):
    """Reading, changing and setting back what was read leaves every later solve's kernels as they were."""
    import subprocess
    import sys
    program = (
        "import ctypes as C, pathlib, sys, tempfile, torch\n"
        "import wobtoolbox_gb300 as wob\n"
        "from tests import test_gpu_configurations as T\n"
        "lib = wob.load(); tmp = pathlib.Path(tempfile.mkdtemp())\n"
        "cases = [T._variant_case(wob, v) for v in range(4)]\n"
        "torch.zeros(1).cuda()\n"
        "seen = lambda: [T.launches(torch, tmp, *c) for c in cases]\n"
        "first = seen()\n"
        "for v in range(4):\n"
        "    old = C.c_int32(-7); wob.check(lib.wob_get_domain_config(v, C.byref(old))); assert old.value == 3, old.value\n"
        "    wob.check(lib.wob_set_domain_config(v, 14)); wob.check(lib.wob_set_domain_config(v, old.value))\n"
        "assert seen() == first, (seen(), first)\n"
        "assert [f[0][1] for f in first] == [1, 8, 1, 5] and [len(f) for f in first] == [1] * 4, first\n"
        "for c in (-1, 16): assert lib.wob_set_domain_config(0, c) != 0\n"
        "print('restored')\n")
    import os
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", program], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "restored" in r.stdout, r.stdout[-500:] + r.stderr[-2000:]


def _paths(engine, torch, scene, params, d, n):
    vals = torch.zeros(n, params.num_sample_paths, scene.dim + 1, device="cuda")
    scene.debug_domain_paths(params, d, n, vals)
    s, q = (torch.zeros(n, scene.dim + 1, dtype=torch.float64, device="cuda") for _ in range(2))
    scene.solve_domain(params, d, n, s, q)
    torch.cuda.synchronize()
    vals = vals.cpu().numpy()
    exact = vals.astype(np.float64)
    m = params.num_sample_paths  # the same addends in another order: FP64 rounding against their magnitude
    assert (np.abs(s.cpu().numpy() - exact.sum(1)) <= m * 2.0 ** -52 * np.abs(exact).sum(1) + 1e-300).all()
    assert (np.abs(q.cpu().numpy() - (exact ** 2).sum(1)) <= m * 2.0 ** -52 * (exact ** 2).sum(1) + 1e-300).all()
    return vals


@pytest.mark.parametrize("points,paths", [(608, 256), (609, 256), (19, 8192), (700, 300), (4865, 31)])
def test_double_layer_on_both_sides_of_its_size_rule(engine, oracle, cuda, tmp_path, configure, points, paths):
    """Launches of 8 blocks per SM and 12, in the per-path and the summing form, against the oracle, and the
    configured occupancies on the same launch."""
    torch = cuda
    sc = S.scene2d(0, False, n_seg=300)
    scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pts = np.random.default_rng(points).uniform(-0.45, 0.45, (points, 2)).astype(np.float32)
    p = engine.EstimatorParams(bie_model=1, path_length=3, num_sample_paths=paths, seed=11)
    configure(1, 3)
    small = points * -(-paths // 32) <= 32 * sms
    assert launches(torch, tmp_path, scene, p, pts) == [("dl2d_kernel", 8 if small else 12)]
    ref = oracle.solve_domain(oracle.Elements(*scene.stored_arrays()), p, pts, per_path=True)[3]
    d = torch.from_numpy(pts).cuda()
    for config in (3, 0, 1, 2, 15):
        configure(1, config)
        got = _paths(engine, torch, scene, p, d, points)
        assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()
    scene.close()


@pytest.mark.parametrize("subdiv,points,paths", [(1, 3040, 32), (1, 3041, 32), (3, 95, 1024), (3, 96, 1024), (0, 10, 9999)])
def test_forward_walk_on_both_sides_of_its_size_rule(engine, oracle, cuda, tmp_path, configure, subdiv, points, paths):
    """Configuration 3 runs the lockstep kernel where its warps are all resident there and the wavefront on
    compressed nodes above; configuration 7 the wavefront at every size. Path values are the oracle's."""
    torch = cuda
    sc = S.scene3d(1, True, subdiv=subdiv)
    scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    u = np.random.default_rng(points).standard_normal((points, 3))
    pts = (1.9 * u / np.linalg.norm(u, axis=1, keepdims=True)).astype(np.float32)
    p = engine.EstimatorParams(bie_model=0, domain=1, estimator=1, problem=1, path_length=2, num_sample_paths=paths, seed=4)
    small = points * -(-paths // 32) <= 20 * sms
    configure(3, 3)
    names = [n for n, _ in launches(torch, tmp_path, scene, p, pts)]
    assert (names == ["domain_kernel"]) == small and ("wave_trace_kernel" in names) == (not small)
    configure(3, 7)
    assert ("wave_trace_kernel", 9) in launches(torch, tmp_path, scene, p, pts[:2])
    ref = oracle.solve_domain(oracle.Elements(*scene.stored_arrays()), p, pts, per_path=True, accel=True)[3]
    d = torch.from_numpy(pts).cuda()
    for config in (3, 7, 0):
        configure(3, config)
        got = _paths(engine, torch, scene, p, d, points)
        assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()
    scene.close()


@pytest.mark.parametrize("n", [1, 3, 5, 13, 21, 80])
def test_compressed_wavefront_on_small_trees(engine, oracle, cuda, configure, n):
    """Roots of one leaf, two-leaf nodes merged into leaves, odd counts, on the compressed nodes."""
    from wobtoolbox_gb300 import workloads as W
    torch = cuda
    V, F, _ = W.displaced_icosphere(1, 0.1, 4, 2)
    verts, normals = W.mesh_elements(V, F)
    verts, normals = verts[:n], normals[:n]
    scene = engine.SceneHost(verts, normals, np.ones((n, 3), np.float32), np.ones(n, np.int32))
    p = engine.EstimatorParams(bie_model=0, domain=1, estimator=1, problem=1, path_length=3, num_sample_paths=70, seed=1)
    pts = np.array([[1.5, 0.2, 0.1], [0.0, -1.9, 0.3]], np.float32)
    configure(3, 7)
    got = _paths(engine, torch, scene, p, torch.from_numpy(pts).cuda(), len(pts))
    ref = oracle.solve_domain(oracle.Elements(*scene.stored_arrays()), p, pts, per_path=True)[3]
    assert ((got == ref) | (np.isnan(got) & np.isnan(ref))).all()
    scene.close()
