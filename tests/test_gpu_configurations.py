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
    """Configuration c of the walk kernels: the (c mod 4)-th of 1, 5, 6, 8 resident blocks per SM."""
    scene, p, pts = _variant_case(engine, variant)
    for config in range(16):
        configure(variant, config)
        assert launches(cuda, tmp_path, scene, p, pts) == [("dl2d_kernel" if variant == 1 else "domain_kernel", (1, 5, 6, 8)[config % 4])]
    scene.close()
