"""A forward walk whose path state comes from the scratch pool, captured as a process's first work on the
device: replays add the paths of eager calls."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

PROGRAM = """
import numpy as np, torch
import wobtoolbox_gb300 as wob
from wobtoolbox_gb300 import workloads as W
V, F, _ = W.displaced_icosphere(2, 0.1, 4, 2)
verts, normals = W.mesh_elements(V, F)
n, paths = 2000, 70
scene = wob.SceneHost(verts, normals, np.ones((len(verts), 3), np.float32), np.ones(len(verts), np.int32))
params = wob.EstimatorParams(bie_model=0, domain=1, estimator=1, problem=1, path_length=3, num_sample_paths=paths, seed=1)
u = np.random.default_rng(0).standard_normal((n, 3))
pts = torch.from_numpy((1.8 * u / np.linalg.norm(u, axis=1, keepdims=True)).astype(np.float32)).cuda()
new = lambda: (torch.zeros(n, 4, dtype=torch.float64, device="cuda"), torch.zeros(n, 4, dtype=torch.float64, device="cuda"))
got, want = new(), new()
torch.cuda.synchronize()
stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    scene.solve_domain(params, pts, n, got[0], got[1], None, stream)
graph.replay()
graph.replay()
for _ in range(2):
    scene.solve_domain(params, pts, n, want[0], want[1])
torch.cuda.synchronize()
# 140 addends in one fixed order per call, two calls: equal up to the rounding of the sums
bound = 140 * 2.0 ** -52 * torch.sqrt(140 * want[1]) + 1e-300
assert (want[1] > 0).any() and (torch.abs(got[0] - want[0]) <= bound).all()
assert (torch.abs(got[1] - want[1]) <= 140 * 2.0 ** -52 * want[1] + 1e-300).all()
scene.close()
print("replayed")
"""


def test_first_walk_of_a_process_is_captured(engine, cuda):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "replayed" in r.stdout, r.stdout[-500:] + r.stderr[-2000:]
