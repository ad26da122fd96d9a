"""wob_clip_magnitude_quantile takes no scene and is stream-ordered without a host synchronisation: as a
process's first engine call it can be captured, and replays clip."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

PROGRAM = """
import torch
import wobtoolbox_gb300 as wob
lib = wob.load()
torch.cuda.set_device(0)
n = 5000
v = torch.randn(n, generator=torch.Generator().manual_seed(1)).cuda()
w, t = v.clone(), torch.zeros(1, device="cuda")
torch.cuda.synchronize()
stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=stream):
    wob.check(lib.wob_clip_magnitude_quantile(w.data_ptr(), n, 0.9, t.data_ptr(), stream.cuda_stream))
for scale in (1.0, 3.0):
    w.copy_(scale * v)
    graph.replay()
    torch.cuda.synchronize()
    want = torch.sort((scale * v).abs()).values[4499]  # the ceil(0.9 n)-th smallest
    assert t.item() == want.item() and torch.equal(w, (scale * v).clamp(-want, want))
print("clipped")
"""


def test_first_call_of_a_process_is_captured(engine, cuda):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "clipped" in r.stdout, r.stdout[-500:] + r.stderr[-2000:]
