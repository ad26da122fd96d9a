"""Inference whose outputs lie over its inputs (in place, or shifted within one allocation) gives what it
gives with buffers of their own."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hidden,out_dim,shift", [(1, 4, 6, 0), (5000, 4, 6, 0), (5000, 4, 1, 0), (20000, 2, 6, 40),
                                                    (3000, 4, 8, -3000), (4000, 16, 3, 23999), (700, 4, 64, 0)])
def test_outputs_over_inputs(engine, cuda, n, hidden, out_dim, shift):
    torch = cuda
    from wobtoolbox_gb300 import cv
    mlp = cv.MLP(32, hidden, out_dim, 1.0, 5)
    x = torch.randn(n, 6, generator=torch.Generator().manual_seed(n)).cuda()
    want = torch.zeros(n, out_dim, device="cuda")
    mlp.forward(x, n, want)
    at = max(0, -shift)  # where the inputs start in the shared allocation
    buf = torch.zeros(at + max(n * 6, max(shift, 0) + n * out_dim) + 64, device="cuda")
    buf[at:at + n * 6] = x.reshape(-1)
    out = buf[at + shift:at + shift + n * out_dim]
    mlp.forward(buf[at:], n, out)
    torch.cuda.synchronize()
    assert torch.equal(out.reshape(n, out_dim), want)
    mlp.close()
