"""The network called from several host threads."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_inference_beside_training_sees_whole_steps(engine, cuda):
    """An inference call made while another thread trains the network returns the network before the
    training call or after it, never parameters of several steps."""
    from wobtoolbox_gb300 import cv
    torch = cuda
    n, rows = 4096, 20000
    g = torch.Generator().manual_seed(1)
    x = torch.randn(n, 6, generator=g).cuda()
    tx, ty = torch.randn(rows, 6, generator=g).cuda(), torch.randn(rows, 1, generator=g).cuda()
    mlp = cv.MLP(32, 4, 1, 1.0, 3)

    own = torch.cuda.Stream()
    y, back = torch.zeros(n, 1, device="cuda"), torch.zeros(n, 1).pin_memory()
    torch.cuda.synchronize()

    def infer():
        # (a device-wide wait is not allowed while the training call captures its step)
        mlp.forward(x, n, y, own)
        with torch.cuda.stream(own):
            back.copy_(y, non_blocking=True)
        own.synchronize()
        return back.numpy().copy()

    whole = [infer()]
    seen = []
    for k in range(6):
        started = threading.Event()

        def train():
            torch.cuda.set_device(0)
            started.set()
            mlp.train(tx, ty, rows, 2000, 4096, 1e-3, seed=k)

        t = threading.Thread(target=train)
        t.start()
        started.wait()
        while t.is_alive():
            seen.append((k, infer()))
        t.join()
        whole.append(infer())
    assert seen and not np.array_equal(whole[0], whole[1])
    for k, y in seen:
        assert np.array_equal(y, whole[k]) or np.array_equal(y, whole[k + 1])
    mlp.close()
