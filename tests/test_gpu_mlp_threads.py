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


def test_inference_of_networks_of_different_depth(engine, cuda):
    """Networks of different depths, which need different amounts of shared memory, evaluated from two
    threads at once: every call is accepted and gives what it gives alone."""
    from wobtoolbox_gb300 import cv
    torch = cuda
    n = 64
    x = torch.randn(n, 6, generator=torch.Generator().manual_seed(1)).cuda()
    nets = [cv.MLP(32, hidden, 1, 1.0, hidden) for hidden in (16, 8)]
    outs = [torch.zeros(n, 1, device="cuda") for _ in nets]
    streams = [torch.cuda.Stream() for _ in nets]
    alone = []
    torch.cuda.synchronize()
    for net, out, st in zip(nets, outs, streams):
        net.forward(x, n, out, st)
        st.synchronize()
        alone.append(out.clone())
        out.zero_()
    torch.cuda.synchronize()
    failed = []

    def loop(i):
        torch.cuda.set_device(0)
        try:
            for _ in range(5000):
                nets[i].forward(x, n, outs[i], streams[i])
        except Exception as ex:  # noqa: BLE001 - reported by the assertion below
            failed.append(repr(ex))

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    for net, out, want in zip(nets, outs, alone):
        assert torch.equal(out, want)
        net.close()
