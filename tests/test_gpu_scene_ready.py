"""A scene is complete on the device when its constructor returns, whatever other threads have queued on
the legacy stream: the first host-buffer walk, on a stream of its own, gives the oracle's sums."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from tests import scenes as S

pytestmark = pytest.mark.gpu


def test_first_walk_after_the_constructor(engine, oracle, cuda):
    torch = cuda
    sc = S.scene2d(0, False, n_seg=600)
    p = engine.EstimatorParams(bie_model=1, path_length=4, num_sample_paths=64, seed=3)
    stop = threading.Event()

    def busy():
        torch.cuda.set_device(0)
        done = torch.cuda.Event()
        while not stop.is_set():
            for _ in range(3):
                torch.cuda._sleep(2_000_000)  # about a millisecond on the legacy stream
            done.record()
            done.synchronize()

    want = None
    other = threading.Thread(target=busy)
    other.start()
    try:
        for _ in range(20):
            scene = engine.SceneHost(sc["verts"], sc["normals"], sc["bvals"], sc["types"])
            got = scene.solve_domain_host(p, sc["points"])
            if want is None:
                want = oracle.solve_domain(oracle.Elements(*scene.stored_arrays()), p, sc["points"], per_path=True)[3]
                want = want.astype(np.float64)
            # 64 addends in another order: FP64 rounding against their magnitude
            assert (np.abs(got[0] - want.sum(1)) <= 64 * 2.0 ** -52 * np.abs(want).sum(1) + 1e-300).all()
            scene.close()
    finally:
        stop.set()
        other.join()
