"""The device build's sampling tables (parallel Kahan prefix sums, guide table) and its sort at the
sizes where they can go wrong: both sides of the serial route's limit (2048), chunk and tile edges,
weights over many binades, runs of zeros. The totals are compared bit for bit with the oracle's serial
sums over the device scene's storage order, the area table through the elements that the boundary
sampler draws (one draw picks the element: the first whose CDF value reaches it)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F32 = np.float32


def _philox_first(n, seed, stream):
    """First uniform of Philox4x32-10 streams (0, 0, 0, i), key (seed, stream) (Salmon et al., SC'11)."""
    m = np.uint64(0xFFFFFFFF)
    c = [np.zeros(n, np.uint64), np.zeros(n, np.uint64), np.zeros(n, np.uint64), np.arange(n, dtype=np.uint64)]
    k0, k1 = np.uint64(seed), np.uint64(stream)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & m, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m, (k1 + np.uint64(0xBB67AE85)) & m
    return ((c[0] >> np.uint64(8)) + np.uint64(1)).astype(F32) * F32(2.0 ** -24)


def _triangles(n, kind, seed):
    """n triangles of seeded sizes at random places; normals encode the index (length within the
    accepted range)."""
    rng = np.random.default_rng(seed)
    size = {"even": np.full(n, 0.01), "binades": np.exp(2.5 * rng.standard_normal(n)) * 1e-3,
            "zeros": np.where((np.arange(n) // 300) % 3 == 1, 0.0, rng.uniform(0.5, 1.0, n))}[kind]
    at = rng.uniform(-1, 1, (n, 3))
    verts = np.repeat(at[:, None, :], 3, axis=1)
    verts[:, 1, 0] += size
    verts[:, 2, 1] += size
    normals = np.zeros((n, 3), F32)
    normals[:, 0] = F32(1.0) + np.arange(n, dtype=F32) * F32(2.0 ** -20)
    data = rng.standard_normal((n, 3)) * (rng.random(n) < 0.7)[:, None]
    return verts.astype(F32), normals, data.astype(F32)


@pytest.mark.parametrize("n,kind", [(2, "even"), (2048, "binades"), (2049, "even"), (2049, "zeros"), (4095, "binades"),
                                    (4097, "zeros"), (20481, "binades"), (70000, "even"), (131073, "zeros")])
def test_device_tables_are_the_serial_ones(engine, oracle, cuda, n, kind):
    torch = cuda
    verts, normals, data = _triangles(n, kind, n)
    t = lambda a: torch.from_numpy(a).cuda()
    scene = engine.SceneHost.build_on_device(t(verts), t(normals), t(data),
                                             torch.ones(n, dtype=torch.int32, device="cuda"))
    order = scene.element_order
    assert np.array_equal(np.sort(order), np.arange(n))
    v, nn, b, ty, al = scene.stored_arrays()
    area_cdf, _, totals = oracle.scene_cdfs(oracle.Elements(v, nn, b, ty, al))
    info = scene.info()
    assert F32(info["total_area"]) == F32(totals[0]) and F32(info["total_boundary_value"]) == F32(totals[1])
    m = 1 << 18
    out = {k: torch.empty(m, *s, device="cuda") for k, s in (("p", (3,)), ("n", (3,)), ("a", ()), ("b", ()))}
    types = torch.empty(m, dtype=torch.int32, device="cuda")
    engine.check(engine.load().wob_scene_sample_boundary(scene.handle, m, 5, out["p"].data_ptr(), out["n"].data_ptr(),
                                                         out["a"].data_ptr(), out["b"].data_ptr(), types.data_ptr(),
                                                         None, None))
    drawn = np.rint((out["n"][:, 0].cpu().numpy().astype(np.float64) - 1.0) * 2.0 ** 20).astype(np.int64)
    pick = np.minimum(np.searchsorted(area_cdf, _philox_first(m, 5, 2), side="left"), n - 1)
    assert np.array_equal(drawn, order[pick])
    scene.close()
