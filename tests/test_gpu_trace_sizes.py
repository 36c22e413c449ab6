"""Ray batches of every size class (one ray per warp, a few, whole warps with
refills; partial chunks and warps) against the host traversal of the same rays,
bit for bit: ids and t of the closest hits, and visibility up to a limit.  Some
rays are axis-parallel, some start inside the cloud, some have a tmin."""
import ctypes as C

import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, TriangleMesh, _lib, configs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TRIS = configs.random_triangles(3000, seed=4)


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-0.2, 1.2, (n, 3))
    d = rng.normal(size=(n, 3))
    d[::7] = np.eye(3)[rng.integers(0, 3, len(d[::7]))] * rng.choice([-1.0, 1.0], (len(d[::7]), 1))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[::5, 3] = 0.2
    r[:, 7] = np.where(np.arange(n) % 3 == 0, 0.7, np.inf)
    return r


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 2431, 2433, 4865, 9729, 19457, 38913, 77825, 160001, 400003])
def test_batches_equal_the_host_traversal(cuda_device, n):
    mats = [configs.Material.CreateDiffusePureColor(configs.GREY)]
    mesh = TriangleMesh(TRIS.reshape(-1, 3), np.arange(3 * len(TRIS), dtype=np.uint32).reshape(-1, 3),
                        np.zeros(len(TRIS), np.int32), mats)
    r = SceneRenderer([], mesh=mesh)
    rays = _rays(n, n)
    ids, t = r.trace_closest(torch.as_tensor(rays, device="cuda"))
    hit = r.trace_any(torch.as_tensor(rays, device="cuda"))
    want_id, want_t, visits = np.zeros(n, np.int32), np.zeros(n, np.float32), C.c_int64()
    assert _lib.load().ar_host_trace_closest(TRIS.ctypes.data, len(TRIS), rays.ctypes.data, n, want_id.ctypes.data,
                                             want_t.ctypes.data, C.byref(visits)) == 0
    assert np.array_equal(ids.cpu().numpy(), want_id)
    assert np.array_equal(t.cpu().numpy().view(np.uint32), want_t.view(np.uint32))
    assert np.array_equal(hit.cpu().numpy(), (want_id >= 0).astype(np.int32))
    assert r.error_word() == 0
