"""GPU-built and refit trees quantise child boxes with float arithmetic rounded
outwards: meshes of tiny, huge, flat and far-off coordinates (steps of a node
from 2^-126 up, differences that round) answer ray queries as the host-built
tree does, bit for bit, from one leaf to several levels."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, TriangleMesh, configs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _mesh(tris):
    mats = [configs.Material.CreateDiffusePureColor(configs.GREY)]
    n = len(tris)
    return TriangleMesh(tris.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), np.zeros(n, np.int32), mats)


def _rays(tris, seed):
    rng = np.random.default_rng(seed)
    v = tris.reshape(-1, 3, 3).astype(np.float64)
    at = v[rng.integers(0, len(v), 4000)].mean(1)
    size = np.ptp(v.reshape(-1, 3), 0).max() + 1e-30
    o = at + size * rng.normal(size=at.shape)
    d = at - o
    r = np.zeros((len(at), 8), np.float32)
    r[:, 0:3], r[:, 4:7], r[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), np.inf
    return torch.as_tensor(r, device="cuda")


@pytest.mark.parametrize("n", [1, 3, 4, 9, 700, 20000])
@pytest.mark.parametrize("kind", ["unit", "tiny", "huge", "far", "flat"])
def test_gpu_build_and_refit_answer_as_the_host_tree(cuda_device, n, kind):
    base = configs.random_triangles(n, seed=n).reshape(-1, 3).astype(np.float64)
    scale, offset = {"tiny": (1e-15, 0.0), "huge": (1e12, 0.0), "far": (1.0, 30000.0)}.get(kind, (1.0, 0.0))
    if kind == "flat":
        base[:, 1] = 0.25
    tris = (base * scale + offset).astype(np.float32).reshape(n, 9)
    moved = (base[:, [1, 0, 2]] * (0.7 * scale) + offset + 0.1 * scale).astype(np.float32).reshape(n, 9)
    for now, make in ((tris, "build"), (moved, "refit")):
        host = SceneRenderer([], mesh=_mesh(now))
        rays = _rays(now, 5)
        want = host.trace_closest(rays)
        gpu = SceneRenderer([], mesh=_mesh(tris))
        gpu.set_build_mode("gpu")
        if make == "refit":
            gpu.refit_mesh(torch.as_tensor(now.reshape(-1, 3), device="cuda"))
        got = gpu.trace_closest(rays)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        assert gpu.error_word() == 0
