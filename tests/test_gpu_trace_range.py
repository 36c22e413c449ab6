"""Ray queries of the GPU over scales and directions at which the traversal's plane
offsets overflow: host-built, GPU-built and refit trees of sheets of 1 to 1e12 units,
thin ones among them, against a test of every triangle in double precision."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, TriangleMesh, configs
from test_traversal_range_host import SHEETS, every_triangle, sheet, sheet_rays

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _mesh(tris):
    mats = [configs.Material.CreateDiffusePureColor(configs.GREY)]
    n = len(tris)
    return TriangleMesh(tris.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), np.zeros(n, np.int32), mats)


@pytest.mark.parametrize("size,direction,thin", SHEETS)
@pytest.mark.parametrize("make", ["host", "gpu", "refit"])
def test_sheets_answer_as_every_triangle(cuda_device, make, size, direction, thin):
    tris = sheet(size, thin=thin)
    rays = sheet_rays(tris, direction, 0.5 * size)
    want, want_t = every_triangle(tris, rays)
    r = SceneRenderer([], mesh=_mesh(tris if make != "refit" else sheet(0.5 * size, thin=thin)))
    if make != "host":
        r.set_build_mode("gpu")
    if make == "refit":
        r.refit_mesh(torch.as_tensor(tris.reshape(-1, 3), device="cuda"))
    rays = torch.as_tensor(rays, device="cuda")
    ids, t = r.trace_closest(rays)
    assert np.array_equal(ids.cpu().numpy(), want)
    assert np.allclose(t.cpu().numpy(), want_t, rtol=1e-5)
    assert r.trace_any(rays).all()
    assert r.error_word() == 0
