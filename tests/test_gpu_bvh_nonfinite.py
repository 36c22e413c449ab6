"""GPU builds of meshes with an infinite or NaN vertex: the triangle that has it is
never met, and rays hit all the others as a test of every triangle in double
precision does.  The sheet is flat, so an infinite box has no area that is a number."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, TriangleMesh, configs
from test_traversal_range_host import every_triangle, sheet, sheet_rays

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 2, 3, 24, 90])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("bad", [1, 40])
def test_other_triangles_are_met(cuda_device, n, value, axis, bad):
    tris = sheet(10.0, n)
    rays = sheet_rays(tris, (0.1, -1.0, 0.2), 5.0)
    which = np.random.default_rng(n).permutation(len(tris))[:bad]
    left = tris.copy()
    left[which] = 0.0
    want, want_t = every_triangle(left, rays)
    tris[which, axis] = value
    m = len(tris)
    mesh = TriangleMesh(tris.reshape(-1, 3), np.arange(3 * m, dtype=np.uint32).reshape(-1, 3), np.zeros(m, np.int32),
                        [configs.Material.CreateDiffusePureColor(configs.GREY)])
    r = SceneRenderer([], mesh=mesh)
    r.set_build_mode("gpu")
    ids, t = r.trace_closest(torch.as_tensor(rays, device="cuda"))
    assert np.array_equal(ids.cpu().numpy(), want)
    hit = want >= 0
    assert np.allclose(t.cpu().numpy()[hit], want_t[hit], rtol=1e-5)
    assert r.error_word() == 0
