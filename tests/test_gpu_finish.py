"""Small waves and the tails of large ones run to their end in one kernel
(k_finish); profiled renders always launch the stages of every depth.  Both
perform the same operations per path, so their images are equal bit for bit:
waves of one path, of a block and one path around it, and waves around the
size where the one-kernel form takes over from the first depth on."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, configs

pytestmark = pytest.mark.gpu


def _scene(name):
    if name == "glass":
        return dict(sceneObjects=configs.glass_test_scene()), configs.GLASS_TEST_CAMERA, 1000
    if name == "cornell":
        return dict(sceneObjects=configs.cornell_triangles()), configs.CORNELL_CAMERA, 8
    if name == "textured":
        objs, mesh, tex = configs.textured_cornell(configs.cornell_textures(16))
        return dict(sceneObjects=objs, mesh=mesh, textures=tex), configs.CORNELL_CAMERA, 6
    objs, mesh = configs.terrain_scene(res=96, n_spheres=8)
    return dict(sceneObjects=objs, mesh=mesh, medium=configs.COMBINED_MEDIUM if name == "medium" else None), \
        configs.TERRAIN_CAMERA, 16


@pytest.mark.parametrize("name", ["cornell", "glass", "textured", "terrain", "medium"])
@pytest.mark.parametrize("size", [(1, 1, 1), (17, 15, 1), (16, 16, 1), (257, 1, 1), (255, 203, 3), (397, 389, 1),
                                  (400, 390, 2)])
def test_one_kernel_equals_the_launches_per_depth(cuda_device, name, size):
    scene, cam, depth = _scene(name)
    r = SceneRenderer(**scene)
    w, h, spp = size
    a = r.Render((w, h), cam["origin"], cam["direction"], spp, fov=cam["fov"], max_depth=depth)
    b = r.Render((w, h), cam["origin"], cam["direction"], spp, fov=cam["fov"], max_depth=depth, profile=1)
    assert np.array_equal(a, b)
    assert r.error_word() == 0
