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


def _sdf_scene(name):
    from aperturerendererv3_gb300._lib import OBJECT_SDF
    from aperturerendererv3_gb300.scene import Material, SceneObject, sdf
    objs, mesh = configs.terrain_scene(res=48, n_spheres=8)
    kw = dict(mesh=mesh)
    if name != "objects":
        kw.update(sdf=configs.sdf_blobs(), medium=configs.COMBINED_MEDIUM)
    if name != "union":
        glass = Material.CreateGlassPureColor((0.9, 1.0, 0.9), 1.5, 1.0)
        objs = objs + [SceneObject((0.4, 0.3, 0.7), (0.15, 0.15, 0.15), glass, (20.0, 30.0, 0.0), OBJECT_SDF,
                                   additionalObjectInfo=sdf.CreateTorus()),
                       SceneObject((0.7, 0.25, 0.6), (0.1, 0.1, 0.1),
                                   Material.CreateGGXPureColor((0.8, 0.5, 0.3), 0.3, 0.0, 0.5), (0.0, 0.0, 0.0),
                                   OBJECT_SDF, additionalObjectInfo=sdf.CreateTorus())]
    return SceneRenderer(objs, **kw)


@pytest.mark.parametrize("name", ["union", "objects", "both"])
@pytest.mark.parametrize("size", [(1, 1, 1), (33, 31, 1), (129, 67, 2), (640, 500, 2)])
def test_sdf_scenes_in_one_kernel(cuda_device, name, size):
    """Scenes with a smooth union, SDF objects (one of them glass: rays inside it
    test only it) or both, below and above the switch."""
    r = _sdf_scene(name)
    cam = configs.COMBINED_CAMERA
    w, h, spp = size
    a = r.Render((w, h), cam["origin"], cam["direction"], spp, fov=cam["fov"], max_depth=24)
    b = r.Render((w, h), cam["origin"], cam["direction"], spp, fov=cam["fov"], max_depth=24, profile=1)
    assert np.array_equal(a, b)
    assert r.error_word() == 0
