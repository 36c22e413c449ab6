"""A GPU build makes the primitive records, the slot and light tables and the
refit levels on the device.  Scenes of objects of every kind (SDF objects live
in their own BVH) and a mesh with materials, some of them lights, render the same
samples as a host build, bit for bit, also after a refit; so do they with the
other build mode's scene built first in the same context."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, configs
from aperturerendererv3_gb300._lib import OBJECT_CUBE, OBJECT_SDF, OBJECT_SPHERE
from aperturerendererv3_gb300.scene import Material, SceneObject, TriangleMesh, sdf

pytestmark = pytest.mark.gpu

ORIGIN, DIRECTION = (0.5, 0.5, 3.0), (0.0, 0.0, -1.0)


def _objects(kinds):
    grey, red = Material.CreateDiffusePureColor((0.6, 0.6, 0.6)), Material.CreateDiffusePureColor((0.8, 0.2, 0.1))
    every = {
        "light": SceneObject((0.5, 1.4, 0.5), (0.3, 0.02, 0.3), Material.CreateLight((9.0, 8.0, 7.0)), (0.0, 0.0, 0.0), OBJECT_CUBE),
        "torus": SceneObject((0.3, 0.2, 0.9), (0.2, 0.2, 0.2), red, (20.0, 30.0, 0.0), OBJECT_SDF,
                             additionalObjectInfo=sdf.CreateTorus()),
        "sphere": SceneObject((0.7, 0.6, 0.8), (0.15, 0.15, 0.15), grey, (0.0, 0.0, 0.0), OBJECT_SPHERE),
        "triangle": SceneObject.Triangle((-1.0, -0.3, -1.0), (2.0, -0.3, -1.0), (0.5, -0.3, 2.0), red),
    }
    return [every[k] for k in kinds]


def _mesh(n, seed):
    tris = configs.random_triangles(n, seed=seed)
    v = tris.reshape(-1, 3).astype(np.float32)
    mats = [Material.CreateDiffusePureColor((0.3, 0.7, 0.5)), Material.CreateLight((2.0, 2.0, 1.0)),
            Material.CreateGGXPureColor((0.8, 0.5, 0.3), 0.3, 0.0, 0.5)]
    return TriangleMesh(v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3),
                        np.random.default_rng(seed).integers(0, 3, n).astype(np.int32), mats)


def _image(r):
    return r.Render((61, 47), ORIGIN, DIRECTION, 2, fov=50.0, max_depth=5)


@pytest.mark.parametrize("kinds", [(), ("light",), ("torus", "light", "sphere"), ("sphere", "torus", "triangle", "light")])
@pytest.mark.parametrize("n", [0, 1, 3, 4, 255, 257, 4097])
def test_gpu_built_scene_renders_like_the_host_built_one(cuda_device, kinds, n):
    objs, mesh = _objects(kinds), _mesh(n, 11 + n) if n else None
    if not objs and mesh is None:
        return
    made = []
    for mode in ("host", "gpu"):
        r = SceneRenderer(objs, mesh=mesh)
        r.set_build_mode(mode)
        made.append(r)
    host, gpu = made
    first = _image(host)
    assert np.array_equal(first, _image(gpu))
    assert gpu.stats()["slots"] == host.stats()["slots"] and gpu.error_word() == 0
    if mesh is not None:
        v = (np.asarray(mesh.vertices) * np.float32(0.9) + np.float32(0.03)).astype(np.float32)
        for r in made:
            r.refit_mesh(v)
        assert np.array_equal(_image(host), _image(gpu))
        gpu.mesh, host.mesh = mesh, mesh
    host.set_build_mode("gpu")
    gpu.set_build_mode("host")
    assert np.array_equal(first, _image(host)) and np.array_equal(first, _image(gpu))
