"""Paths inside an object (the camera in a room, the SDF union in glass) count as inside
the last surface they left, which may be a mesh triangle or the SDF union as well
as an entry of the object table.  A mesh renders as the same triangles given one by one as objects, bit for
bit, and paths traced to their end in one launch as those traced depth by depth."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, TriangleMesh, configs
from aperturerendererv3_gb300._lib import OBJECT_CUBE, OBJECT_SDF, OBJECT_SPHERE
from aperturerendererv3_gb300.scene import Material, SceneObject, SdfUnion, sdf

pytestmark = pytest.mark.gpu

GREY = Material.CreateDiffusePureColor((0.7, 0.6, 0.5))
RED = Material.CreateDiffusePureColor((0.8, 0.2, 0.1))
LIGHT = Material.CreateLight((9.0, 9.0, 9.0))
GLASS = Material.CreateGlassPureColor((0.9, 1.0, 0.9), 1.5, 1.0)

ROOMS = {"room": SceneObject((0.0, 0.0, 0.0), (2.0, 2.0, 2.0), GREY, (0.0, 0.0, 0.0), OBJECT_CUBE),
         "glass": SceneObject((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), GLASS, (0.0, 0.0, 0.0), OBJECT_SPHERE)}
KW = dict(fov=70.0, max_depth=6)
VIEW = ((0.1, 0.05, 0.3), (0.0, 0.0, -1.0))


def _scene(room, as_mesh, union, torus, n=300):
    objs = [ROOMS[room], SceneObject((0.0, 0.6, 0.0), (0.2, 0.02, 0.2), LIGHT, (0.0, 0.0, 0.0), OBJECT_CUBE)]
    if torus:
        objs.append(SceneObject((-0.4, -0.3, -0.4), (0.4, 0.4, 0.4), RED, (20.0, 0.0, 10.0), OBJECT_SDF, sdf.CreateTorus(1.0)))
    v = 1.2 * configs.random_triangles(n, seed=2).reshape(n, 3, 3) - np.float32(0.6)
    mesh = None
    if as_mesh:
        mesh = TriangleMesh(v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), np.zeros(n, np.int32), [RED])
    else:
        objs += [SceneObject.Triangle(*t, RED) for t in v.tolist()]
    blobs = SdfUnion([(0, (0.3, 0.0, -0.3), (0.2, 0.2, 0.2)), (1, (0.3, 0.25, -0.3), (0.1, 0.1, 0.1))], 0.1, GREY) if union else None
    return SceneRenderer(objs, mesh=mesh, sdf=blobs)


@pytest.mark.parametrize("room", list(ROOMS))
@pytest.mark.parametrize("torus", [False, True])
@pytest.mark.parametrize("size,spp", [((40, 30), 4), ((420, 400), 2)])  # one launch; depth by depth, then one launch
def test_a_mesh_renders_as_its_triangles(cuda_device, room, torus, size, spp):
    mesh, single = (_scene(room, m, False, torus) for m in (True, False))
    a, b = (r.Render(size, *VIEW, spp, **KW) for r in (mesh, single))
    assert a.max() > 0 and np.array_equal(a, b)
    assert mesh.error_word() == 0


@pytest.mark.parametrize("room", list(ROOMS))
@pytest.mark.parametrize("torus", [False, True])
@pytest.mark.parametrize("union", [False, True])
@pytest.mark.parametrize("view", [VIEW, ((0.2, 0.3, 1.7), (-0.05, -0.15, -1.0))])  # from inside, and into the glass
def test_one_launch_and_depth_by_depth_agree(cuda_device, room, torus, union, view):
    r = _scene(room, True, union, torus)
    a, b = (r.Render((64, 48), *view, 4, profile=p, **KW) for p in (0, 1))
    assert a.max() > 0 and np.array_equal(a, b)
    assert r.error_word() == 0
