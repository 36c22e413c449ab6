"""Scenes of opaque surfaces run shading instantiations without the glass and
medium code; a glass object anywhere selects the full one.  With a glass cube too
small to be hit, inside an opaque box, both render the same samples bit for bit,
unguided, guided from the same saved probes, and textured; the gradients differ
only in the order of their float sums."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, configs
from aperturerendererv3_gb300._lib import OBJECT_CUBE
from aperturerendererv3_gb300.scene import Material, SceneObject

pytestmark = pytest.mark.gpu

CAM = configs.CORNELL_CAMERA


def _sealed_glass():
    # inside the tall box; a path in some 500,000 slips in at an edge and meets a
    # cube of 0.01
    return SceneObject((-0.17, -0.2, -0.15), (1.0e-6, 1.0e-6, 1.0e-6),
                       Material.CreateGlassPureColor((0.9, 1.0, 0.9), 1.5, 1.0), (0.0, 0.0, 0.0), OBJECT_CUBE)


def _pair(textured):
    out = []
    for extra in ([], [_sealed_glass()]):
        if textured:
            objs, mesh, tex = configs.textured_cornell(configs.cornell_textures(8, seed=11))
            out.append(SceneRenderer(objs + extra, mesh=mesh, textures=tex))
        else:
            out.append(SceneRenderer(configs.cornell_triangles() + extra))
    return out


SIZES = [((1, 1), 1), ((33, 31), 2), ((421, 397), 3)]  # the last is above the one-kernel form


@pytest.mark.parametrize("size,spp", SIZES)
@pytest.mark.parametrize("textured", [False, True])
def test_opaque_forms_equal_the_full_one(cuda_device, textured, size, spp):
    kw = dict(fov=CAM["fov"], max_depth=9)
    a, b = (r.Render(size, CAM["origin"], CAM["direction"], spp, **kw) for r in _pair(textured))
    assert np.array_equal(a, b)


@pytest.mark.parametrize("size,spp", SIZES)
def test_guided_opaque_form_equals_the_full_one(cuda_device, size, spp):
    lean, full = _pair(False)
    kw = dict(fov=CAM["fov"], max_depth=9, guide=1)
    lean.Render((96, 96), CAM["origin"], CAM["direction"], 4, **kw)
    p = lean.guide_probes()
    out = []
    for r in (lean, full):
        r.set_guide_probes(p["keys"], p["texels"], p["counts"])
        out.append(r.Render(size, CAM["origin"], CAM["direction"], spp, first_frame=64, guide_frames=spp, **kw))
    assert np.array_equal(*out)


@pytest.mark.parametrize("size,spp", SIZES[1:2])
def test_replay_gradients_of_both_forms(cuda_device, size, spp):
    """At most 1023 x 2 x 9 = 18414 vertices over 8 textures of 64 texels; no texel
    takes more than 3000 of them, so any order of its float sum stays within
    3000 x 2^-24 = 1.8e-4 of the sum of its magnitudes.  The weights are one sign."""
    import torch
    grads = []
    for r in _pair(True):
        d = torch.ones((size[1], size[0], 3), dtype=torch.float32, device="cuda")
        g = torch.empty(r.texel_count(), dtype=torch.float64, device="cuda")
        r.adjoint(d, g, size, CAM["origin"], CAM["direction"], spp, fov=CAM["fov"], max_depth=9)
        grads.append(g.cpu().numpy())
    assert np.abs(grads[0]).max() > 0
    assert np.abs(grads[0] - grads[1]).max() <= 1.8e-4 * np.abs(grads[0]).max()


@pytest.mark.parametrize("size,spp", [((33, 32), 2), ((421, 397), 3)])
@pytest.mark.parametrize("glass", [False, True])
def test_recorded_gradients_equal_the_replayed_ones(cuda_device, size, spp, glass):
    """A wave whose records (paths x depth limit) would pass 2^27 is replayed: limit
    65535 here, 255 is recorded.  Roulette ends every path before 255 (the images
    are equal), so the gradients differ only in the order of their float sums.  A
    texel of the small image takes at most 3000 records: 3000 x 2^-24 = 1.8e-4.  Of
    the large one (501411 paths of about four vertices over 512 texels) a texel
    takes some 4000 on average, 20 times that at most, whose rounding errors of
    either sign give sqrt(80000) x 2^-24 = 1.7e-5.  2e-4 covers both."""
    import torch
    r = _pair(True)[int(glass)]
    grads, images = [], []
    for depth in (255, 65535):
        kw = dict(fov=CAM["fov"], max_depth=depth)
        images.append(r.Render(size, CAM["origin"], CAM["direction"], spp, **kw))
        d = torch.ones((size[1], size[0], 3), dtype=torch.float32, device="cuda")
        g = torch.empty(r.texel_count(), dtype=torch.float64, device="cuda")
        r.adjoint(d, g, size, CAM["origin"], CAM["direction"], spp, **kw)
        grads.append(g.cpu().numpy())
    assert np.array_equal(*images)
    assert np.abs(grads[0] - grads[1]).max() <= 2e-4 * np.abs(grads[1]).max()
