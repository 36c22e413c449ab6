"""Per-pixel sums: straight from the path state, or from the stored samples that
per-sample output asks for.  Both add the same floats in sample order, so the
images are equal bit for bit, and equal to the samples' own mean taken in that
order, whatever the blocks of samples, the ragged last pixels and the waves
(which end inside a pixel here)."""
import numpy as np
import pytest

from aperturerendererv3_gb300 import SceneRenderer, configs

pytestmark = pytest.mark.gpu
CAM = configs.CORNELL_CAMERA


@pytest.mark.parametrize("size", [(1, 1), (33, 1), (31, 29), (64, 32)])
@pytest.mark.parametrize("spp", [1, 5, 32, 33, 70])
@pytest.mark.parametrize("wave", [0, 997])
def test_sums_of_samples(cuda_device, size, spp, wave):
    r = SceneRenderer(configs.cornell_triangles())
    kw = dict(fov=CAM["fov"], max_depth=3, wave_paths=wave)
    a = r.Render(size, CAM["origin"], CAM["direction"], spp, **kw)
    b, samples = r.Render(size, CAM["origin"], CAM["direction"], spp, per_sample=True, **kw)
    assert np.array_equal(a, b)
    total = np.zeros_like(a)
    for s in np.asarray(samples, np.float32).reshape(spp, *a.shape):
        total += s.astype(np.float64)
    assert np.allclose(a, total / spp, rtol=4e-16, atol=0)  # one multiply or one division at the end
