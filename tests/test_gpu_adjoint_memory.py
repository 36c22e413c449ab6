"""The vertex records of ar_adjoint (8 bytes per path of a wave and depth) are
released when a render makes larger waves: the context then holds what one that
never took a gradient holds, apart from the gradient's small buffers."""
import pytest

from aperturerendererv3_gb300 import SceneRenderer, configs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CAM = configs.CORNELL_CAMERA


def _used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def _held(gradient):
    objs, mesh, tex = configs.textured_cornell(configs.cornell_textures(8, seed=11))
    r = SceneRenderer(objs, mesh=mesh, textures=tex)
    r.build()
    before = _used()
    if gradient:
        d = torch.ones((64, 64, 3), dtype=torch.float32, device="cuda")
        g = torch.empty(r.texel_count(), dtype=torch.float64, device="cuda")
        # 65,536 paths at a limit of 1000: 524 MB of records
        r.adjoint(d, g, (64, 64), CAM["origin"], CAM["direction"], 16, fov=CAM["fov"], max_depth=1000)
        assert _used() - before > 500 << 20
    r.Render((512, 512), CAM["origin"], CAM["direction"], 4, fov=CAM["fov"], max_depth=8)
    held = _used() - before
    r.close()
    return held


def test_records_are_released_with_the_waves(cuda_device):
    _held(True)  # the process's first use of the kernels: their code and local memory stay with it
    assert _held(False) > 64 << 20
    assert abs(_held(True) - _held(False)) < 64 << 20
