"""What the library keeps for later builds is in use while it runs and given back by rgl_cleanup."""
import numpy as np
import pytest

from tests.test_gpu_collapse import cast, down_rays

pytestmark = pytest.mark.gpu


def scan_soup(rgl, triangles):
    v = np.random.default_rng(4).uniform(-10, 10, (3 * triangles, 3)).astype(np.float32)
    rgl.entity_create(rgl.mesh_create(v, np.arange(3 * triangles, dtype=np.int32).reshape(triangles, 3)))
    cast(rgl, down_rays(np.zeros((64, 2), np.float32), np.float32(20.0)))


def test_cleanup_gives_everything_back(rgl):
    import torch

    def cleanup():
        rgl.check(rgl.lib().rgl_cleanup())
        rgl.check(rgl.lib().rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))

    scan_soup(rgl, 3000)  # loads the kernels
    cleanup()
    before = torch.cuda.mem_get_info()[0]
    triangles = 400_000  # 36 bytes of vertices, 12 of indices, 128 of the tree's storage each
    scan_soup(rgl, triangles)
    assert before - torch.cuda.mem_get_info()[0] > 176 * triangles
    cleanup()
    assert abs(before - torch.cuda.mem_get_info()[0]) < 8 << 20
