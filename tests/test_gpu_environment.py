"""GPU checks of the environment's sampling distribution at the sizes where
its kernels' warps and tables end (one cell, a warp's 32 columns and rows,
the tables' 2048 x 1024), with dark rows, dark columns and a dark last cell:
each path equals the oracle's, whose tables its own host code builds."""

import numpy as np
import pytest

from hydra_lotus_b200 import abi, scenes
from oracle import oracle

from parity import PathParity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height,width", [(1, 1), (1, 33), (3, 2), (31, 32), (32, 31), (33, 65), (64, 100),
                                          (1023, 2047), (1030, 2050)])
@pytest.mark.parametrize("dark", [False, True])
def test_environment_sizes(cuda, height, width, dark):
    rng = np.random.default_rng(height * 4096 + width)
    texels = rng.uniform(0.05, 1.0, (height, width, 4)).astype(np.float32) ** 4
    if dark and height * width > 1:
        texels[rng.uniform(size=height) < 0.3] = 0.0
        texels[:, rng.uniform(size=width) < 0.3] = 0.0
        texels[-1, -1] = 0.0
        texels[0, 0] = 3.0
    scene = scenes.Scene("environment")
    m = scene.add_material(scenes.preview_material((0.7, 0.6, 0.5), roughness=0.4, ior=1.5))
    scene.add_instance(scene.add_geometry(*scenes.quad([[-1, -1, 1], [1, -1, 1], [1, -1, -1], [-1, -1, -1]])), m)
    scene.set_environment(texels, (1.0, 0.9, 0.8))
    scene.world_to_clip = scenes.cornell_camera()
    scene.width = scene.height = 32
    st = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS,
                              max_bounces=3, sample_index=5)
    frame = scene.frame(st, frame_count=1)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        res, color = r.render_scene(frame)
        cuda.check(res, "render_scene")
    want, _ = oracle.OracleScene(scene).sample(frame, 5)
    PathParity(color, want).assert_ok()
