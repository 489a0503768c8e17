"""GPU checks of what RenderScene's path state and queues hold on to: a large
call's arrays are given back when the renderer turns to a small target, small
targets in turn keep theirs, and neither changes an image."""

import numpy as np
import pytest

from hydra_lotus_b200 import abi, scenes

pytestmark = pytest.mark.gpu

BYTES_PER_PATH = 164
WAVE_PATHS = 1 << 21


def free_bytes():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def render(cuda, r, scene, spp, first=0):
    st = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS,
                              max_bounces=2, sample_index=first)
    res, color = r.render_scene(scene.frame(st, frame_count=spp))
    cuda.check(res, "render_scene")
    return color


@pytest.mark.parametrize("preview_spp", [1, 64])
def test_large_call_then_preview(cuda, preview_spp):
    large, preview = scenes.box_room_wide(seed=0, width=1600, height=1200), scenes.box_room(seed=0, size=64)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(large), "update_scene")
        want = render(cuda, r, preview, preview_spp)
        before = free_bytes()
        # Waves of eight, two in flight.
        image = render(cuda, r, large, 16)
        held = before - free_bytes()
        sets = 2 * 8 * large.width * large.height * BYTES_PER_PATH
        assert held > 0.9 * sets
        assert np.array_equal(render(cuda, r, preview, preview_spp), want)
        kept = before - free_bytes()
        # At most two sets of kWavePaths stay, beside what the targets' own arrays differ by.
        assert kept <= 2 * WAVE_PATHS * BYTES_PER_PATH + (64 << 20)
        assert np.array_equal(render(cuda, r, large, 16), image)


def test_small_targets_in_turn_keep_their_arrays(cuda):
    """A target that needs less than kWavePaths paths leaves the arrays where
    they are: the path state of the larger of the two stays allocated."""
    small, other = scenes.box_room(seed=0, size=256), scenes.box_room(seed=0, size=64)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(small), "update_scene")
        image = render(cuda, r, small, 64)
        before = free_bytes()
        render(cuda, r, other, 1)
        assert abs(free_bytes() - before) < (64 << 20)
        assert np.array_equal(render(cuda, r, small, 64), image)


def test_large_waves_need_not_fit(cuda):
    """Where the device has no memory for two waves of 2^21 paths, a call that
    waves of eight samples fit runs in those, to the same image."""
    import torch

    scene = scenes.box_room(seed=0, size=256)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        want = render(cuda, r, scene, 64)
    large, default = 2 * WAVE_PATHS * BYTES_PER_PATH, 2 * 8 * scene.width * scene.height * BYTES_PER_PATH
    left = (large + default) // 2  # 430 MB
    filler = None
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        try:
            filler = torch.empty(free_bytes() - left, dtype=torch.uint8, device="cuda:0")
            assert default < free_bytes() < large
            images = [render(cuda, r, scene, 64), render(cuda, r, scene, 64, first=64), render(cuda, r, scene, 64)]
        finally:
            del filler
            torch.cuda.empty_cache()
        images.append(render(cuda, r, scene, 64, first=128))
        images.append(render(cuda, r, scene, 64))
    assert np.array_equal(images[0], want) and np.array_equal(images[2], want) and np.array_equal(images[4], want)
