"""GPU checks of RenderScene's waves: however a call's samples are split into
wavefronts (large waves on small targets, smaller ones for what is left over,
chains with two in flight), the accumulated image is the one that one sample
at a time gives, bit for bit."""

import numpy as np
import pytest

from hydra_lotus_b200 import abi, scenes

pytestmark = pytest.mark.gpu


def render(cuda, r, scene, spp, integrator, first=0):
    st = abi.default_settings(integrator=integrator, light_sampling=abi.LIGHT_SAMPLING_MIS, max_bounces=5,
                              sample_index=first)
    res, color = r.render_scene(scene.frame(st, frame_count=spp))
    cuda.check(res, "render_scene")
    assert res.samples_per_pixel == spp
    return color


# 32 and 33 samples: waves of eight, then two of sixteen; 77 and 259: waves
# with 13 and 3 samples left over; 256 and more: waves of 64.
@pytest.mark.parametrize("size", [33, 96])
@pytest.mark.parametrize("spp", [2, 13, 32, 33, 77, 256, 259])
def test_waves_match_one_sample_at_a_time(cuda, size, spp):
    scene = scenes.box_room(seed=3, size=size)
    with cuda.CudaOffscreenRenderer(0, samples_per_wave=1) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        want = render(cuda, r, scene, spp, abi.INTEGRATOR_WAVEFRONT)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        for integrator in (abi.INTEGRATOR_WAVEFRONT, abi.INTEGRATOR_REFERENCE):
            assert np.array_equal(render(cuda, r, scene, spp, integrator), want)


def test_targets_in_turn(cuda):
    """Another target size in between moves the targets, a longer call the
    path state: neither leaves a captured graph with the old arrays."""
    small, large = scenes.box_room(seed=3, size=48), scenes.box_room(seed=3, size=80)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(small), "update_scene")
        first = [render(cuda, r, small, 16, abi.INTEGRATOR_WAVEFRONT), render(cuda, r, large, 1, abi.INTEGRATOR_WAVEFRONT),
                 render(cuda, r, small, 64, abi.INTEGRATOR_WAVEFRONT)]
        again = [render(cuda, r, small, 16, abi.INTEGRATOR_WAVEFRONT, first=64),
                 render(cuda, r, small, 16, abi.INTEGRATOR_WAVEFRONT),
                 render(cuda, r, large, 1, abi.INTEGRATOR_WAVEFRONT), render(cuda, r, small, 64, abi.INTEGRATOR_WAVEFRONT)]
    for a, b in zip(first, again[1:]):
        assert np.array_equal(a, b)
