"""GPU checks of RenderScene's captured graphs. The first launch of a shape
goes to the streams directly, the second is captured and from the third on the
graph is replayed: each gives the image of one sample at a time, bit for bit,
and a graph is not replayed over arrays that have moved since its capture. The
rounds are fixed, so that every call of a shape launches the same keys."""

import numpy as np
import pytest

from hydra_lotus_b200 import abi, scenes

pytestmark = pytest.mark.gpu

SMALL, LARGE = 48, 80


def render(cuda, r, scene, spp, first):
    """A call whose `first` sample differs from the one before resets the
    accumulation, so that each renders an image of its own."""
    st = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS, max_bounces=5,
                              sample_index=first)
    res, color = r.render_scene(scene.frame(st, frame_count=spp))
    cuda.check(res, "render_scene")
    assert res.samples_per_pixel == spp
    return color


@pytest.fixture(scope="module")
def rooms():
    return {size: scenes.box_room(seed=3, size=size) for size in (SMALL, LARGE)}


def play(cuda, rooms, calls, **options):
    with cuda.CudaOffscreenRenderer(0, wavefront_rounds=4, **options) as r:
        cuda.check(r.update_scene(rooms[SMALL]), "update_scene")
        return [render(cuda, r, rooms[size], spp, first) for size, spp, first in calls]


def check(cuda, rooms, calls):
    # Each call's own image: a new renderer, one sample at a time.
    want = {call: play(cuda, rooms, [call], samples_per_wave=1)[0] for call in set(calls)}
    for call, image in zip(calls, play(cuda, rooms, calls)):
        assert np.array_equal(image, want[call]), call


# One sample, a chain of waves, and waves with samples left over.
@pytest.mark.parametrize("spp", [1, 13, 16, 33])
def test_direct_capture_replay(cuda, rooms, spp):
    check(cuda, rooms, [(SMALL, spp, 100 * k) for k in range(5)])


@pytest.mark.parametrize("spp", [1, 16])
@pytest.mark.parametrize("between", [
    (LARGE, 1),    # another target: the images move
    (SMALL, 64),   # a longer call: the path state and queues of both waves move
    (LARGE, 64)])  # both
def test_replay_after_arrays_move(cuda, rooms, spp, between):
    size, samples = between
    replayed = [(SMALL, spp, 100 * k) for k in range(4)]
    check(cuda, rooms, replayed + [(size, samples, 1000)] + [(SMALL, spp, 2000 + 100 * k) for k in range(4)])


def test_more_shapes_than_graphs(cuda, rooms):
    """More keys than the renderer keeps graphs of, each launched again after
    its graph was given up."""
    shapes = [(SMALL, spp) for spp in (1, 2, 4, 8, 16, 24, 32, 64)] + [(LARGE, 8)]
    calls = [(size, spp, 1000 * turn + 100 * k) for turn in range(4) for k, (size, spp) in enumerate(shapes)]
    check(cuda, rooms, calls)
