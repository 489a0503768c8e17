"""The host copy of a large scene's positions and triangles is given back when
a small scene takes its place."""

import os

import pytest

from hydra_lotus_b200 import scenes

pytestmark = pytest.mark.gpu


def resident_bytes():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGESIZE")


def test_large_scene_then_small(cuda):
    large, small = scenes.grid_mesh(quads=2048), scenes.box_room(seed=0, size=64)
    positions, triangles = large.geometries[0][0], large.geometries[0][1]
    copy = positions.nbytes + triangles.nbytes
    assert copy > 128 << 20
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(large), "update_scene")
        held = resident_bytes()
        cuda.check(r.update_scene(small), "update_scene")
        assert held - resident_bytes() > 0.8 * copy
        # The same room again, and back to the large scene.
        cuda.check(r.update_scene(small), "update_scene")
        cuda.check(r.update_scene(large), "update_scene")
