"""GPU checks of the SAH builder at the sizes where its kernels hand over
(a warp's 32 primitives, the medium subtrees' 512, the blocks above), with
coincident centroids and every leaf size: each path equals the oracle's,
whose BVH is its own."""

import numpy as np
import pytest

from hydra_lotus_b200 import abi, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def soup(triangles, seed=0, size=24, coincident=False, instances=1):
    """A seeded cloud of small triangles (or copies of a few of them), lit by
    a constant sky, over a floor."""
    rng = np.random.default_rng(seed)
    distinct = max(1, triangles // 40) if coincident else triangles
    centre = rng.uniform(-0.8, 0.8, (distinct, 1, 3))
    corners = (centre + rng.uniform(-1.0, 1.0, (distinct, 3, 3)) * 0.4 / max(1.0, distinct ** (1.0 / 3.0)))
    corners = corners[np.arange(triangles) % distinct]
    s = scenes.Scene(f"soup-{triangles}")
    g = s.add_geometry(corners.reshape(-1, 3), np.arange(3 * triangles).reshape(-1, 3))
    m = s.add_material(scenes.preview_material((0.7, 0.5, 0.4), ior=1.0))
    for k in range(instances):
        offset = (0.0, 0.0, 0.0) if k == 0 else tuple(rng.uniform(-1.0, 1.0, 3))
        s.add_instance(g, m, scenes.affine(np.eye(3) * (1.0 if instances == 1 else 0.2), offset))
    s.add_instance(s.add_geometry(*scenes.quad([[-1, -1, 1], [1, -1, 1], [1, -1, -1], [-1, -1, -1]])), m)
    s.environment_constant = (0.6, 0.7, 0.9)
    s.world_to_clip = scenes.cornell_camera()
    s.width = s.height = size
    return s


def check(cuda, scene, **options):
    st = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_BSDF,
                              max_bounces=3, sample_index=5)
    frame = scene.frame(st, frame_count=1)
    with cuda.CudaOffscreenRenderer(0, **options) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        res, color = r.render_scene(frame)
        cuda.check(res, "render_scene")
    want, _ = oracle.OracleScene(scene).sample(frame, 5)
    assert np.array_equal(color[..., :3], want[..., :3])


@pytest.mark.parametrize("coincident", [False, True])
@pytest.mark.parametrize("triangles", [1, 2, 3, 31, 32, 33, 511, 512, 513, 1100, 5000])
def test_mesh_sizes(cuda, triangles, coincident):
    check(cuda, soup(triangles, seed=triangles, coincident=coincident))


@pytest.mark.parametrize("leaf", [2, 3, 8])
@pytest.mark.parametrize("triangles", [2, 8, 9, 33, 700])
def test_leaf_sizes(cuda, triangles, leaf):
    check(cuda, soup(triangles, seed=triangles), bvh_leaf_size=leaf)


@pytest.mark.parametrize("instances", [2, 31, 32, 520])
def test_instance_counts(cuda, instances):
    check(cuda, soup(12, seed=instances, instances=instances))


def test_point_edit_with_larger_leaves(cuda):
    """A refit of a tree whose leaves leave node slots unused."""
    before, after = soup(700, seed=1), soup(700, seed=2)
    after.geometries[0] = (after.geometries[0][0], before.geometries[0][1], None)
    st = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_BSDF, max_bounces=3)
    images = []
    for edit in (True, False):
        with cuda.CudaOffscreenRenderer(0, bvh_leaf_size=4) as r:
            cuda.check(r.update_scene(before if edit else after), "update_scene")
            if edit:
                cuda.check(r.update_geometry(after, 0), "update_geometry")
            res, color = r.render_scene(after.frame(st, frame_count=2))
            cuda.check(res, "render_scene")
            images.append(color)
    assert np.array_equal(images[0], images[1])
