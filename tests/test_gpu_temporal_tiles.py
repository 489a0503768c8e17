"""GPU checks of the temporal passes' pixel tiles (16 x 8 to a block) on
frames smaller than a tile and with ragged edges: surface metadata and
reservoirs equal the oracle's bit for bit, and the last filter iteration,
from its own input and guides, equals a float64 restatement."""

import numpy as np
import pytest

from hydra_lotus_b200 import abi, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -24


def frames(width, height, count, iterations):
    settings = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT,
                                    light_sampling=abi.LIGHT_SAMPLING_RESTIR_INITIAL, max_bounces=2,
                                    sample_index=40, restir_candidates=4, restir_temporal=1,
                                    restir_max_history_candidates=20, restir_spatial=1, restir_spatial_radius=2)
    previous = None
    for k in range(count):
        view, w2c = scenes.orbit_camera(k, frames=24, aspect=width / height)
        frame = abi.make_frame(w2c, width, height, settings, 1)
        yield abi.temporal_desc(frame, view, previous[0] if previous else None, previous[1] if previous else None,
                                history_available=k > 0, accumulate_radiance=True, max_history_samples=6,
                                filter_iterations=iterations)
        previous = (view, w2c)


def exact(a, b):
    return a.tobytes() == b.tobytes()


SIZES = [(1, 1), (3, 17), (16, 8), (17, 9), (15, 7), (65, 33)]


@pytest.mark.parametrize("width,height", SIZES)
def test_reservoirs(cuda, width, height):
    scene = scenes.restir_room(seed=0, size=height, emitters=40, aspect=width / height)
    o = oracle.OracleTemporalScene(scene)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        for k, d in enumerate(frames(width, height, 2, 0)):
            res, _ = r.render_temporal(d)
            cuda.check(res, "render_temporal")
            p = {n: r.read_product(getattr(abi, "PRODUCT_" + n.upper()), height, width)
                 for n in ("surface", "validity", "restir_initial", "restir_temporal", "restir_previous",
                           "restir_surfaces", "restir_previous_surfaces", "restir_spatial", "restir_sources")}
            tc, si = oracle.oracle_temporal(d), d.frame.settings.sample_index + k
            assert exact(p["surface"], o.temporal_surface(d.frame, tc))
            assert exact(p["restir_initial"], o.restir_initial(d.frame, tc, si))
            reuse, surfaces = o.restir_temporal(d.frame, tc, si, p["restir_initial"], p["validity"], p["surface"],
                                                p["restir_previous"], p["restir_previous_surfaces"])
            assert exact(p["restir_temporal"], reuse)
            assert exact(p["restir_surfaces"], surfaces)
            spatial, sources = o.restir_spatial(d.frame, tc, si, p["restir_temporal"], p["restir_surfaces"])
            assert exact(p["restir_spatial"], spatial)
            assert np.array_equal(p["restir_sources"], sources)


def unpack_normals(packed):
    e = np.stack([packed.astype(np.uint32).astype(np.uint16).view(np.int16),
                  (packed >> 16).astype(np.uint16).view(np.int16)], -1)
    e = np.maximum(e.astype(np.float64) / 32767.0, -1.0)
    z = 1.0 - np.abs(e).sum(-1)
    fold = np.maximum(-z, 0.0)[..., None]
    n = np.concatenate([e + np.where(e >= 0.0, -fold, fold), z[..., None]], -1)
    return n / np.linalg.norm(n, axis=-1, keepdims=True)


def filter_iteration(planes, iteration):
    """The a-trous iteration in float64 from the filter's planes (two of
    values, then the guides), and each value's error bound in FP32: a tap's
    weight carries 128 times its normals' dot product's rounding (3.5 units,
    and 4 of each normal), the two luminances' (4 units each, over phi_l), 8
    units of the exponent's argument and 16 of its own; a weighted mean then
    moves by at most twice the weights' mean error, and 32 units of its own
    sums."""
    values, guide = planes[iteration & 1].astype(np.float64), planes[2]
    bits = np.ascontiguousarray(guide).view(np.uint32)
    normals = unpack_normals(bits[..., 3])
    ids = bits[..., 0].astype(np.uint64) | bits[..., 1].astype(np.uint64) << np.uint64(32)
    ok = bits[..., 2] != 0xFFFFFFFF
    depth = np.where(ok, guide[..., 2], 0.0).astype(np.float64)
    lum = values[..., :3] @ np.array([0.2126, 0.7152, 0.0722], np.float32).astype(np.float64)
    h, w = ok.shape
    step = 1 << iteration
    out, bound = np.zeros((h, w, 3)), np.zeros((h, w, 3))

    def near(y, x, y2, x2):
        return 0 <= y2 < h and 0 <= x2 < w and ok[y2, x2] and ids[y2, x2] == ids[y, x]

    for y in range(h):
        for x in range(w):
            if not ok[y, x]:
                continue
            g = gw = 0.0
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if near(y, x, y + dy, x + dx):
                        k = (0.5 if dx == 0 else 0.25) * (0.5 if dy == 0 else 0.25)
                        g, gw = g + k * values[y + dy, x + dx, 3], gw + k
            phi_l = 4.0 * np.sqrt(max(g / gw, 0.0) + 1e-10)
            phi_z = 0.0
            for a, b in (((y, x - 1), (y, x + 1)), ((y - 1, x), (y + 1, x))):
                steps = [abs(depth[y, x] - depth[q]) for q in (a, b) if near(y, x, *q)]
                phi_z += min(steps) if steps else 0.0
            phi_z = max(phi_z, 1e-8)
            total, sums, errors = 0.0, np.zeros(3), np.zeros(3)
            for ty in range(-2, 3):
                for tx in range(-2, 3):
                    y2, x2 = y + ty * step, x + tx * step
                    if not near(y, x, y2, x2):
                        continue
                    weight, eps = (0.375, 0.25, 0.0625)[abs(tx)] * (0.375, 0.25, 0.0625)[abs(ty)], 0.0
                    if tx or ty:
                        wz = abs(depth[y, x] - depth[y2, x2]) / (phi_z * step * np.hypot(tx, ty))
                        wl = abs(lum[y, x] - lum[y2, x2]) / phi_l
                        facing = min(max(normals[y, x] @ normals[y2, x2], 0.0), 1.0)
                        weight *= np.exp(-(wl + wz)) * facing ** 128
                        eps = ULP * (128 * 11.5 + 4 * (lum[y, x] + lum[y2, x2]) / phi_l + 8 * (wl + wz) + 16)
                    total += weight
                    sums += weight * values[y2, x2, :3]
                    errors += weight * min(eps, 1.0) * np.maximum(np.abs(values[y2, x2, :3]), np.abs(values[y, x, :3]))
            out[y, x] = sums / total
            bound[y, x] = 2.0 * errors / total + 32 * ULP * np.abs(out[y, x])
    return out, bound


@pytest.mark.parametrize("iterations", [1, 2, 5])
@pytest.mark.parametrize("width,height", SIZES)
def test_filter(cuda, width, height, iterations):
    scene = scenes.restir_room(seed=1, size=height, emitters=40, aspect=width / height)
    with cuda.CudaOffscreenRenderer(0) as r:
        cuda.check(r.update_scene(scene), "update_scene")
        for d in frames(width, height, 2, iterations):
            res, color = r.render_temporal(d)
            cuda.check(res, "render_temporal")
            planes = r.read_product(abi.PRODUCT_FILTER, height, width).reshape(3, height, width, 4)
            surface = r.read_product(abi.PRODUCT_SURFACE, height, width)
            radiance = r.read_product(abi.PRODUCT_RADIANCE, height, width)
            want, bound = filter_iteration(planes, iterations - 1)
            packed = surface["albedo"][..., None] >> np.array([0, 8, 16], np.uint32) & 255
            albedo = packed / 255.0
            scale = np.where(albedo > 0.0, albedo, 1.0)
            hit = radiance["sample_count"] != 0
            assert np.array_equal(color[~hit], radiance["color"][~hit])
            error = np.abs(color[..., :3] - want * scale)
            assert np.all(error[hit] <= (bound * scale + 8 * ULP * np.abs(want * scale))[hit])
