"""The performance cases of this framework: the calls its users make, at the
sizes they make them, each through the public Python host (which binds the C
ABI one call to one entry point).

Rendering cases return the image the call hands back in host memory (a pinned
buffer the program keeps, as a viewport or an image writer does). Scenes are
the repository's seeded procedural ones; where a scene has no seed of its own
(the fixtures with fixed geometry), the seed picks the range of sample indices
that the frames draw, so that every seed follows other paths.
"""

import math

import numpy as np
import torch

from hydra_lotus_b200 import abi, renderer, scenes

# Radiance-cache network: six layers, the last 16 columns wide.
_LAYERS = ((64, 64),) * 5 + ((64, 16),)
_SAMPLING = {"mis": abi.LIGHT_SAMPLING_MIS, "bsdf": abi.LIGHT_SAMPLING_BSDF}
_INTEGRATOR = {"wavefront": abi.INTEGRATOR_WAVEFRONT, "reference": abi.INTEGRATOR_REFERENCE}


def listed():
    return [
        # An interactive viewport's frame on a tiny scene: launches and the
        # latency of the longest path are all there is.
        {"name": "cornell_128_reference", "path": "frame", "scene": "cornell", "width": 128, "height": 128,
         "integrator": "reference", "sampling": "bsdf", "spp": 1, "bounces": 64, "detail": 0},
        # A headless render of a small image: many samples in one call.
        {"name": "room_256_64spp", "path": "frame", "scene": "room", "width": 256, "height": 256,
         "integrator": "wavefront", "sampling": "mis", "spp": 64, "bounces": 6, "detail": 0},
        # The benchmark's scene: millions of instanced triangles, an
        # importance-sampled sky, conductors and glass, a final-frame call.
        {"name": "field_720p_16spp", "path": "frame", "scene": "field", "width": 1280, "height": 720,
         "integrator": "wavefront", "sampling": "mis", "spp": 16, "bounces": 8, "detail": 320},
        # A progressive viewport over many analytic lights, deep paths.
        {"name": "lights_512_progressive", "path": "frame", "scene": "lights", "width": 512, "height": 512,
         "integrator": "wavefront", "sampling": "mis", "spp": 1, "bounces": 64, "detail": 16},
        # The composed glTF PBR closure, one progressive sample.
        {"name": "gltf_1024_progressive", "path": "frame", "scene": "cornell-gltf", "width": 1024, "height": 1024,
         "integrator": "wavefront", "sampling": "bsdf", "spp": 1, "bounces": 64, "detail": 0},
        # A validation render of a texture fixture: an odd image size, texture
        # lookups, the reference integrator.
        {"name": "textures_161_128spp", "path": "frame", "scene": "textures", "width": 161, "height": 161,
         "integrator": "reference", "sampling": "mis", "spp": 128, "bounces": 16, "detail": 0},
        # Real-time frames of a moving camera: ReSTIR DI with temporal and
        # spatial reuse over 10,000 emitters, SVGF with FP16 moments.
        {"name": "temporal_720p", "path": "temporal", "width": 1280, "height": 720, "emitters": 10000,
         "bounces": 6, "filter": 5, "neighbours": 5, "moments": abi.MOMENTS_FP16},
        # Progressive frames whose paths end into the radiance cache, which
        # trains as they render.
        {"name": "cache_720p", "path": "cached", "width": 1280, "height": 720, "bounces": 6, "emitters": 0},
        # The cache network's forward and backward pass on host data, as a
        # program that trains or checks the cache from outside calls it.
        {"name": "cache_gradient_32k", "path": "gradient", "records": 32768},
        # Opening a scene: upload, on-device BVH builds, light and sky tables,
        # then the first preview frame.
        {"name": "load_field", "path": "load", "scene": "field", "detail": 320, "width": 480, "height": 270},
        # Editing: a sculpted mesh's points and a moved object, each followed
        # by a preview frame.
        {"name": "edit_grid_512", "path": "edit", "quads": 512, "size": 96},
        # A batch of independent scenes rendered as one wavefront.
        {"name": "batch_16_rooms", "path": "batch", "scenes": 16, "spp": 4, "bounces": 8},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the same kinds, its sizes spread over their ranges."""
    path = rng.choice(["frame", "frame", "frame", "temporal", "cached", "gradient", "load", "edit", "batch"])
    if path == "frame":
        scene = rng.choice(["cornell", "room", "field", "lights", "cornell-gltf", "textures"])
        width = _log_uniform(rng, 96, 1280)
        height = max(64, min(1024, int(width * rng.uniform(0.5, 1.0))))
        # At most the paths of the largest listed call.
        spp = min(_log_uniform(rng, 1, 64), max(1, 14_000_000 // (width * height)))
        bounces = rng.choice([4, 6, 8, 16, 64])
        detail = {"field": rng.randint(16, 320), "lights": rng.randint(1, 20)}.get(scene, 0)
        if scene == "field":
            bounces = min(bounces, 8)
        elif scene in ("textures", "cornell-gltf"):
            spp = max(1, spp // 4)
        return {"path": path, "scene": scene, "width": width, "height": height,
                "integrator": rng.choice(["wavefront", "wavefront", "reference"]),
                "sampling": rng.choice(["mis", "mis", "bsdf"]), "spp": spp, "bounces": bounces, "detail": detail}
    if path in ("temporal", "cached"):
        width = _log_uniform(rng, 160, 1280)
        case = {"path": path, "width": width, "height": max(90, int(width * rng.uniform(0.5, 0.5625))),
                "bounces": rng.randint(2, 8), "emitters": _log_uniform(rng, 100, 10000)}
        if path == "temporal":
            case.update(filter=rng.randint(0, 5), neighbours=rng.choice([0, 0, 3, 5]),
                        moments=rng.choice([abi.MOMENTS_FP32, abi.MOMENTS_FP16]))
        return case
    if path == "gradient":
        return {"path": path, "records": _log_uniform(rng, 100, 32768)}
    if path == "load":
        width = _log_uniform(rng, 96, 480)
        scene = rng.choice(["field", "mesh", "room", "textures"])
        return {"path": path, "scene": scene, "detail": rng.randint(16, 320) if scene == "field" else rng.randint(3, 6),
                "width": width, "height": max(64, int(width * rng.uniform(0.5, 1.0)))}
    if path == "edit":
        return {"path": path, "quads": _log_uniform(rng, 16, 512), "size": rng.randint(64, 128)}
    return {"path": path, "scenes": rng.randint(2, 16), "spp": rng.randint(1, 4), "bounces": rng.randint(3, 8)}


def _first_sample(seed):
    """The first sample index of a program's frames: another range per seed."""
    return (seed * 7919) % (1 << 20)


def _scene(case, seed):
    kind, width, height, detail = case["scene"], case["width"], case["height"], case["detail"]
    if kind == "room":
        scene = scenes.box_room(seed=seed, size=width)
    elif kind == "field":
        scene = scenes.sphere_field(seed=seed, width=width, height=height, prototypes=detail)
    elif kind == "lights":
        scene = scenes.light_grid(side=detail, size=width, seed=seed)
    elif kind == "mesh":
        scene = scenes.big_mesh(seed=seed, size=width, subdivisions=detail)
    elif kind == "cornell-gltf":
        scene = scenes.cornell_gltf(size=width)
    elif kind == "textures":
        scene = scenes.material_textures(size=width)
    else:
        scene = scenes.cornell_reference(size=width)
    scene.width, scene.height = width, height
    return scene


def _host_image(width, height):
    return torch.empty((height, width, 4), dtype=torch.float32, pin_memory=True).numpy()


class _Program:
    """What a rendering program holds between calls."""


def _prepare_frame(p, case, seed):
    p.renderer = renderer.CudaOffscreenRenderer(0)
    p.scene = _scene(case, seed)
    renderer.check(p.renderer.update_scene(p.scene), "update_scene")
    settings = abi.default_settings(integrator=_INTEGRATOR[case["integrator"]],
                                    light_sampling=_SAMPLING[case["sampling"]], max_bounces=case["bounces"],
                                    sample_index=_first_sample(seed))
    p.frame = p.scene.frame(settings, frame_count=case["spp"])
    p.image = _host_image(case["width"], case["height"])


def _run_frame(p):
    result, image = p.renderer.render_scene(p.frame, p.image)
    renderer.check(result, "render_scene")
    return image


def _prepare_temporal(p, case, seed):
    p.renderer = renderer.CudaOffscreenRenderer(0)
    p.scene = scenes.box_room_wide(seed=seed, width=case["width"], height=case["height"], emitters=case["emitters"])
    renderer.check(p.renderer.update_scene(p.scene), "update_scene")
    p.settings = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT,
                                      light_sampling=abi.LIGHT_SAMPLING_RESTIR_INITIAL, max_bounces=case["bounces"],
                                      sample_index=_first_sample(seed), restir_candidates=8, restir_temporal=1,
                                      restir_max_history_candidates=20, restir_spatial=1, restir_spatial_radius=30,
                                      restir_spatial_neighbours=case["neighbours"])
    p.image = _host_image(case["width"], case["height"])
    p.index, p.previous = 0, None


def _run_temporal(p):
    case = p.case
    view, world_to_clip = scenes.orbit_camera(p.index, frames=120, aspect=case["width"] / case["height"])
    frame = abi.make_frame(world_to_clip, case["width"], case["height"], p.settings, 1)
    previous = p.previous or (None, None)
    temporal = abi.temporal_desc(frame, view, previous[0], previous[1], history_available=p.previous is not None,
                                 accumulate_radiance=True, max_history_samples=5, filter_iterations=case["filter"],
                                 moment_precision=case["moments"])
    result, image = p.renderer.render_temporal(temporal, p.image)
    renderer.check(result, "render_temporal")
    p.index, p.previous = p.index + 1, (view, world_to_clip)
    return image


def _prepare_cached(p, case, seed):
    p.renderer = renderer.CudaOffscreenRenderer(0)
    p.scene = scenes.box_room_wide(seed=seed, width=case["width"], height=case["height"], emitters=case["emitters"])
    renderer.check(p.renderer.update_scene(p.scene), "update_scene")
    p.renderer.configure_cache(enable=True, seed=1 + seed % 1000)
    settings = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS,
                                    max_bounces=case["bounces"], sample_index=_first_sample(seed))
    p.frame = p.scene.frame(settings, frame_count=1)
    p.image = _host_image(case["width"], case["height"])


def _run_cached(p):
    image = _run_frame(p)
    return {"image": image, "weights": p.renderer.cache_weights()}


def _gradient_inputs(case, seed):
    """Weights (Glorot uniform), encoded inputs (hash-grid features, spherical
    harmonics of a direction, normal, roughness, albedo, the constant) and
    radiance targets (long-tailed, as path tracing gives them)."""
    rng = np.random.default_rng(seed)
    weights = []
    for rows, columns in _LAYERS:
        limit = math.sqrt(6.0 / (rows + columns))
        weights.append(rng.uniform(-limit, limit, (rows, columns)))
    n = case["records"]
    x = np.zeros((n, 64))
    x[:, 0:32] = rng.normal(0.0, 0.3, (n, 32))
    x[:, 32:48] = rng.uniform(-1.0, 1.0, (n, 16))
    normal = rng.normal(0.0, 1.0, (n, 3))
    x[:, 48:51] = normal / np.linalg.norm(normal, axis=1, keepdims=True)
    x[:, 51:55] = rng.uniform(0.0, 1.0, (n, 4))
    x[:, 55] = 1.0
    targets = np.exp(rng.normal(-1.0, 1.0, (n, 3)))
    flat = np.concatenate([w.ravel() for w in weights])
    return flat.astype(np.float32), x.astype(np.float32), targets.astype(np.float32)


def _prepare_gradient(p, case, seed):
    p.renderer = renderer.CudaOffscreenRenderer(0)
    p.scene = scenes.box_room(seed=seed, size=64)
    renderer.check(p.renderer.update_scene(p.scene), "update_scene")
    p.renderer.configure_cache(enable=False, seed=1)
    weights, p.inputs, p.targets = _gradient_inputs(case, seed)
    p.renderer.cache_weights(weights)


def _run_gradient(p):
    weight_gradients, input_gradients, loss = p.renderer.cache_gradient(p.inputs, p.targets)
    return {"weights": weight_gradients, "inputs": input_gradients, "loss": loss}


def _prepare_load(p, case, seed):
    p.renderer = renderer.CudaOffscreenRenderer(0)
    p.scene = _scene(case, seed)
    settings = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS,
                                    max_bounces=4, sample_index=_first_sample(seed))
    p.frame = p.scene.frame(settings, frame_count=1)
    p.image = _host_image(case["width"], case["height"])


def _run_load(p):
    renderer.check(p.renderer.update_scene(p.scene), "update_scene")
    return _run_frame(p)


def _prepare_edit(p, case, seed):
    p.renderer = renderer.CudaOffscreenRenderer(0)
    p.scene = scenes.grid_mesh(quads=case["quads"], size=case["size"])
    renderer.check(p.renderer.update_scene(p.scene), "update_scene")
    rng = np.random.default_rng(seed)
    points = p.scene.geometries[0][0]
    p.poses = []
    for k in range(2):
        bent = points.copy()
        bent[:, 1] += (0.05 * rng.uniform(0.5, 1.0) * np.sin(rng.uniform(1.0, 8.0) * points[:, 0] + k)
                       * np.cos(rng.uniform(1.0, 8.0) * points[:, 2])).astype(np.float32)
        moved = p.scene.instances[0][0].copy()
        moved[12:15] = rng.uniform(-0.1, 0.1, 3)
        p.poses.append((bent, moved))
    settings = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS,
                                    max_bounces=4, sample_index=_first_sample(seed))
    p.frame = p.scene.frame(settings, frame_count=1)
    p.images = [_host_image(case["size"], case["size"]) for _ in range(2)]
    p.index = 0


def _run_edit(p):
    points, transform = p.poses[p.index % 2]
    p.index += 1
    p.scene.set_positions(0, points)
    renderer.check(p.renderer.update_geometry(p.scene, 0), "update_geometry")
    result, sculpted = p.renderer.render_scene(p.frame, p.images[0])
    renderer.check(result, "render_scene")
    p.scene.set_instance(0, transform)
    renderer.check(p.renderer.update_instances(p.scene), "update_instances")
    result, moved = p.renderer.render_scene(p.frame, p.images[1])
    renderer.check(result, "render_scene")
    return {"sculpted": sculpted, "moved": moved}


def _prepare_batch(p, case, seed):
    p.batch = renderer.CudaBatch(0)
    # The batch workload's sizes; the rooms in them are the seed's.
    rng = np.random.default_rng(4000)
    p.rooms = []
    for k in range(case["scenes"]):
        triangles = int(math.exp(rng.uniform(math.log(1e4), math.log(2e6))))
        size = int(rng.choice([256, 512, 768, 1024]))
        p.rooms.append(scenes.batch_room(seed=(seed % 100_000) * 1000 + k, triangles=triangles, size=size))
    for result in p.batch.set_scenes(p.rooms):
        renderer.check(result, "set_scenes")
    p.frames = []
    for k, room in enumerate(p.rooms):
        settings = abi.default_settings(integrator=abi.INTEGRATOR_WAVEFRONT, light_sampling=abi.LIGHT_SAMPLING_MIS,
                                        max_bounces=case["bounces"], sample_index=1000 * k + _first_sample(seed))
        p.frames.append(room.frame(settings, frame_count=case["spp"]))


def _run_batch(p):
    results, images, total = p.batch.render(p.frames)
    renderer.check(total, "batch render")
    return images


_PATHS = {"frame": (_prepare_frame, _run_frame), "temporal": (_prepare_temporal, _run_temporal),
          "cached": (_prepare_cached, _run_cached), "gradient": (_prepare_gradient, _run_gradient),
          "load": (_prepare_load, _run_load), "edit": (_prepare_edit, _run_edit),
          "batch": (_prepare_batch, _run_batch)}


def prepare(case, seed):
    p = _Program()
    p.case = dict(case)
    _PATHS[case["path"]][0](p, case, seed)
    return p


def run(state):
    return _PATHS[state.case["path"]][1](state)


# Unique triangles, instances and rays per camera path of the scenes (about:
# a path's length depends on the scene, not on the code that follows it).
_SIZES = {"cornell": (36, 8, 6.0), "cornell-gltf": (36, 8, 6.0), "room": (36, 8, 6.5), "lights": (34, 7, 7.0),
          "textures": (52, 26, 3.0)}


def _tracing(rays, triangles, instances):
    """Arithmetic of `rays` rays: a box pair per level of a balanced tree over
    the instances and over one mesh, one triangle test, one shading."""
    levels = math.log2(max(2, triangles / max(1, instances) + 1)) + math.log2(max(2, instances))
    return rays * (levels * 24.0 + 60.0 + 200.0)


def work(case):
    path = case["path"]
    if path == "gradient":
        n = case["records"]
        weights = sum(rows * columns for rows, columns in _LAYERS)
        # Inputs, targets and input gradients cross once, with the weights'
        # gradients; forward, input gradients, weight gradients.
        return {"bytes": 4.0 * (n * (64 + 64 + 3) + 2 * weights), "flops": 6.0 * n * weights}
    if path == "batch":
        pixels = case["scenes"] * 444_000.0  # the mean of the four target sizes
        rays = pixels * case["spp"] * 6.0
        return {"bytes": pixels * 16.0 + case["scenes"] * 20_516 * 160.0, "flops": _tracing(rays, 20_516, 70)}
    if path == "edit":
        triangles, pixels = 2.0 * case["quads"] ** 2, 2.0 * case["size"] ** 2
        # New points in, triangle records and 4-wide nodes rewritten.
        return {"bytes": triangles * (6 + 64 + 64) + pixels * 16.0, "flops": _tracing(pixels * 6.0, triangles, 2)}
    pixels = float(case["width"] * case["height"])
    if path in ("temporal", "cached"):
        triangles = 36 + case["emitters"]
        # The image, and the histories that a temporal frame reads and writes.
        state = (2 * (64 + 32 + 64 + 160) if path == "temporal" else 2 * 32) + 16.0
        return {"bytes": pixels * state + triangles * 160.0,
                "flops": _tracing(pixels * 2.0 * case["bounces"], triangles, triangles)}
    if case["scene"] == "field":
        triangles, instances, rays = 3_344.0 * case["detail"], 4161, 3.0
    elif case["scene"] == "mesh":
        triangles, instances, rays = 20.0 * 4 ** case["detail"], 3, 4.0
    else:
        triangles, instances, rays = _SIZES[case["scene"]]
    samples = pixels * case.get("spp", 1)
    # Corners, indices and normals in once; triangle records and nodes out.
    built = triangles * (24.0 + 36.0 + 64.0 + 64.0) if path == "load" else 0.0
    return {"bytes": pixels * (16.0 + 64.0) + triangles * 100.0 + built,
            "flops": _tracing(samples * rays, triangles, instances)}


def exact(case, seed):
    """The gradient case in 64 bits, but for the inputs' gradients: a
    pre-activation near zero falls on the other side of its ReLU in 16-bit
    operands, and those gradients then go through other weights. The other
    cases follow paths whose branches are decisions on 32-bit random numbers
    and hits: a 64-bit evaluation follows other paths, so they have no such
    value."""
    if case["path"] != "gradient":
        return None
    flat, x, targets = (a.astype(np.float64) for a in _gradient_inputs(case, seed))
    weights, at = [], 0
    for rows, columns in _LAYERS:
        weights.append(flat[at:at + rows * columns].reshape(rows, columns))
        at += rows * columns
    activations = [x]
    for w in weights[:-1]:
        activations.append(np.maximum(activations[-1] @ w, 0.0))
    y = (activations[-1] @ weights[-1])[:, :3]
    # The relative squared error, its denominator held constant.
    scale = y * y + 0.01
    loss = float(np.sum((y - targets) ** 2 / scale))
    gradient = np.zeros((x.shape[0], 16))
    gradient[:, :3] = 2.0 * (y - targets) / scale
    weight_gradients = []
    for k in range(len(weights) - 1, -1, -1):
        weight_gradients.append((activations[k].T @ gradient).ravel())
        if k > 0:
            gradient = (gradient @ weights[k].T) * (activations[k] > 0.0)
    return {"weights": np.concatenate(weight_gradients[::-1]), "inputs": None, "loss": loss}
