"""The renderer's work as its users call it: film renders, explicit path batches, ray queries, a batch
of scenes and the path-replay adjoint, each through the public Python binding of the C ABI.

Every call is synchronous: when it returns, its results are complete. The scenes are the
repository's own workloads (bf200.scenes); what varies with the seed is the camera position, the
sampling seed, the rays and the adjoint's target image.
"""
import ctypes as C
import functools
import math
import os
import sys
import weakref

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "blackframe-renderer_b200"))

from bf200 import abi, runtime, scenes  # noqa: E402

# CIE 1931 sensor constants of the workloads' wavelength packet (407, 524.5, 642 and 759.5 nm).
RESPONSE = ((0.029782479628920555, 0.0008254999993368983, 0.14170169830322266),
            (0.10452822595834732, 0.7855184078216553, 0.05901917815208435),
            (0.4120979905128479, 0.1596464067697525, 1.6199999663513154e-05),
            (0.00017210794612765312, 6.215133180376142e-05, 0.0))
WAVELENGTH_PDF = 0.0021276595070958138
NORMALIZATION = 0.002339577069506049

# Scenes: (unique triangles, extension segments per path, shadow segments per path), the last two as the
# renderer reports them for its own depth (16; 8 for the plain box and the adjoint).
SCENES = {
    "cornell": (24, 3.19, 2.02),
    "cornell_spheres": (3992, 3.39, 2.11),
    "cornell_analytic": (26, 3.39, 2.12),
    "cornell_layered": (3992, 3.07, 1.22),
    "stress_small": (63_490, 2.03, 0.82),  # 3 x 20,480 triangles, 40 instances
    "stress": (985_090, 2.03, 0.82),       # 3 x 327,680 triangles, 40 instances
    "adjoint": (85_900, 6.24, 3.87),       # no roulette
}
BATCH_JOBS = 64  # scenes.batch_job(0..63)


def film(name, scene, width, height, spp, depth=16, mis="power", sampler=0, precision=0, host=False):
    return {"name": name, "kind": "film", "scene": scene, "width": width, "height": height, "spp": spp, "depth": depth,
            "mis": mis, "sampler": sampler, "precision": precision, "host": host}


def listed():
    return [
        # an interactive preview pass: one sample per pixel of a small box, where latency is all
        film("preview_64", "cornell", 64, 64, 1, depth=8, mis="balance"),
        # the plain 64 x 64 x 16 box with the Owen-Sobol sampler into host memory, as a caller of the
        # reference's film loop has it
        film("cornell_64_owen_host", "cornell", 64, 64, 16, depth=8, mis="balance", sampler=1, host=True),
        # a full frame of the box with GGX spheres
        film("cornell_spheres_256", "cornell_spheres", 256, 256, 256),
        # an odd-sized frame of mixtures, specular closures and punctual lights, compensated-double film
        film("layered_odd_double", "cornell_layered", 333, 217, 23, precision=1),
        # analytic spheres, Owen-Sobol, the film in host memory
        film("analytic_host", "cornell_analytic", 256, 256, 32, sampler=1, host=True),
        # the headline scene and frame size: 985,090 triangles in 42 instances
        film("stress_1080p", "stress", 1920, 1080, 16),
        # a small batch of explicit paths with ray cones from host memory, as the drop-in adapter
        # passes a tile
        {"name": "tile_cones_host", "kind": "paths", "scene": "cornell_spheres", "paths": 4097, "depth": 16,
         "mis": "power", "cones": True, "host": True},
        # one sample per pixel of the headline frame as explicit device paths
        {"name": "paths_stress_device", "kind": "paths", "scene": "stress", "paths": 2_073_600, "depth": 16,
         "mis": "power", "cones": False, "host": False},
        # closest hits of a picking or baking pass
        {"name": "hits_cornell", "kind": "hits", "scene": "cornell_spheres", "rays": 20_001},
        # visibility of many point pairs in the large scene
        {"name": "occlusion_stress", "kind": "occlusions", "scene": "stress", "rays": 500_000},
        # image loss and gradients: forward and replay
        {"name": "adjoint_256", "kind": "adjoint", "side": 256, "spp": 16},
        # sixteen scenes of uneven size in one call
        {"name": "batch_16", "kind": "batch", "first": 0, "jobs": 16},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["film", "film", "film", "paths", "paths", "hits", "occlusions", "adjoint", "batch"])
    small = ["cornell", "cornell_spheres", "cornell_analytic", "cornell_layered", "stress_small"]
    if kind == "film":
        scene = rng.choice(small + ["stress"])
        width, height = _log_uniform(rng, 17, 1920), _log_uniform(rng, 17, 1080)
        most = 16_000_000 if scene.startswith("stress") else 8_000_000  # paths
        spp = _log_uniform(rng, 1, max(1, min(256, most // (width * height))))
        case = film(None, scene, width, height, spp, depth=rng.randint(2, 16), mis=rng.choice(["power", "balance"]),
                    sampler=rng.randint(0, 1), precision=rng.randint(0, 1), host=rng.random() < 0.3)
        del case["name"]
        return case
    if kind == "paths":
        return {"kind": kind, "scene": rng.choice(small + ["stress"]), "paths": _log_uniform(rng, 16, 2_073_600),
                "depth": rng.randint(2, 16), "mis": rng.choice(["power", "balance"]), "cones": rng.random() < 0.5,
                "host": rng.random() < 0.5}
    if kind in ("hits", "occlusions"):
        return {"kind": kind, "scene": rng.choice(["cornell", "cornell_spheres", "stress_small", "stress"]),
                "rays": _log_uniform(rng, 16, 1_000_000)}
    if kind == "adjoint":
        side = _log_uniform(rng, 16, 256)
        return {"kind": kind, "side": side, "spp": _log_uniform(rng, 1, max(1, min(64, 1_048_576 // (side * side))))}
    return {"kind": kind, "first": rng.randrange(4, BATCH_JOBS - 12), "jobs": rng.randint(2, 12)}


# ------------------------------------------------------------------------------------------------
# Preparation: contexts, scenes, cameras and inputs
# ------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _builder(scene):
    """The scene's description arrays: a user's own data, made once."""
    if scene == "stress":
        return scenes.bvh_stress(scenes.SceneBuilder(environment=(0.5, 0.5, 0.5, 0.5)))
    if scene == "stress_small":
        return scenes.bvh_stress(scenes.SceneBuilder(environment=(0.5, 0.5, 0.5, 0.5)), subdivisions=5)
    if scene == "cornell_layered":
        return scenes.cornell_layered(scenes.SceneBuilder())
    if scene == "adjoint":
        return scenes.adjoint_icosphere(scenes.SceneBuilder(), scenes.adjoint_parameters())
    if scene == "adjoint_target":
        return scenes.adjoint_icosphere(scenes.SceneBuilder(),
                                        scenes.perturbed_parameters(scenes.adjoint_parameters()))
    return scenes.cornell_box(scenes.SceneBuilder(), with_spheres=scene != "cornell",
                              analytic_spheres=scene == "cornell_analytic")


@functools.lru_cache(maxsize=BATCH_JOBS)
def _batch_job(index):
    return scenes.batch_job(index)


class Program:
    """What a rendering program keeps: a context, its scenes and its buffers."""

    def __init__(self):
        self.context = runtime.Context(0)
        self.scenes = []
        weakref.finalize(self, Program._release, self.context, self.scenes)

    def scene(self, builder):
        self.scenes.append(self.context.create_scene(builder))
        return self.scenes[-1]

    @staticmethod
    def _release(context, held):
        for scene in held:
            scene.close()
        context.close()


def _sensor():
    sensor = abi.Sensor()
    for lane in range(4):
        for k in range(3):
            sensor.response_xyz[lane][k] = RESPONSE[lane][k]
        sensor.wavelength_pdf[lane] = WAVELENGTH_PDF
    sensor.normalization = NORMALIZATION
    return sensor


def _camera(scene, width, height, rng):
    """The workload's camera, moved a little by the seed."""
    if scene.startswith("stress"):
        (origin, target), vfov, reach = scenes.BVH_STRESS_CAMERA, scenes.BVH_STRESS_VFOV, 0.5
    else:
        (origin, target), vfov, reach = (scenes.CAMERA_ORIGIN, scenes.CAMERA_TARGET), scenes.CAMERA_VFOV, 0.05
    origin = tuple(np.asarray(origin) + rng.uniform(-reach, reach, 3))
    return runtime.camera_create(*scenes.camera_frame_inputs(origin, target), width, height, vfov, scenes.PATH_TIME)


def _film_buffers(width, height, precision):
    shape, kind = ((height, width, 8), torch.float64) if precision else ((height, width, 4), torch.float32)
    return (torch.zeros(shape, dtype=kind, device="cuda"),
            torch.zeros((height, width), dtype=torch.int64, device="cuda"))


def _options(case):
    options = abi.default_options(mis=case["mis"], max_depth=case["depth"])
    options.sampler = case.get("sampler", 0)
    return options


def _path_inputs(program, case, rng):
    """Camera paths: consecutive pixels of a 1080p frame (square tiles of small counts), one sample."""
    n = case["paths"]
    width = 1920 if n > 65_536 else max(1, math.isqrt(n))
    height = -(-n // width)
    camera = _camera(case["scene"], width, height, rng)
    y, x = np.divmod(np.arange(n, dtype=np.uint64), np.uint64(width))
    table = np.zeros(n, dtype=[("x", "<u4"), ("y", "<u4"), ("s", "<u8"), ("seed", "<u8")])
    table["x"], table["y"] = x, y
    table["s"], table["seed"] = int(rng.integers(0, 1 << 20)), int(rng.integers(0, 1 << 62))
    samples = (abi.SampleIndex * n).from_buffer_copy(table.tobytes())
    rays, status = program.context.camera_rays(camera, samples)
    if status.any():
        raise RuntimeError("a camera ray was refused")
    paths = np.zeros(n, dtype=[("ray", "V48"), ("sample", "V24"), ("reserved", "<u8")])
    paths["ray"] = np.frombuffer(rays, dtype="V48")
    paths["sample"] = np.frombuffer(samples, dtype="V24")
    # a pinhole camera's primary cones: no width at the origin, half a pixel's slope
    slope = camera.half_height / height
    cones = np.stack([np.zeros(n), np.full(n, slope) * rng.uniform(0.9, 1.0, n)], axis=1).astype(np.float32)
    return paths, cones


def _rays(case, rng):
    """Origins across the scene's free space (above the box's cuboids), isotropic directions;
    shadow-like segments for occlusion."""
    n = case["rays"]
    if case["scene"].startswith("stress"):
        low, high = np.array([-11.0, -11.0, -11.0]), np.array([11.0, 13.0, 11.0])
    else:
        low, high = np.array([-0.95, 0.25, 0.05]), np.array([0.95, 0.95, 1.95])
    direction = rng.normal(size=(n, 3))
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    table = np.zeros(n, dtype=[("o", "<f4", 3), ("d", "<f4", 3), ("t_min", "<f4"), ("t_max", "<f4"), ("time", "<f4"),
                               ("mask", "<u4"), ("medium", "<u4"), ("reserved", "<u4")])
    table["o"] = rng.uniform(low, high, (n, 3))
    table["d"] = direction
    extent = float(np.max(high - low))
    table["t_max"] = rng.uniform(0.05, 1.0, n) * extent if case["kind"] == "occlusions" else np.inf
    table["time"], table["mask"] = scenes.PATH_TIME, 0xFFFFFFFF
    return table


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    program = Program()
    kind = case["kind"]
    if kind == "film":
        scene = program.scene(_builder(case["scene"]))
        camera = _camera(case["scene"], case["width"], case["height"], rng)
        state = {"args": (scene, camera, _sensor(), _options(case), case["spp"], int(rng.integers(0, 1 << 62)), 0,
                          case["precision"])}
        if not case["host"]:
            state["film"] = _film_buffers(case["width"], case["height"], case["precision"])
    elif kind == "paths":
        scene = program.scene(_builder(case["scene"]))
        inputs, cones = _path_inputs(program, case, rng)
        n = case["paths"]
        state = {"scene": scene, "options": _options(case), "cones": cones}
        if case["host"]:
            state["inputs"] = (abi.PathInput * n).from_buffer_copy(inputs.tobytes())
        else:
            state["inputs"] = torch.from_numpy(inputs.view(np.uint8).reshape(n, 80).copy()).cuda()
            state["device_cones"] = torch.from_numpy(cones).cuda()
            state["results"] = torch.zeros((n, 32), dtype=torch.int32, device="cuda")
            state["terminal"] = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
    elif kind in ("hits", "occlusions"):
        state = {"scene": program.scene(_builder(case["scene"])),
                 "rays": (abi.Ray * case["rays"]).from_buffer_copy(_rays(case, rng).tobytes())}
    elif kind == "adjoint":
        side, spp, sensor = case["side"], case["spp"], _sensor()
        scene = program.scene(_builder("adjoint"))
        camera = _camera("adjoint", side, side, rng)
        # Russian roulette off: the gradients are then the exact derivatives of the rendered loss
        options = abi.default_options(mis="power", max_depth=8, roulette=False)
        sums, counts = _film_buffers(side, side, 1)
        wanted = program.scene(_builder("adjoint_target"))
        program.context.render_film_device(wanted, camera, sensor, options, 4, int(rng.integers(0, 1 << 62)), 0, 1,
                                           sums.data_ptr(), counts.data_ptr())
        target = ((sums[..., :3] + sums[..., 4:7]) / (sums[..., 3:4] + sums[..., 7:8])).float().contiguous()
        gradients = torch.zeros((len(scene.builder.materials), 8), dtype=torch.float64, device="cuda")
        emission = torch.zeros(1, dtype=torch.float64, device="cuda")
        state = {"args": (scene, camera, sensor, options, spp, int(rng.integers(0, 1 << 62)), 0, 1, sums.data_ptr(),
                          counts.data_ptr(), target.data_ptr(), gradients.data_ptr(), emission.data_ptr()),
                 "film": (sums, counts), "target": target, "gradients": gradients, "emission": emission}
    else:
        jobs, films = [], []
        for index in range(case["first"], case["first"] + case["jobs"]):
            builder, options, (width, height, spp) = _batch_job(index)
            sums, counts = _film_buffers(width, height, 0)
            jobs.append((program.scene(builder), _camera("batch", width, height, rng), _sensor(), options, spp,
                         int(rng.integers(0, 1 << 62)), 0, 0, sums.data_ptr(), counts.data_ptr()))
            films.append((sums, counts))
        state = {"jobs": jobs, "films": films}
    state["case"], state["program"] = case, program
    torch.cuda.synchronize()
    return state


# ------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------

def _clear(films):
    """Starts new frames; the renderer adds to a film on a stream of its own, so the clears finish first."""
    for sums, counts in films:
        sums.zero_()
        counts.zero_()
    torch.cuda.current_stream().synchronize()


def _path_outputs(words):
    """A path result's fields (n x 32 words): throughput, radiance and eta scale; depth, counters,
    flags, termination, lane status and segments; the terminal ray."""
    real = words.view(np.float32) if isinstance(words, np.ndarray) else words.view(torch.float32)
    return {"beta": real[:, 0:4], "radiance": real[:, 4:8], "depth": words[:, 8:14], "eta_scale": real[:, 14],
            "outcome": words[:, 15:20], "terminal_ray": real[:, 20:29], "terminal_mask": words[:, 29:31]}


def run(state):
    case, context = state["case"], state["program"].context
    kind = case["kind"]
    if kind == "film":
        if case["host"]:
            sums, counts, _ = context.render_film(*state["args"][:4], case["spp"], seed=state["args"][5],
                                                  precision=case["precision"])
            return {"sums": sums, "counts": counts.view(np.int64)}
        sums, counts = state["film"]
        _clear([state["film"]])
        context.render_film_device(*state["args"], sums.data_ptr(), counts.data_ptr())
        return {"sums": sums, "counts": counts}
    if kind == "paths":
        scene, options = state["scene"], state["options"]
        if case["host"]:
            if case["cones"]:
                results, terminal, _ = context.trace_paths_with_cones(scene, state["inputs"], state["cones"], options)
            else:
                results, _ = context.trace_paths(scene, state["inputs"], options)
            out = _path_outputs(np.frombuffer(results, dtype=np.int32).reshape(-1, 32))
        else:
            inputs, results, terminal = state["inputs"], state["results"], state["terminal"]
            if case["cones"]:
                context.trace_paths_with_cones_device(scene, inputs.data_ptr(), state["device_cones"].data_ptr(),
                                                      case["paths"], options, results.data_ptr(), terminal.data_ptr())
            else:
                context.trace_paths_device(scene, inputs.data_ptr(), case["paths"], options, results.data_ptr())
            out = _path_outputs(results)
        if case["cones"]:
            out["terminal_cone"] = terminal
        return out
    if kind == "hits":
        hits = np.frombuffer(context.closest_hits(state["scene"], state["rays"]), dtype=np.float32).reshape(-1, 8)
        return {"t": hits[:, 0], "barycentrics": hits[:, 1:4], "ids": hits.view(np.int32)[:, 4:7]}
    if kind == "occlusions":
        return {"occluded": context.occlusions(state["scene"], state["rays"]).view(np.int32)}
    if kind == "adjoint":
        loss, _ = context.render_adjoint_device(*state["args"])
        sums, counts = state["film"]
        return {"loss": float(loss), "gradients": state["gradients"], "emission": state["emission"], "sums": sums,
                "counts": counts}
    _clear(state["films"])
    context.render_films_device(state["jobs"])
    return {"sums": [sums for sums, _ in state["films"]], "counts": [counts for _, counts in state["films"]]}


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without, and what its results are held to
# ------------------------------------------------------------------------------------------------

# Operations of one ray through a good four-wide hierarchy: about two node visits (4 boxes of 18
# operations) per factor of four in triangles, and two triangle tests of 80 operations; of one shaded
# vertex: closure sampling and evaluation, one light sample and its weights over four lanes.
BOX_FLOPS, TRIANGLE_FLOPS, VERTEX_FLOPS = 72, 80, 500


def _ray_flops(triangles):
    return 2 * BOX_FLOPS * max(1.0, math.log(max(4, triangles), 4)) + 2 * TRIANGLE_FLOPS


def _path_flops(scene, paths, depth):
    triangles, extension, shadow = SCENES[scene]
    extension, shadow = min(extension, depth + 1), min(shadow, depth)
    return paths * ((extension + shadow) * _ray_flops(triangles) + extension * VERTEX_FLOPS)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for index in range(case["first"], case["first"] + case["jobs"]):
            builder, options, (width, height, spp) = _batch_job(index)
            total["bytes"] += 36.0 * builder.triangle_count + 24.0 * width * height
            total["flops"] += width * height * spp * 4.0 * (_ray_flops(builder.triangle_count) + VERTEX_FLOPS)
        return total
    scene = case.get("scene", "adjoint")
    geometry = 36.0 * SCENES[scene][0]  # three vertices per triangle, read once
    if kind == "film":
        pixels = case["width"] * case["height"]
        return {"bytes": geometry + pixels * (72.0 if case["precision"] else 24.0),
                "flops": _path_flops(scene, pixels * case["spp"], case["depth"])}
    if kind == "paths":
        return {"bytes": geometry + case["paths"] * (80.0 + 128.0 + (16.0 if case["cones"] else 0.0)),
                "flops": _path_flops(scene, case["paths"], case["depth"])}
    if kind == "adjoint":
        pixels = case["side"] ** 2
        return {"bytes": geometry + pixels * (72.0 + 12.0),
                "flops": 2.0 * _path_flops(scene, pixels * case["spp"], 8)}
    return {"bytes": geometry + case["rays"] * (48.0 + (32.0 if kind == "hits" else 4.0)),
            "flops": case["rays"] * _ray_flops(SCENES[scene][0])}


def tolerance(case):
    """The renderer promises the reference's scalar result path for path, samples summed in sample
    order: hits, paths and films are reproduced to the bit. Only the adjoint's gradients and loss are
    sums in no fixed order, in 64 bits."""
    return {"rel": 1e-11} if case["kind"] == "adjoint" else "exact"


def exact(case, seed):
    """Closest hits and visibility against every triangle, in 64 bits, for scenes small enough.

    A Monte Carlo path has no 64-bit counterpart: each hit, lobe and roulette decision branches on
    the rounded value before it, so films, paths and gradients give None. So do the large scenes,
    where testing every instanced triangle takes minutes."""
    if case["kind"] not in ("hits", "occlusions") or not case["scene"].startswith("cornell"):
        return None
    builder = _builder(case["scene"])
    table = _rays(case, np.random.default_rng(seed))
    corners, instance, primitive = [], [], []
    for k, (mesh, _, matrix, _) in enumerate(builder.instances):
        mesh = builder.meshes[mesh]
        m = np.asarray(matrix, np.float64).reshape(4, 4)
        world = np.asarray(mesh.positions, np.float64) @ m[:3, :3].T + m[:3, 3]
        corners.append(world[np.asarray(mesh.triangles, np.int64)])
        instance.append(np.full(len(mesh.triangles), k))
        primitive.append(np.arange(len(mesh.triangles)))
    v = torch.from_numpy(np.concatenate(corners)).cuda()
    instance = torch.from_numpy(np.concatenate(instance)).cuda()
    primitive = torch.from_numpy(np.concatenate(primitive)).cuda()
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = len(table)
    origin = torch.from_numpy(table["o"].astype(np.float64)).cuda()
    direction = torch.from_numpy(table["d"].astype(np.float64)).cuda()
    limit = torch.from_numpy(table["t_max"].astype(np.float64)).cuda()
    t_out = torch.zeros(n, dtype=torch.float64, device="cuda")
    bary = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    ids = torch.full((n, 3), -1, dtype=torch.int32, device="cuda")
    ids[:, 2] = 0
    chunk = max(1, 40_000_000 // len(v))
    for a in range(0, n, chunk):
        o, d = origin[a:a + chunk, None, :], direction[a:a + chunk, None, :]
        p = torch.linalg.cross(d, e2[None])
        det = (e1 * p).sum(-1)
        s = o - v0
        b1 = (s * p).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        b2 = (d * q).sum(-1) / det
        t = (e2 * q).sum(-1) / det
        hit = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= 0) & (t <= limit[a:a + chunk, None])
        t = torch.where(hit, t, torch.inf)
        best, which = t.min(dim=1)
        found = torch.isfinite(best)
        rows = torch.arange(len(best), device="cuda")
        t_out[a:a + chunk] = torch.where(found, best, 0.0)
        w1, w2 = b1[rows, which], b2[rows, which]
        weights = torch.stack([1.0 - w1 - w2, w1, w2], dim=1)
        bary[a:a + chunk] = torch.where(found[:, None], weights, 0.0)
        named = torch.stack([instance[which], primitive[which]], dim=1).int()
        ids[a:a + chunk, :2] = torch.where(found[:, None], named, -1)
    if case["kind"] == "occlusions":
        return {"occluded": (ids[:, 0] >= 0).int().cpu().numpy()}
    return {"t": t_out, "barycentrics": bary, "ids": ids}
