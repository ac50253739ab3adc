"""The traversal's warp ray pools at the edges of their sizes: ray counts around the lanes, warps and
blocks, and walks whose stacks outgrow the entries kept in shared memory."""
import numpy as np
import pytest

from bf200 import abi, runtime, scenes
from oracle.bindings import Oracle

pytestmark = pytest.mark.gpu


def ray_array(n, seed):
    """n rays from above the Cornell box's cuboids, every seventh along an axis."""
    rng = np.random.default_rng(seed)
    table = np.zeros(n, dtype=[("o", "<f4", 3), ("d", "<f4", 3), ("t", "<f4", 2), ("time", "<f4"), ("mask", "<u4"),
                               ("rest", "<u4", 2)])
    table["o"] = rng.uniform([-0.95, 0.3, 0.05], [0.95, 0.95, 1.95], (n, 3))
    d = rng.normal(size=(n, 3))
    d[::7] = np.eye(3)[rng.integers(0, 3, len(d[::7]))] * rng.choice([-1.0, 1.0], (len(d[::7]), 1))
    table["d"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    table["t"] = [0.0, np.inf]
    table["time"], table["mask"] = scenes.PATH_TIME, 0xFFFFFFFF
    return (abi.Ray * n).from_buffer_copy(table.tobytes())


def check_queries(builder, rays):
    oracle = Oracle(device_trig=True)
    handle = oracle.scene(builder)
    expected = oracle.closest_hits(handle, rays)
    oracle.destroy(handle)
    with runtime.Context(0, path_capacity=1 << 12) as ctx:
        scene = ctx.create_scene(builder)
        got = ctx.closest_hits(scene, rays)
        occluded = ctx.occlusions(scene, rays)
        scene.close()
    assert bytes(got) == bytes(expected)
    hit = np.array([h.instance_index != 0xFFFFFFFF for h in expected], np.uint32)
    assert np.array_equal(occluded, hit)
    return hit


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 257, 4099])
def test_ray_counts(n):
    builder = scenes.SceneBuilder()
    scenes.cornell_box(builder, with_spheres=True)
    check_queries(builder, ray_array(n, n))


@pytest.mark.parametrize("instances", [15, 31, 32, 60])  # and the light: at most 32 are eager
def test_overlapping_instances_fill_the_stack(instances):
    """Nested shells of one mesh: every ray from outside meets all of their boxes, so up to 32 eager
    instance entries (or a TLAS of them) lie under a BLAS walk, beyond the shared entries."""
    builder = scenes.SceneBuilder()
    mesh = builder.add_mesh(scenes.displaced_icosphere(3, 0.05, 1))
    material = builder.add_material(scenes.lambertian([0.5] * 4))
    for i in range(instances):
        builder.add_instance(mesh, material, scenes.uniform_scale_translate(0.2 + 0.01 * i, (0.0, 0.6, 1.0)))
    builder.add_instance(builder.add_mesh(scenes.grid_quad((0.0, 1.0), 0.5, 1, 1.9)),
                         builder.add_material(scenes.lambertian([0.0] * 4), emission=(1.0,) * 4))
    hit = check_queries(builder, ray_array(1024, instances))
    assert hit.any() and not hit.all()


@pytest.mark.parametrize("n", [1, 33, 257, 1030])
def test_path_counts(n):
    """A trace of any number of paths gives each path what a trace of all of them gives it."""
    builder = scenes.SceneBuilder()
    scenes.cornell_box(builder, with_spheres=True)
    options = abi.default_options(mis="power", max_depth=8)
    camera = runtime.camera_create(*scenes.camera_frame_inputs(), 64, 64, scenes.CAMERA_VFOV, scenes.PATH_TIME)
    samples = (abi.SampleIndex * 4096)()
    for i in range(4096):
        samples[i].pixel_x, samples[i].pixel_y, samples[i].sample_index = i % 64, i // 64, 3
    with runtime.Context(0, path_capacity=1 << 9) as ctx:  # fewer slots than paths: slots are refilled
        rays, status = ctx.camera_rays(camera, samples)
        assert not status.any()
        inputs = (abi.PathInput * 4096)()
        for i, ray in enumerate(rays):
            inputs[i].primary_ray, inputs[i].sample = ray, samples[i]
        scene = ctx.create_scene(builder)
        every, _ = ctx.trace_paths(scene, inputs, options)
        few, report = ctx.trace_paths(scene, (abi.PathInput * n)(*inputs[:n]), options)
        scene.close()
    assert report.path_count == n
    assert bytes(few) == bytes(every)[:128 * n]
