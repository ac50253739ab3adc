"""The device's certified short forms at extreme scales: closest hits of very small and very large meshes seen
from near and far (the single-precision filter and the barycentrics around the hit), and paths whose
emission is near either end of the float range (the exponent-split products)."""
import numpy as np
import pytest

from bf200 import abi, runtime, scenes
from helpers import arrays, bit_equal
from oracle.bindings import Oracle

pytestmark = pytest.mark.gpu


def sphere_scene(size):
    builder = scenes.SceneBuilder(environment=(0.5, 0.5, 0.5, 0.5))
    mesh = scenes.displaced_icosphere(3, 0.05, 7)
    light = scenes.grid_quad((0.0, 0.0), 2.0, 2, 3.0)
    for m in (mesh, light):
        m.positions = (m.positions * np.float32(size)).astype(np.float32)
    builder.add_instance(builder.add_mesh(mesh), builder.add_material(scenes.lambertian([0.5] * 4)))
    builder.add_instance(builder.add_mesh(light), builder.add_material(scenes.lambertian([0.0] * 4), emission=(1.0,) * 4))
    return builder, mesh


def rays_at(mesh, n, distance, seed):
    """Rays at points inside triangles, a third each at general points, near edges and near corners."""
    rng = np.random.default_rng(seed)
    triangles = mesh.positions[mesh.triangles[rng.integers(0, len(mesh.triangles), n)]].astype(np.float64)
    weights = rng.dirichlet((1.0, 1.0, 1.0), n)
    small = 10.0 ** rng.uniform(-8.0, -2.0, n)
    weights[::3, 0] = small[::3]
    weights[1::3, :2] = small[1::3, None]
    weights = rng.permuted(weights / weights.sum(axis=1, keepdims=True), axis=1)
    target = (weights[:, :, None] * triangles).sum(axis=1)
    direction = rng.normal(size=(n, 3))
    direction = (direction / np.linalg.norm(direction, axis=1, keepdims=True)).astype(np.float32)
    table = np.zeros(n, dtype=[("o", "<f4", 3), ("d", "<f4", 3), ("t", "<f4", 2), ("time", "<f4"), ("mask", "<u4"),
                               ("rest", "<u4", 2)])
    table["o"], table["d"], table["t"] = target - distance * direction, direction, [0.0, np.inf]
    table["time"], table["mask"] = scenes.PATH_TIME, 0xFFFFFFFF
    return (abi.Ray * n).from_buffer_copy(table.tobytes())


@pytest.mark.parametrize("distance", [0.0, 1.0, 100.0, 1e4])  # in units of the mesh's size
@pytest.mark.parametrize("size", [1e-15, 1e-12, 1e-6, 1e6, 1e12, 1e18])
def test_closest_hits_at_any_scale(size, distance):
    builder, mesh = sphere_scene(size)
    rays = rays_at(mesh, 1200, distance * size, int(distance) + 1)
    oracle = Oracle(device_trig=True)
    handle = oracle.scene(builder)
    expected = oracle.closest_hits(handle, rays)
    oracle.destroy(handle)
    with runtime.Context(0, path_capacity=1 << 12) as ctx:
        scene = ctx.create_scene(builder)
        got = ctx.closest_hits(scene, rays)
        scene.close()
    want = np.frombuffer(expected, np.uint32).reshape(-1, 8)
    assert (want[:, 4] != 0xFFFFFFFF).mean() > 0.5
    assert np.array_equal(np.frombuffer(got, np.uint32).reshape(-1, 8), want)


@pytest.mark.parametrize("emission", [1e-44, 1e-40, 2e-38, 1e-37, 1e-30, 1e30, 1e37])
def test_paths_of_extreme_emission_match_the_oracle_bit_for_bit(emission):
    """Light that is subnormal, crosses the smallest normal number along a path, or nears the largest. The
    device evaluates a light's contribution before its shadow ray, the oracle after it: so where a
    contribution underflows, the device also fails paths whose shadow ray is blocked, and never fewer."""
    builder = scenes.SceneBuilder()
    scenes.cornell_box(builder, with_spheres=True)
    for k, material in enumerate(builder.materials):
        if any(material[1]):
            builder.materials[k] = (material[0], tuple(emission * s for s in (1.0, 0.7, 0.4, 0.2)), *material[2:])
    options = abi.default_options(mis="power", max_depth=6)
    side = 48
    camera = runtime.camera_create(*scenes.camera_frame_inputs(), side, side, scenes.CAMERA_VFOV, scenes.PATH_TIME)
    samples = (abi.SampleIndex * (side * side))()
    for i in range(side * side):
        samples[i].pixel_x, samples[i].pixel_y, samples[i].sample_index = i % side, i // side, 2
    oracle = Oracle(device_trig=True)
    rays = oracle.camera_rays(camera, samples)
    inputs = (abi.PathInput * len(samples))()
    for i, ray in enumerate(rays):
        inputs[i].primary_ray, inputs[i].sample = ray, samples[i]
    handle = oracle.scene(builder)
    expected, _ = oracle.trace(handle, inputs, options)
    oracle.destroy(handle)
    with runtime.Context(0, path_capacity=1 << 12) as ctx:
        scene = ctx.create_scene(builder)
        results, _ = ctx.trace_paths(scene, inputs, options)
        scene.close()
    got, want = arrays(results), arrays(expected)
    failed, wanted = got["lane_status"] != 0, want["lane_status"] != 0
    assert failed[wanted].all()
    if emission >= 1e-30:
        assert not failed.any()
    keep = ~failed
    assert keep.any()
    assert bit_equal(got["radiance"][keep], want["radiance"][keep]).all()
    assert np.array_equal(got["termination"][keep], want["termination"][keep])
