"""The wavefront's forms against one another: three-launch and one-block compaction with every shading route in
use, chained and unchained launches at the line between them, shading branches and the instrumented loop.
Which form a trace takes changes none of its results."""
import numpy as np
import pytest

from bf200 import abi, runtime, scenes
from helpers import arrays, check_paths
from oracle.bindings import Oracle
from test_gpu_routes import sequences

pytestmark = pytest.mark.gpu

CHAIN_SLOTS = 1 << 18  # kChainSlots


def camera_paths(ctx, n, width):
    """The first n pixels of a frame of this width, one sample each."""
    camera = runtime.camera_create(*scenes.camera_frame_inputs(), width, -(-n // width), scenes.CAMERA_VFOV,
                                   scenes.PATH_TIME)
    table = np.zeros(n, dtype=[("x", "<u4"), ("y", "<u4"), ("s", "<u8"), ("seed", "<u8")])
    table["y"], table["x"] = np.divmod(np.arange(n), width)
    table["s"] = np.arange(n) % 5
    samples = (abi.SampleIndex * n).from_buffer_copy(table.tobytes())
    rays, status = ctx.camera_rays(camera, samples)
    assert not status.any()
    paths = np.zeros(n, dtype=[("ray", "V48"), ("sample", "V24"), ("reserved", "<u8")])
    paths["ray"], paths["sample"] = np.frombuffer(rays, "V48"), np.frombuffer(samples, "V24")
    return (abi.PathInput * n).from_buffer_copy(paths.tobytes())


def trace(builder, capacity, inputs, options, instrumentation=0):
    options.instrumentation = instrumentation
    with runtime.Context(0, path_capacity=capacity) as ctx:
        scene = ctx.create_scene(builder)
        results, report = ctx.trace_paths(scene, inputs, options)
        scene.close()
    return results, (report.extension_segments, report.shadow_segments, report.failed_lanes)


def every_route_scene():
    """All eleven shading routes: eleven closure sequences over the generic ones, single conductor and dielectric
    instances, Lambert walls and misses through the open front."""
    builder = scenes.SceneBuilder()
    scenes.cornell_box(builder, with_spheres=True)
    box = builder.add_mesh(scenes.unit_box())
    for i, closures in enumerate(sequences(builder.nanometers)):
        builder.add_instance(box, builder.add_material(closures), scenes.uniform_scale_translate(
            0.2, (-0.75 + 0.3 * (i % 6), 0.2 + 0.3 * (i // 6), 0.6 + 0.1 * (i % 3))))
    return builder


def test_every_route_in_a_long_queue_matches_the_oracle():
    """25,600 slots take the three-launch compaction with eleven routes, 4,096 the one-block form."""
    builder = every_route_scene()
    options = abi.default_options(mis="power", max_depth=6)
    with runtime.Context(0, path_capacity=1 << 10) as ctx:
        inputs = camera_paths(ctx, 25_600, 160)
    many, counts = trace(builder, 1 << 15, inputs, options)
    few, few_counts = trace(builder, 1 << 12, inputs, options)
    assert bytes(many) == bytes(few) and counts == few_counts
    oracle = Oracle(device_trig=True)
    handle = oracle.scene(builder)
    expected, _ = oracle.trace(handle, inputs, options)
    oracle.destroy(handle)
    got, want = arrays(many), arrays(expected)
    assert np.array_equal(got["lane_status"] != 0, want["lane_status"] != 0)
    keep = want["lane_status"] == 0
    assert keep.mean() > 0.99
    check_paths({k: v[keep] for k, v in got.items()}, {k: v[keep] for k, v in want.items()}, "every route")


@pytest.mark.parametrize("n", [CHAIN_SLOTS, CHAIN_SLOTS + 1, 300_001])
def test_long_unchained_traces_equal_chained_and_instrumented_ones(n):
    builder = scenes.cornell_box(scenes.SceneBuilder(), with_spheres=True)
    options = abi.default_options(mis="power", max_depth=8)
    with runtime.Context(0, path_capacity=1 << 10) as ctx:
        inputs = camera_paths(ctx, n, 1024)
    whole, counts = trace(builder, 1 << 19, inputs, options)  # unchained beyond 2^18 paths
    assert counts[0] > n and counts[1] > 0
    for capacity, instrumentation in [(CHAIN_SLOTS, 0), (1 << 16, 0), (1 << 19, 1)]:
        other, other_counts = trace(builder, capacity, inputs, options, instrumentation)
        assert other_counts == counts, (capacity, instrumentation)
        assert bytes(other) == bytes(whole), (capacity, instrumentation)
    part, _ = trace(builder, 1 << 12, (abi.PathInput * 5000)(*inputs[:5000]), options)
    assert bytes(part) == bytes(whole)[:128 * 5000]
