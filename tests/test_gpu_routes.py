"""The generic shading routes: one per sequence of closure kinds, the last for all further ones."""
import numpy as np
import pytest

from bf200 import abi, runtime, scenes
from helpers import arrays, check_paths
from oracle.bindings import Oracle

pytestmark = pytest.mark.gpu


def sequences(nm):
    """Eleven materials of distinct closure-kind sequences, none of which a specialised kernel takes."""
    eta, k = scenes.tabulated_spectrum(scenes.GOLD_ETA, nm), scenes.tabulated_spectrum(scenes.GOLD_K, nm)
    lambert = scenes.lambertian([0.3] * 4)
    rough = scenes.rough_diffuse([0.3, 0.35, 0.4, 0.3], 0.5)
    metal = scenes.rough_conductor([0.3] * 4, eta, k, 0.3, 0.2)
    mirror = scenes.specular_reflection([0.25] * 4)
    return [rough, mirror, lambert + rough, rough + lambert, lambert + metal, metal + lambert, rough + metal,
            metal + rough, lambert + mirror, mirror + lambert, lambert + rough + metal]


@pytest.mark.parametrize("count", [1, 6, 7, 8, 11])
def test_paths_of_many_closure_sequences_match_the_oracle(count):
    builder = scenes.SceneBuilder()
    scenes.cornell_box(builder, with_spheres=False)
    materials = [builder.add_material(m) for m in sequences(builder.nanometers)[:count]]
    box = builder.add_mesh(scenes.unit_box())
    for i, material in enumerate(materials):
        builder.add_instance(box, material, scenes.uniform_scale_translate(
            0.2, (-0.75 + 0.3 * (i % 6), 0.2 + 0.3 * (i // 6), 0.6 + 0.1 * (i % 3))))
    options = abi.default_options(mis="power", max_depth=6)
    width = height = 24
    camera = runtime.camera_create(*scenes.camera_frame_inputs(), width, height, scenes.CAMERA_VFOV, scenes.PATH_TIME)
    samples = (abi.SampleIndex * (width * height))()
    for i in range(width * height):
        samples[i].pixel_x, samples[i].pixel_y, samples[i].sample_index = i % width, i // width, i % 5
    oracle = Oracle(device_trig=True)
    handle = oracle.scene(builder)
    with runtime.Context(0, path_capacity=1 << 12) as ctx:
        scene = ctx.create_scene(builder)
        rays, status = ctx.camera_rays(camera, samples)
        assert not status.any()
        inputs = (abi.PathInput * len(samples))()
        for i, ray in enumerate(rays):
            inputs[i].primary_ray, inputs[i].sample = ray, samples[i]
        results, _ = ctx.trace_paths(scene, inputs, options)
        scene.close()
    expected, _ = oracle.trace(handle, inputs, options)
    oracle.destroy(handle)
    got, want = arrays(results), arrays(expected)
    assert np.array_equal(got["lane_status"] != 0, want["lane_status"] != 0)
    keep = want["lane_status"] == 0
    assert keep.mean() > 0.99 and got["radiance"][keep].any()
    check_paths({k: v[keep] for k, v in got.items()}, {k: v[keep] for k, v in want.items()}, f"{count} sequences")


@pytest.mark.parametrize("n", [0, 1, 31, 33, 1023, 1024, 1025, 16383, 16384, 16385])
@pytest.mark.parametrize("routes", [1, 3, 4])
def test_one_block_compaction_keeps_slot_order(n, routes):
    """Queues of up to 16,384 slots come from one block, longer ones from three launches."""
    import torch
    rng = np.random.default_rng(n + routes)
    keys = rng.choice(np.array([*range(routes), 0xFF], np.uint8), max(n, 1))
    device = torch.from_numpy(keys).cuda()
    queue = torch.full((max(n, 1),), -1, dtype=torch.int32, device="cuda")
    offsets = torch.zeros(routes + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with runtime.Context(0, path_capacity=1 << 12) as ctx:
        ctx.compact_routes_device(device.data_ptr(), n, routes, queue.data_ptr(), offsets.data_ptr())
    wanted = [np.nonzero(keys[:n] == r)[0] for r in range(routes)]
    ends = np.cumsum([0] + [len(w) for w in wanted])
    assert np.array_equal(offsets.cpu().numpy(), ends)
    assert np.array_equal(queue.cpu().numpy()[:ends[-1]], np.concatenate(wanted))
