"""Device memory of ray queries: the context keeps staging for small and moderate calls; a large call gives its
memory back."""
import ctypes as C

import numpy as np
import pytest

from bf200 import abi, runtime, scenes

pytestmark = pytest.mark.gpu

KEPT = 128 << 20
RAY = np.dtype([("o", "<f4", 3), ("d", "<f4", 3), ("t", "<f4", 2), ("time", "<f4"), ("mask", "<u4"), ("rest", "<u4", 2)])


def ray_table(n, seed):
    rng = np.random.default_rng(seed)
    table = np.zeros(n, RAY)
    table["o"] = rng.uniform([-0.95, 0.3, 0.05], [0.95, 0.95, 1.95], (n, 3))
    table["d"] = rng.normal(size=(n, 3))
    table["t"], table["time"], table["mask"] = [0.0, np.inf], scenes.PATH_TIME, 0xFFFFFFFF
    return table


def records(table):
    return (abi.Ray * len(table)).from_buffer(table)


def device_bytes(context):
    out = C.c_uint64()
    f = runtime.library().bf200_context_device_bytes
    f.argtypes, f.restype = [C.c_void_p, C.POINTER(C.c_uint64)], C.c_uint32
    assert f(context.handle, C.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("kind", ["hits", "occlusions"])
def test_large_queries_release_their_memory(kind):
    per_ray = RAY.itemsize + (C.sizeof(abi.Hit) if kind == "hits" else 4)
    most = KEPT // per_ray - 512  # its span stays within the kept bytes
    large = KEPT // per_ray + 100_000
    table = ray_table(large, 5)
    builder = scenes.cornell_box(scenes.SceneBuilder(), with_spheres=True)
    with runtime.Context(0, path_capacity=1 << 12) as ctx:
        scene = ctx.create_scene(builder)

        def query(part):
            answers = (ctx.closest_hits if kind == "hits" else ctx.occlusions)(scene, records(part))
            return np.frombuffer(answers, np.uint8).copy()

        whole = query(table)
        assert device_bytes(ctx) == 0
        few = query(table[:1000])
        assert 0 < device_bytes(ctx) <= 1000 * per_ray + 256
        part = query(table[:most])
        kept = device_bytes(ctx)
        assert KEPT - 1024 * per_ray < kept <= KEPT
        again = query(table)
        assert device_bytes(ctx) == kept
        scene.close()
    assert np.array_equal(whole, again)
    assert np.array_equal(whole[:len(part)], part) and np.array_equal(part[:len(few)], few)
