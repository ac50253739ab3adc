"""The wait of a long render: a process whose device is set to blocking waits spends little processor time in it,
and the film is the same as with the default flags."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BLOCKING = 4  # CU_CTX_SCHED_BLOCKING_SYNC

PROGRAM = """
import ctypes, sys, time
import numpy as np
driver = ctypes.CDLL("libcuda.so.1")
device = ctypes.c_int()
assert driver.cuInit(0) == 0 and driver.cuDeviceGet(ctypes.byref(device), 0) == 0
if int(sys.argv[1]):
    assert driver.cuDevicePrimaryCtxSetFlags_v2(device, int(sys.argv[1])) == 0
from bf200 import abi, runtime, scenes
from helpers import sensor_from_golden
golden = dict(np.load(sys.argv[2]))
builder = scenes.cornell_box(scenes.SceneBuilder(), with_spheres=True)
options = abi.default_options(mis="power", max_depth=16)
camera = runtime.camera_create(*scenes.camera_frame_inputs(), 256, 256, scenes.CAMERA_VFOV, scenes.PATH_TIME)
with runtime.Context(0) as ctx:
    scene = ctx.create_scene(builder)
    render = lambda: ctx.render_film(scene, camera, sensor_from_golden(golden), options, 256)
    render()
    wall, own = time.perf_counter(), time.thread_time()
    sums, counts, report = render()
    wall, own = time.perf_counter() - wall, time.thread_time() - own
    scene.close()
np.savez(sys.argv[3], sums=sums, counts=counts, share=own / wall, segments=report.extension_segments)
"""


def render(repo_root, tmp_path, flags):
    out = str(tmp_path / f"film{flags}.npz")
    env = dict(os.environ)
    env["PYTHONPATH"] = os.pathsep.join([os.path.join(repo_root, "blackframe-renderer_b200"), repo_root,
                                         os.path.join(repo_root, "tests")])
    golden = os.path.join(repo_root, "tests", "golden", "cornell_spheres_256.npz")
    subprocess.run([sys.executable, "-c", PROGRAM, str(flags), golden, out], check=True, env=env, timeout=300)
    return dict(np.load(out))


def test_blocking_waits_leave_the_processor_free(repo_root, tmp_path):
    plain, blocking = render(repo_root, tmp_path, 0), render(repo_root, tmp_path, BLOCKING)
    assert np.array_equal(plain["sums"].view(np.uint32), blocking["sums"].view(np.uint32))
    assert np.array_equal(plain["counts"], blocking["counts"]) and plain["segments"] == blocking["segments"]
    print(f"thread's share of the call: {plain['share']:.2f} default flags, {blocking['share']:.2f} blocking")
    assert blocking["share"] < 0.5
