"""The shading stage's fork and join of its streams, over a fake of the CUDA runtime (tests/branches_probe.cpp):
whichever call fails, the caller's wait for the main stream leaves no work of a branch in flight."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CUDA_INCLUDE = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def probe(repo_root, tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    library = tmp_path_factory.mktemp("branches") / "branches_probe.so"
    source = os.path.join(repo_root, "blackframe-renderer_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", f"-I{CUDA_INCLUDE}", f"-I{source}", "-o",
                    str(library), os.path.join(repo_root, "tests", "branches_probe.cpp")], check=True)
    return C.CDLL(str(library))


@pytest.mark.parametrize("branches", [0, 1])
def test_no_branch_work_outlives_a_failed_stage(probe, branches):
    made = C.c_int()
    assert probe.run_fork_join(0, branches, C.byref(made)) == 0
    calls = made.value
    assert calls == (14 if branches else 4)  # 1 + 3 to fork, 4 launches, 2 x 3 to join
    for failing in range(1, calls + 1):
        assert probe.run_fork_join(failing, branches, C.byref(made)) == 0, f"call {failing}"
