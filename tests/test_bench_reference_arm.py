"""bench.py on a machine without the reference build: the reference arm and the CPU baseline of the product's
line say so, and neither loses the line."""
import json
import types

import pytest

import bench
import oracle.bindings


@pytest.fixture
def no_reference(monkeypatch):
    monkeypatch.setattr(oracle.bindings, "reference_available", lambda: False)


def test_the_reference_arm_prints_its_unavailable_line(no_reference, capsys):
    args = types.SimpleNamespace(workload="cornell_plain_64", warmup=0, steps=1, reference_seconds=0.1)
    bench.run_reference_arm(args, 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "libbfref.so" in line["unavailable"] and "\n" not in line["unavailable"]


def test_the_reference_cuda_arm_prints_its_unavailable_line(no_reference, capsys):
    bench.run_reference_cuda_arm(types.SimpleNamespace(workload="cornell_plain_64"), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference-cuda" and "libbfrefcuda.so" in line["unavailable"]


def test_the_cpu_baseline_is_marked_unavailable(no_reference):
    assert list(bench.cpu_baseline("cornell_plain_64", 0.1)) == ["unavailable"]
