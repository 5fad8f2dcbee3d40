"""The order in which the decode step kernel refills its ring (csrc/ring_order.h), in a model of the ring on the CPU: warps at
random speeds, barriers waited on by phase parity."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compile(folder, *flags):
    exe = os.path.join(str(folder), "ring_model")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-Wall", *flags, "-I", os.path.join(ROOT, "ml-drift_b200", "csrc"), "-o", exe,
                           os.path.join(ROOT, "tests", "ring_model.cc")])
    return exe


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("ring"))


# 12 is the shortest ring that the kernel takes (a stage per warp and one), 20 to 24 what shared memory leaves it, 32 a lane
# of the producer per stage; 21 is the shortest where all eleven warps take attention tiles
@pytest.mark.parametrize("stages", [12, 13, 16, 20, 21, 22, 23, 24, 32])
def test_no_wait_passes_in_another_phase(model, stages):
    out = subprocess.run([model, str(stages), "150", "1"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout


@pytest.mark.parametrize("stages", [12, 16, 20, 21, 24])
def test_the_model_tells_boxes_asked_for_out_of_order(tmp_path, stages):
    out = subprocess.run([_compile(tmp_path, "-DUNORDERED"), str(stages), "150", "1"], capture_output=True, text=True, timeout=300)
    assert out.returncode == 1 and "not" in out.stdout
