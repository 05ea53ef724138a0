"""The ring that tracers pass through between the warps of a launch (csrc/ring.cuh),
compiled for the host and run under many interleavings of its memory operations: with
as few entries as tracers (one among them) no tracer is taken twice and none is lost."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ring") / "ring_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(HERE, "..", "rapt_gb300", "csrc"),
                    os.path.join(HERE, "ring_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("values", [1, 2, 5])
@pytest.mark.parametrize("agents", [2, 3, 8])
def test_no_value_is_taken_twice_or_lost(check, values, agents):
    r = subprocess.run([check, str(values), str(agents), "4000"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
    assert int(r.stdout.split()[1]) > 4000  # takes did happen
