"""Launch shapes of the FSE decoder (host logic, no GPU): what the autotuner
times (tests/native/fse_shape_check.cpp)."""
import os
import subprocess

from conftest import ROOT


def test_autotuner_times_the_untuned_shape(tmp_path):
    exe = str(tmp_path / "fse_shape_check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-I",
                           os.path.join(ROOT, "openzl_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "native", "fse_shape_check.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "bad=0" in r.stdout, (r.stdout[-2000:], r.stderr[-2000:])
