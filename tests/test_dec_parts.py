"""Which frames of a batch decode ahead of the others because of their content
checksums (host logic, no GPU; tests/native/dec_parts_check.cpp)."""
import os
import subprocess

from conftest import ROOT


def test_rule_for_long_checksums(tmp_path):
    exe = str(tmp_path / "dec_parts_check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-I",
                           os.path.join(ROOT, "openzl_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "native", "dec_parts_check.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "bad=0" in r.stdout, (r.stdout[-2000:], r.stderr[-2000:])
