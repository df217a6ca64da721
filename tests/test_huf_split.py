"""Runs of a Huffman stream (host logic, no GPU): they start where codes can
start, also where all code lengths have a common divisor
(tests/native/huf_split_check.cpp)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("seed", [1, 2])
def test_runs_start_at_code_boundaries(tmp_path, seed):
    exe = str(tmp_path / "huf_split_check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-I",
                           os.path.join(ROOT, "openzl_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "native", "huf_split_check.cpp"), "-o", exe])
    r = subprocess.run([exe, str(seed)], capture_output=True, text=True)
    assert r.returncode == 0 and "bad=0" in r.stdout, (r.stdout[-2000:], r.stderr[-2000:])
