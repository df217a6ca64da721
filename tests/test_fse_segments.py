"""Segments of the long FSE chunks (host logic, no GPU): what each thread of
kFseEncLong reads of the coding table before the first barrier, and the counts
that follow (tests/native/fse_segments_check.cpp)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.parametrize("seed", [1, 2])
def test_threads_count_their_own_symbols(tmp_path, seed):
    exe = str(tmp_path / "fse_segments_check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-I",
                           os.path.join(ROOT, "openzl_gb300", "csrc"),
                           os.path.join(ROOT, "tests", "native", "fse_segments_check.cpp"), "-o", exe])
    r = subprocess.run([exe, str(seed)], capture_output=True, text=True)
    assert r.returncode == 0 and "bad=0" in r.stdout, (r.stdout[-2000:], r.stderr[-2000:])
