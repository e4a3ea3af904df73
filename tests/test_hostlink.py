"""The blocks of host memory that transfers pass through
(csrc/dsmc_hostlink.h), on the CPU with a stand-in for the CUDA runtime
(tests/cpp/fake_cuda): values at the ends of a block, through ordinary and
page-locked memory and where none can be page-locked; a handle's first small
transfers page-lock nothing, and the others the blocks of the threads they
use; the blocks are left out of a fork."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_hostlink_blocks(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = os.path.join(str(tmp_path), "hostlink_test")
    cpp = os.path.join(ROOT, "tests", "cpp")
    cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-pthread",
           "-I", os.path.join(cpp, "fake_cuda"), "-I", os.path.join(ROOT, "dig-appolo_b200", "csrc"),
           os.path.join(cpp, "hostlink_test.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
