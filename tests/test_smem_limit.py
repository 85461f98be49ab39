"""The kernels' dynamic shared-memory limits only rise (crd_b200/csrc/smem_limit.hpp): the rule checked on the host with
a stand-in for the CUDA call (tests/cpp/smem_limit_check.cpp, compiled with g++), and every launcher goes through it."""

from __future__ import annotations

import glob
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "crd_b200", "csrc")


def test_limit_never_falls(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ missing")
    exe = str(tmp_path / "smem_limit_check")
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-Wall", "-pthread", "-I", CSRC,
                        os.path.join(ROOT, "tests", "cpp", "smem_limit_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "smem limit ok" in r.stdout, r.stdout + r.stderr


def test_every_launcher_asks_here():
    for path in glob.glob(os.path.join(CSRC, "*")):
        if os.path.isfile(path) and os.path.basename(path) != "smem_limit.hpp":
            with open(path) as f:
                assert "cudaFuncAttributeMaxDynamicSharedMemorySize" not in f.read(), path
