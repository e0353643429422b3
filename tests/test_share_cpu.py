"""How a persistent FP32 launch shares few items out over its warps
(csrc/ldp_share.h), on the CPU: share_check.cpp goes over launch shapes, those
of fewer warps to an SM than schedulers among them, and item counts."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "langevindynamicsforpcp_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_one_launch_claims_every_item(tmp_path):
    exe = tmp_path / "share_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-I", CSRC, os.path.join(HERE, "share_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
