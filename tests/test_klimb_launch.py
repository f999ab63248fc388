"""CPU: the K-limb passes' launch shapes (csrc/klimb_plan.hpp) against what the
kernel is built for, by a small g++ program."""
import os
import subprocess

from conftest import ROOT


def test_launch_shapes(tmp_path):
    exe = str(tmp_path / "klimb_launch_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror",
                        "-I" + os.path.join(ROOT, "ntt-tensorcore_b200", "csrc"),
                        os.path.join(ROOT, "tests", "klimb_launch_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-2000:]
