"""``fa::launch_dependent`` (csrc/host_common.h) when a launch fails, on the host with a stand-in runtime."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_failed_launch_leaves_no_pending_error(tmp_path):
    nvcc = os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    exe = tmp_path / "launch_host"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include"),
                    "-I", os.path.join(ROOT, "flash-attention-ptx-cuda_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpu", "launch_host.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr
