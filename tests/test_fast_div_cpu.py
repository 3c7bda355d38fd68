"""``fa::FastDiv`` (csrc/fast_div.h), the division of the kernels' work lists, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fast_div_is_exact(tmp_path):
    exe = tmp_path / "fast_div_host"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "flash-attention-ptx-cuda_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpu", "fast_div_host.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr
