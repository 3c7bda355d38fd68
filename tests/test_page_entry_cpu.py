"""``fa::page_entry`` (csrc/page_entry.h), the block-table look-up of the paged cache, on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_page_entry_stays_inside_the_table(tmp_path):
    exe = tmp_path / "page_entry_host"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                    os.path.join(ROOT, "flash-attention-ptx-cuda_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpu", "page_entry_host.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr
