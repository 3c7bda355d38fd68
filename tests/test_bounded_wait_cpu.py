"""The give-up branch of the device-side waits, without a GPU.

Every wait in the kernels (mbarrier waits, the shared-memory slot poll) is one loop,
``fa::bounded_wait`` in ``csrc/bounded_wait.h``, written so that it also compiles for the host.
No test makes a GPU wait run out; instead the same code is built with g++ here and driven with
polls that never succeed and a fake clock (``tests/cpu/bounded_wait_host.cpp``), alone and as the 32
lanes of a warp of which only some run out of time.  The second test holds the kernels to the
warp-wide form, the third checks the host's mapping from a recorded status word to the error code of
the C ABI."""
import glob
import os
import re
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "flash-attention-ptx-cuda_b200", "csrc")


def test_give_up_branch_on_the_host(tmp_path):
    exe = tmp_path / "bounded_wait_host"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpu", "bounded_wait_host.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout.strip() == "ok", res.stdout + res.stderr


def test_no_kernel_leaves_a_loop_lane_by_lane():
    """Outside of ptx.cuh a kernel uses the voting waits, votes on ``bounded_wait`` itself, or votes on the
    ``LaneWaits`` that an issue or several waits share."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            text = f.read()
        assert not re.search(r"lane_(mbar_)?wait\(|mbar_try_wait", text), path
        polls = len(re.findall(r"\bbounded_wait\(", text))
        assert len(re.findall(r"__all_sync\(0xffffffffu, w == kWaitDone\)", text)) == polls, path
        for name in ("lw", "lq"):
            waits = list(re.finditer(r"\bLaneWaits " + name + r";", text))
            for m, end in zip(waits, [w.start() for w in waits[1:]] + [len(text)]):
                use = text[m.end():end]
                vote = re.search(r"warp_all\(" + name + r"\.ok\)", use)
                assert vote, (path, text.count("\n", 0, m.start()) + 1)
                rest = re.sub(r"elect_one\(\) && " + name + r"\.ok\)", "", use[:vote.start()].removesuffix("return "))
                assert name + ".ok" not in rest and not re.search(r"\b(break|return|continue)\b", rest), use
    with open(os.path.join(CSRC, "ptx.cuh")) as f:
        text = f.read()
    body = text[text.index("bool mbar_wait("):]
    assert "return warp_wait(" in body[:body.index("\n}\n")] and "warp_all);" in body[:body.index("\n}\n")]


def test_status_word_maps_to_device_timeout():
    sys.path.insert(0, ROOT)
    import __graft_entry__ as ge
    fa = ge.load_package()
    lib = fa.lib()
    assert lib.fa_status_word_to_error(0) == fa.FA_OK
    for barrier_id in (1, 14, 0x41, 0x4F):
        assert lib.fa_status_word_to_error((1 << 16) | barrier_id) == fa.FA_ERR_DEVICE_TIMEOUT
    assert fa.error_string(fa.FA_ERR_DEVICE_TIMEOUT) == "a kernel gave up on a bounded wait"
