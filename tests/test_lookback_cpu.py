"""The two-level look-back with its warp run as 32 host threads whose reads of a published word
become visible at different times (tests/lookback_host.cpp): every lane must reach every vote and
shuffle of the function, and all must return the prefix."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "massively_b200", "csrc")


def test_lanes_leave_every_wait_together(tmp_path):
    # The header is compiled alone: what it includes is defined by the host file.
    shutil.copy(os.path.join(CSRC, "lookback_group.cuh"), tmp_path)
    (tmp_path / "lookback.cuh").write_text("#pragma once\n")
    exe = str(tmp_path / "lookback_host")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-w", f"-I{tmp_path}",
                    os.path.join(HERE, "lookback_host.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
