"""The waits of the dataflow launches' warps (csrc/rc_flowc.cuh) on processor
threads as lanes, with words that change between the lanes' readings: every
warp-wide operation is met by all lanes at the same place.  With lanes that
decide by their own readings the check has to notice it."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "rocketcombustor_gb300", "csrc")


@pytest.mark.parametrize("per_lane", [False, True])
def test_lanes_decide_together(tmp_path, per_lane):
    exe = str(tmp_path / "warp_wait")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", f"-I{CSRC}"] + (["-DPER_LANE"] if per_lane else []) +
                   ["-o", exe, os.path.join(HERE, "cuda", "warp_wait_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert (r.returncode != 0) == per_lane, r.stdout + r.stderr
    assert r.stdout.startswith("mismatches 0 errors 0") != per_lane
