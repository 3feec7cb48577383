"""The table gathers that the mu/M kernels share among a block's points
(pf5d_gather.cuh), compiled for the host and run by 128 threads: every index
stays inside its array (address and undefined-behaviour sanitizers), no two
threads touch a word without a barrier between them (thread sanitizer), and
each point gets the bits and the flags of an evaluation by itself.  Blocks of
all sizes K and PER, partly filled ones among them; points of one cell, of
cells that share a bin, outside the linear region, far off the simplex and not
finite."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "phasefield5d_b200", "csrc")


@pytest.mark.parametrize("sanitizer", ["address,undefined", "thread"])
def test_block_stays_in_bounds_and_without_races(tmp_path, sanitizer):
    exe = str(tmp_path / "gather")
    # the stand-ins' folder comes first: their cuda_runtime.h is the one that is found
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-w", f"-fsanitize={sanitizer}",
                    "-fno-sanitize-recover=all", "-ffp-contract=off",
                    "-I", os.path.join(HERE, "host_block"), "-I", CSRC,
                    os.path.join(HERE, "host_block", "gather.cpp"), "-o", exe, "-lpthread"],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
