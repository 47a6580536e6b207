"""The copying thread of the banded preconditioner's shared-memory ring, on the CPU.

``channel3d_parallel_b200/csrc/copy_ring.cuh`` is compiled with g++ against a
model of its barriers.  Whatever gives up (readers that stop releasing slots, a
copy that never lands), it must bring no block into a slot that is not released,
report the failure, and end with none of its copies in flight.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_copy_ring(tmp_path):
    exe = str(tmp_path / "copy_ring_check")
    src = os.path.join(HERE, "host_kernels", "copy_ring_check.cpp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(HERE, "host_kernels"), src, "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert ", 0 mismatches" in r.stdout
