"""What the training kernel does after a wait for its MMAs ran out (csrc/mma_drain.h), on a host model of the
barrier: nothing may be in flight when the tensor-memory columns are freed."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_nothing_is_in_flight_after_a_timeout(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "drain_check")
    r = subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", "-I" + os.path.join(HERE, "..", "swpathtracer_b200", "csrc"),
                        os.path.join(HERE, "drain_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
