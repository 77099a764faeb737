"""The face test without divisions (facing.cuh) against the plain IEEE form,
host-compiled."""
import os
import subprocess
import tempfile

from tests.conftest import ROOT


def test_faces_away_equals_the_ieee_form():
    src = os.path.join(ROOT, "tests", "native", "facing_check.cpp")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "facing_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "lighthugger_gb300", "csrc"), src, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad 0" in r.stdout
