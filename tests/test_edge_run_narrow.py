"""The 32-bit form of the chunk kernel's row runs (edge_run.cuh,
clip_run_as<int32_t>) against the 64-bit one, host-compiled, over triangles
up to the limit under which the kernel takes it."""
import os
import subprocess
import tempfile

from tests.conftest import ROOT


def test_narrow_runs_equal_the_wide_ones():
    src = os.path.join(ROOT, "tests", "native", "edge_run_narrow_check.cpp")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "edge_run_narrow_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fsanitize=signed-integer-overflow",
                        "-fno-sanitize-recover", "-I", os.path.join(ROOT, "lighthugger_gb300", "csrc"), src, "-o", exe],
                       check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad 0" in r.stdout
