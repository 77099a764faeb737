"""The big-triangle queue's entries where chunk numbers run past 32 bits
(big_queue.cuh), host-compiled: a dropped triangle leaves an entry that covers
nothing, never one of an earlier pass."""
import os
import subprocess
import tempfile

from tests.conftest import ROOT


def test_dropped_triangles_leave_empty_entries():
    src = os.path.join(ROOT, "tests", "native", "big_queue_check.cpp")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "big_queue_check")
        subprocess.run(["g++", "-O2", "-std=c++17", "-fsanitize=address,undefined", "-fno-sanitize-recover", "-I",
                        os.path.join(ROOT, "lighthugger_gb300", "csrc"), src, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad 0" in r.stdout
