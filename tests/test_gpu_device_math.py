"""The approximate forms that decide a byte of the display transform and a
normal-cone test, compared on the device with the plain forms they stand for:
every float, and 159 million cones of which three quarters lie at their cutoff."""
import os
import subprocess
import tempfile

import pytest

from lighthugger_gb300 import build
from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


def test_approximate_decisions_are_the_plain_ones():
    src = os.path.join(ROOT, "tests", "native", "device_math_check.cu")
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "device_math_check")
        subprocess.run([build.NVCC] + build.ARCH + build.NVCC_FLAGS + ["-cudart", "static", src, "-o", exe], check=True,
                       capture_output=True)
        r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bytes 4294967296 bad 0" in r.stdout and r.stdout.rstrip().endswith("bad 0"), r.stdout
