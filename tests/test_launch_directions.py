"""Launch directions subdivided on the device against the host's, bit for bit:
no level, the first, those where one block scans the half-edges and those where
many do."""
import os
import subprocess

import pytest

from sbrsolver_gb300 import build

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_device_directions_are_the_hosts(built, tmp_path):
    exe = str(tmp_path / "dirs_check")
    csrc = os.path.join(ROOT, "sbrsolver_gb300", "csrc")
    build.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off",
               "-I", csrc, "-I", os.path.join(ROOT, "include"),
               os.path.join(ROOT, "tests", "cpp", "dirs_check.cu"),
               os.path.join(csrc, "sbr_host.cpp"), "-o", exe])
    r = subprocess.run([exe, "0", "1", "2", "3", "4", "5", "6", "7", "8"], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
