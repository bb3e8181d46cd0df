"""FP64 operations in integer arithmetic (csrc/sbr_soft64.cuh): the device's own
compilation against its FP64 instructions, and the host's with the FP32 seeds off
by more than the device's 2^-22."""
import os
import subprocess

import pytest

from sbrsolver_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sbrsolver_gb300", "csrc")


def _run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_device_soft64_gives_the_devices_bits(tmp_path):
    exe = str(tmp_path / "soft64_device_check")
    build.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off",
               "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "soft64_device_check.cu"), "-o", exe])
    _run(exe, str(1 << 22))


@pytest.mark.parametrize("seed_error", ["3.5e-7f", "-3.5e-7f"])
def test_soft64_holds_beyond_the_devices_seed_error(tmp_path, seed_error):
    exe = str(tmp_path / "soft64_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off",
                    f"-DSBR_SOFT64_SEED_ERROR={seed_error}", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "soft64_check.cpp"), "-o", exe], check=True)
    _run(exe, "3000000")
