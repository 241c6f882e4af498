"""The double operations that FP64 Hydro runs on the integer pipes
(csrc/exact_f64.cuh) on the device, with its approximate seeds, against the
device's own IEEE operations bit for bit: extreme operands pair by pair and
random ones near exact quotients and squares."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "paraiso_gb300", "csrc")


def test_device_operations_are_ieee(om_lib, tmp_path):
    from paraiso_gb300 import build
    exe = str(tmp_path / "check")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", f"-I{CSRC}",
                    os.path.join(HERE, "cpp", "exact_f64_device.cu"), "-o", exe], check=True)
    r = subprocess.run([exe, "400"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
