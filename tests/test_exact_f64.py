"""The double operations that FP64 Hydro runs on the integer pipes
(csrc/exact_f64.cuh), compiled for the host and compared with the host's own
IEEE operations bit for bit."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "paraiso_gb300", "csrc")


def test_integer_double_operations_are_ieee(tmp_path):
    exe = str(tmp_path / "check")
    # no contraction: aarch64 GCC would fuse the reference expressions
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", f"-I{CSRC}",
                    os.path.join(HERE, "cpp", "exact_f64_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "5000000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
