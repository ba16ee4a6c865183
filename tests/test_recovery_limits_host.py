"""What the recovery's two root solves report at their limits, on the CPU
(tests/recovery_limits_check.cu)."""
import os
import subprocess

from grdzhadzha_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_root_solves_report_alike(tmp_path):
    exe = str(tmp_path / "recovery_limits_check")
    subprocess.run([B.nvcc(), "-std=c++17", "-O2", "-I", B.CSRC, "-Xcompiler",
                    "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "recovery_limits_check.cu")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
