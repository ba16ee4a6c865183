"""The reverse of a recovery decides at the floors as the forward did, on the
CPU (tests/adjoint_floors_check.cu)."""
import os
import subprocess

from grdzhadzha_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_reverse_floors_decide_as_the_forward(tmp_path):
    exe = str(tmp_path / "adjoint_floors_check")
    subprocess.run([B.nvcc(), "-std=c++17", "-O2", "-I", B.CSRC, "-Xcompiler",
                    "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "adjoint_floors_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
