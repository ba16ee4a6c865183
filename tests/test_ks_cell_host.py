"""The FP64 Kerr-Schild cell, the recovery's root solve, the limiter and the
face flux against the general functions they replace, on the CPU
(tests/ks_cell_check.cu)."""
import os
import subprocess

from grdzhadzha_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_ks_cell_matches_general_functions(tmp_path):
    exe = str(tmp_path / "ks_cell_check")
    subprocess.run([B.nvcc(), "-std=c++17", "-O2", "-I", B.CSRC, "-Xcompiler",
                    "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "ks_cell_check.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
