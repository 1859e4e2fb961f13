"""The solve's CSR kernels walk a row's links eight at a time in 32-bit
indices (interflect_b200/csrc/rowspan.h). This compiles the header for the host
and walks rows up to the last link that 32 bits can number, where sums of
indices wrap; no GPU holds a matrix of that size."""
import os
import subprocess

from conftest import ROOT


def test_rows_are_walked_to_their_ends(tmp_path):
    exe = str(tmp_path / "rowspan_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "rowspan_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "rows walked to their ends" in r.stdout
