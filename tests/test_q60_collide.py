"""The F64_Q60 collision's shortened products, its branch for positive nodes and its range test against a plain
formulation on the host, bit for bit (csrc/plbm_q60.cuh)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_products_and_relaxation(tmp_path, seed):
    out = str(tmp_path / "q60_test")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fwrapv", "-I", os.path.join(ROOT, "portlbm_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "q60_test.cpp"), "-o", out], check=True)
    r = subprocess.run([out, "300000", str(seed)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert int(r.stdout.split()[-1]) > 400000
