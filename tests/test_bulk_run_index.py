"""bulk_runs_kernel's index at the run counts of the largest bulk lists, checked
on the host (2^27 runs are a list of tens of GB)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_runs_past_2_to_the_27(tmp_path):
    exe = str(tmp_path / "bulk_run_index")
    subprocess.run([NVCC, "-std=c++17", "-ccbin", "/usr/bin/g++", "--expt-relaxed-constexpr",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    os.path.join(ROOT, "biofvm_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-o", exe, os.path.join(ROOT, "tests", "native", "bulk_run_index.cu")],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
