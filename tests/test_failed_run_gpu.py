"""What a block run that fails late leaves behind (an allocation that the host
refuses; tests/helpers/failed_run_check.cu)."""
import os
import shutil
import subprocess

import pytest

from curc_b200._native import LIB_PATH

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_a_failed_run_names_no_streams(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe, where = str(tmp_path / "failed_run_check"), os.path.dirname(LIB_PATH)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    os.path.join(HERE, "helpers", "failed_run_check.cu"), "-o", exe, "-L", where, "-lcurc_b200",
                    "-Xlinker", f"-rpath={where}"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
