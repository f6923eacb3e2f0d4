"""What a block run that fails late leaves behind (an allocation that the host
refuses; tests/helpers/failed_run_check.cu)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from curc_b200._native import LIB_PATH
from tests.cases import CASES

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


@pytest.mark.parametrize("then", ["refused run", "trim"])
def test_the_learned_coder_has_no_block_left(then):
    """Its anchors come from the last block's records in the device arena."""
    from curc_b200 import Context, CurcError
    from curc_b200._native import Learner
    seqs, po, pe = CASES["se75_20k"]()
    with Context(0) as ctx, Learner(0) as lrn:
        ctx.block_run(seqs, po, pe)
        lrn.add_block(ctx)
        first = lrn.anchors
        if then == "trim":
            ctx.trim()
        else:
            with pytest.raises(CurcError):
                ctx.block_run(np.full((3, 513), ord("A"), dtype=np.uint8))
        lrn.add_block(ctx)
        assert first > 0 and lrn.anchors == first
        ctx.block_run(seqs, po, pe)
        lrn.add_block(ctx)
        assert lrn.anchors == 2 * first
