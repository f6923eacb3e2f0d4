"""Waits of the one-launch scan, selection, sort and compaction never end in a
void result: a tile that has waited long enough counts the tiles before it
itself (tests/helpers/lookback_check.cu, built with no and with the usual
waits, against the standard library; whole numbers, so equal).  And no run
depends on work of the default stream."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.cases import CASES
from tests.oracle_lib import STAGE_RESULTS

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("spins", ["0", "3", "(1u<<22)"])
def test_tiles_that_do_not_wait_count_themselves(tmp_path, spins):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "lookback_check")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    f"-DCURC_LOOK_SPINS={spins}", os.path.join(HERE, "helpers", "lookback_check.cu"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_first_block_while_the_default_stream_is_busy():
    import torch
    from curc_b200 import Context
    seqs, po, pe = CASES["pe133_po_tail"]()
    with Context(0) as ctx:
        ctx.block_run(seqs, po, pe)
        want = {n: ctx.get(n, dt) for n, dt in STAGE_RESULTS.items()}
    with Context(0) as ctx:
        torch.cuda._sleep(200_000_000)  # a tenth of a second of the default stream
        ctx.block_run(seqs[:0], po, pe)
        ctx.block_run(seqs, po, pe)
        assert all(np.array_equal(want[n], ctx.get(n, dt)) for n, dt in STAGE_RESULTS.items())
        torch.cuda.synchronize()
