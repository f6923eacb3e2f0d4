"""The overlap walk on both sides of its limits: offsets with more meetings
than one block takes (2048), runs of as many suffixes and prefixes as a thread
pairs in registers (4) and more, and reads that meet themselves.  Whole
numbers: equal to the oracle."""
import numpy as np
import pytest

from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 3, 4, 5, 9, 40])
@pytest.mark.parametrize("n", [1500, 16_000])
def test_runs_of_copies(copies, n):
    """Every segment lies `copies` times between spacers of its own, so that
    reads into and out of it share their ends."""
    from curc_b200 import Context
    rng = np.random.default_rng([copies, n])
    L, parts = 60, []
    while sum(map(len, parts)) < n:
        seg = synth.ACGT[rng.integers(0, 4, size=90)]
        if len(parts) % 5 == 0:
            seg = np.resize(seg[:7], 90)  # a short period
        for _ in range(copies):
            parts += [seg, synth.ACGT[rng.integers(0, 4, size=40)]]
    g = np.concatenate(parts)
    reads = np.lib.stride_tricks.sliding_window_view(g, L)
    seqs = reads[rng.permutation(len(reads))[:n]].copy()
    ora = OracleBlock(seqs)
    with Context(0) as ctx:
        ctx.block_run(seqs)
        bad = [nm for nm, dt in STAGE_RESULTS.items() if not np.array_equal(ctx.get(nm, dt), ora.get(nm, dt))]
    assert not bad, bad
