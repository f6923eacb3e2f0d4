"""Reads around the mapping's k-mer length (28): shorter ones are not probed,
whatever their last bases.  Whole numbers: equal to the oracle."""
import numpy as np
import pytest

from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS, stream_dtype, stream_names

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", range(24, 33))
def test_mapping_of_short_reads(L):
    """A genome of which A is half, so that many 28-mers end in the base that
    pads a packed read of 27."""
    from curc_b200 import Context
    rng = np.random.default_rng(L)
    g = synth.ACGT[rng.choice(4, p=[0.5, 0.2, 0.15, 0.15], size=3000)]
    reads = np.lib.stride_tricks.sliding_window_view(g, L)[rng.integers(0, len(g) - L + 1, size=6000)].copy()
    err = rng.random(reads.shape) < 0.01
    reads[err] = synth.ACGT[rng.integers(0, 4, size=int(err.sum()))]
    reads[rng.random(reads.shape) < 0.001] = ord("N")
    ora = OracleBlock(reads)
    with Context(0) as ctx:
        ctx.block_run(reads)
        names = list(STAGE_RESULTS.items()) + [(s, stream_dtype(s)) for s in stream_names(L)]
        bad = [nm for nm, dt in names if not np.array_equal(ctx.get(nm, dt), ora.get(nm, dt))]
    assert not bad, bad
