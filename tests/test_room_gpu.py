"""Listings of meetings that ask for more than their room are repeated for
fewer offsets, in the overlap (in one stage and in stages of a long list) and
in the full match: the results are the oracle's.  Whole numbers."""
import numpy as np
import pytest

from bench import block_stats
from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS, stream_dtype, stream_names
from tests.test_stats_gpu import deep

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from curc_b200 import Context
    with Context(0) as c:
        yield c


def results(ctx, seqs):
    ctx.block_run(seqs)
    return {nm: ctx.get(nm, dt) for nm, dt in
            list(STAGE_RESULTS.items()) + [(s, stream_dtype(s)) for s in stream_names(seqs.shape[1])]}


@pytest.mark.parametrize("n,L,genome", [(250_000, 100, 260_000), (1_600_000, 60, 1_000_000)])
def test_overlap_listing_repeated(ctx, n, L, genome):
    seqs = deep(n, L, genome, 3)
    ora = OracleBlock(seqs)
    got = results(ctx, seqs)
    st = block_stats(ctx)
    offs = min(L * 65 // 100 - 1, 8 if st["overlap_suffixes"] > 1 << 19 else 10**6)
    met = st["overlap_suffixes"] / genome * offs * st["overlap_suffixes"]  # of the first listing
    assert met > 1.1 * max(4 << 20, 2 * st["overlap_suffixes"])
    bad = [nm for nm, v in got.items() if not np.array_equal(v, ora.get(nm, v.dtype.type))]
    assert not bad, bad


def test_full_match_listing_repeated(ctx):
    """Reads that start and end in one letter 85 bases long meet each other at
    every length from 16 to 85, and overlap nowhere: 70 meetings a read, with
    room for 67 and fewer."""
    n, L, k = 62_000, 250, 85
    rng = np.random.default_rng(8)
    seqs = synth.ACGT[rng.integers(0, 4, size=(n, L))]
    seqs[:, :k] = ord("A")
    seqs[:, -k:] = ord("A")
    default = ctx.tuning()
    listed = results(ctx, seqs)
    ctx.set_tuning(**dict(default, fm_loop=0))
    passes = results(ctx, seqs)
    ctx.set_tuning(**default)
    assert len(listed["unmatch_ids"]) > n - 10
    bad = [nm for nm in listed if not np.array_equal(listed[nm], passes[nm])]
    assert not bad, bad
