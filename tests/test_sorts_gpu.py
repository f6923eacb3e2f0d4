"""Sorts, scans and compactions at the edges of their tiles, through blocks
whose sizes lie there: up to 4096 reads (one launch), one and several tiles, runs of reads that share their first 32 bases of every length
around a thread's, a warp's and the radix path's limits.  Whole numbers: equal
to the oracle."""
import numpy as np
import pytest

from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from curc_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("n", [1, 2, 2047, 2048, 2049, 4095, 4096, 4097, 8193, 20_000])
@pytest.mark.parametrize("run", [1, 2, 4, 5, 32, 33, 300])
@pytest.mark.parametrize("L", [30, 33, 75, 140])
def test_read_order(ctx, n, run, L):
    rng = np.random.default_rng([n, run, L])
    heads = synth.ACGT[rng.integers(0, 4, size=(max(1, n // run), min(L, 32)))]
    reads = synth.ACGT[rng.integers(0, 4, size=(n, L))]
    reads[:, :32] = heads[rng.permutation(np.arange(n) % len(heads))]
    # repeated tails: equal reads, and reads that differ in their last base only
    tails = rng.integers(0, max(1, n // 3), size=n)
    reads[:, 32:] = reads[tails, 32:]
    reads[::7, -1] = ord("T")
    ctx.block_run(reads)
    ora_order = np.array(sorted(range(n), key=lambda i: reads[i].tobytes()), dtype=np.uint32)
    assert np.array_equal(ctx.get("sorted_ids", np.uint32), ora_order)


@pytest.mark.parametrize("n", [5000, 12_289])
def test_blocks_of_long_runs(ctx, n):
    rng = np.random.default_rng(n)
    reads = synth.ACGT[rng.integers(0, 4, size=(n, 80))]
    reads[: n // 2, :40] = reads[0, :40]
    ora = OracleBlock(reads)
    ctx.block_run(reads)
    bad = [nm for nm, dt in STAGE_RESULTS.items() if not np.array_equal(ctx.get(nm, dt), ora.get(nm, dt))]
    assert not bad, bad


@pytest.mark.parametrize("n", [148 * 4096 - 1, 148 * 4096])
def test_few_or_many_items(ctx, n):
    """On both sides of the size from which the sort's passes take full tiles."""
    L = 40
    rng = np.random.default_rng(n)
    reads = np.ascontiguousarray(synth.ACGT[rng.integers(0, 4, size=(n, L))])
    reads[::5] = reads[0]
    ctx.block_run(reads)
    assert np.array_equal(ctx.get("sorted_ids", np.uint32), np.argsort(reads.view(f"S{L}").ravel(), kind="stable"))
