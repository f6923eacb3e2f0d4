"""Mapping at the edges of its kernel: read lengths around a chunk of 32
probes and of 32-base words, many reads with N (which differs from every base
on both strands), repeats that put many
entries in one bucket and many equal counts in one chunk.  Whole numbers:
equal to the oracle."""
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


def block(L, kind):
    rng = np.random.default_rng([L, len(kind)])
    if kind == "repeats":  # a genome of 40 diverged copies of one segment: full buckets, ties
        seg = synth.ACGT[rng.integers(0, 4, size=max(3 * L, 300))]
        copies = []
        for _ in range(40):
            c = seg.copy()
            m = rng.random(len(c)) < 0.004
            c[m] = synth.ACGT[rng.integers(0, 4, size=int(m.sum()))]
            copies.append(c)
        g = np.concatenate(copies)
    else:
        g = synth.ACGT[rng.integers(0, 4, size=40 * L + 2000)]
    reads = synth.sample_single(rng, g, 3000, L, 0.01, 0.002 if kind == "many_n" else 0.0005)
    return reads


@pytest.mark.parametrize("L", [28, 29, 33, 64, 90, 91, 92, 96, 129, 155, 250, 300])
@pytest.mark.parametrize("kind", ["plain", "repeats", "many_n"])
def test_mapping(ctx, L, kind):
    seqs = block(L, kind)
    ora = OracleBlock(seqs)
    ctx.block_run(seqs)
    bad = [nm for nm in ("hq_seq", "map_mm", "map_strand", "map_pos")
           if not np.array_equal(ctx.get(nm, STAGE_RESULTS[nm]), ora.get(nm, STAGE_RESULTS[nm]))]
    assert not bad, bad
