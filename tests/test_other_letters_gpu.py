"""N reads with letters beyond A, C, G, N and T in the full match of the
unmapped N reads: the oracle's links, the same in every run and for every
tuning.  Whole numbers: equal."""
import numpy as np
import pytest

from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS, stream_dtype, stream_names

pytestmark = pytest.mark.gpu


def reads_of(n, L, letters, share, seed):
    """N reads that meet each other often: starts and ends from a few strings
    of their own, with `letters` strewn over them."""
    rng = np.random.default_rng([n, L, len(letters), seed])
    r = synth.ACGT[rng.integers(0, 4, size=(n, L))]
    k = L // 3
    ends = synth.ACGT[rng.integers(0, 4, size=(max(2, n // 40), k))]
    other = rng.random(ends.shape) < share
    ends[other] = np.frombuffer(letters, dtype=np.uint8)[rng.integers(0, len(letters), size=int(other.sum()))]
    r[:, :k] = ends[rng.integers(0, len(ends), size=n)]
    r[:, -k:] = ends[rng.integers(0, len(ends), size=n)]
    for i in range(n):  # ends of every length
        j = int(rng.integers(1, k))
        r[i, :k] = np.roll(r[i, :k], -j)
        r[i, k - j:k] = ord("C")
    mid = rng.integers(k, L - k, size=n)
    r[np.arange(n), mid] = ord("N")
    return r


def results(ctx, seqs, **knobs):
    default = ctx.tuning()
    ctx.set_tuning(**dict(default, **knobs))
    ctx.block_run(seqs)
    ctx.set_tuning(**default)
    return {nm: ctx.get(nm, dt) for nm, dt in
            list(STAGE_RESULTS.items()) + [(s, stream_dtype(s)) for s in stream_names(seqs.shape[1])]}


@pytest.mark.parametrize("letters", [b"R", b"RT", b"RYKMacgtn", b"*. -"], ids=["oneletter", "RT", "many", "signs"])
@pytest.mark.parametrize("n,L", [(2, 30), (400, 60), (1024, 40), (3000, 60), (2500, 90)])
@pytest.mark.parametrize("share", [0.03, 0.3])
def test_links_are_the_oracles(letters, n, L, share):
    from curc_b200 import Context
    seqs = reads_of(n, L, letters, share, 1)
    if letters == b"R":
        seqs[seqs == ord("T")] = ord("G")
    ora = OracleBlock(seqs)
    with Context(0) as ctx:
        for knobs in ({}, {}, {"fm_loop": 0}):
            got = results(ctx, seqs, **knobs)
            bad = [nm for nm, v in got.items() if not np.array_equal(v, ora.get(nm, v.dtype.type))]
            assert not bad, (knobs, bad)
