"""The overlap's and the full match's counters count what their names say:
links made and members of contested runs against a plain restatement of the
overlap loop and the oracle's log, in one stage and in several, with a listing
that had to be repeated, and the same number of meetings in every form of the
full match that lists them.  Whole numbers: equal."""
import numpy as np
import pytest

from bench import block_stats
from curc_b200 import synth
from tests.cases import CASES
from tests.oracle_lib import OracleBlock

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from curc_b200 import Context
    with Context(0) as c:
        yield c


def overlap_counts(seqs):
    """Links and contested suffixes (compress.cu:1427-1532 on strings)."""
    n, L = seqs.shape
    reads = [r.tobytes() for r in seqs]
    ids = sorted(range(n), key=lambda i: reads[i])
    pre = [b for a, b in zip([None] + ids, ids) if a is None or reads[a] != reads[b]]
    suf = [a for a, b in zip(ids, ids[1:] + [None]) if b is None or reads[a] != reads[b]]
    links = contested = 0
    taken = set()
    for off in range(1, L * 65 // 100):
        runs = {}
        for p in pre:
            runs.setdefault(reads[p][: L - off], []).append(p)
        met, left = {}, []
        free = {k for k, run in runs.items() if any(p not in taken for p in run)}
        for s in suf:
            run = runs.get(reads[s][off:], [])
            if reads[s][off:] in free:
                met[reads[s][off:]] = met.get(reads[s][off:], 0) + 1
            p = next((p for p in run if p not in taken and p != s), None)
            if p is None:
                left.append(s)
            else:
                taken.add(p)
                links += 1
        contested += sum(c for c in met.values() if c > 1)
        suf = left
    return links, contested


def deep(n, L, genome, seed, copies=1):
    rng = np.random.default_rng([n, L, genome, seed])
    g = synth.ACGT[rng.integers(0, 4, size=genome // copies)]
    g = np.concatenate([np.tile(g, copies), g[:L]])
    at = rng.integers(0, len(g) - L + 1, size=n)
    return np.ascontiguousarray(np.lib.stride_tricks.sliding_window_view(g, L)[at])


@pytest.mark.parametrize("n,L,genome,copies", [(1, 50, 200, 1), (1500, 60, 3000, 1), (1500, 60, 2000, 4),
                                               (3000, 100, 4000, 12), (2500, 40, 1200, 60), (4000, 90, 3000, 2)])
def test_links_and_contested(ctx, n, L, genome, copies):
    seqs = deep(n, L, genome, 1, copies)
    # some reads end differently, so that runs hold several suffixes
    seqs[::3, : L // 4] = synth.ACGT[np.random.default_rng(n).integers(0, 4, size=(len(seqs[::3]), L // 4))]
    seqs[1::3, -(L // 4):] = synth.ACGT[np.random.default_rng(L).integers(0, 4, size=(len(seqs[1::3]), L // 4))]
    ctx.block_run(seqs)
    st = block_stats(ctx)
    assert (st["overlap_links"], st["contested"]) == overlap_counts(seqs)


@pytest.mark.parametrize("case", ["dups", "se250_8k", "se100_deep"])
def test_contested_is_the_oracles(ctx, case):
    seqs, po, pe = CASES[case]()
    ctx.block_run(seqs, po, pe)
    # (the oracle also logs runs that had no free prefix: none of their members took one)
    rows = OracleBlock(seqs, po, pe).contests()
    run = rows[:, 0].astype(np.uint64) << np.uint64(32) | rows[:, 1]
    took = np.unique(run[rows[:, 3] != 0xFFFFFFFF])
    assert block_stats(ctx)["contested"] == int(np.isin(run, took).sum())


def test_links_in_several_stages(ctx):
    seqs = deep(620_000, 26, 6_000_000, 2)
    ctx.block_run(seqs)
    st = block_stats(ctx)
    assert st["overlap_suffixes"] > 1 << 19
    assert st["overlap_links"] == overlap_counts(seqs)[0]


def test_counters_after_a_repeated_listing(ctx):
    """More meetings than a listing of all offsets has room for (4 Mi): the
    offsets are listed in parts, and what the first listing counted is not."""
    seqs = deep(250_000, 100, 260_000, 3)
    ctx.block_run(seqs)
    st = block_stats(ctx)
    density = st["overlap_suffixes"] / 260_000  # of the places, reads of a random sequence
    assert 63 * density * st["overlap_suffixes"] > 1.1 * (4 << 20)
    assert st["overlap_hits"] <= st["overlap_searched"] < 1.2 * st["overlap_hits"]
    assert st["overlap_compares"] < 4 * st["overlap_searched"]


def test_full_match_meetings_in_both_forms(ctx):
    """Chains of four reads, of which the chain filter keeps the two in the
    middle, and what is left of one ends as another starts: a pair of chains has
    one meeting of 20 to 30 bases, below and above the one-block limit."""
    per = {}
    for pairs in (200, 1500):
        rng = np.random.default_rng(pairs)
        x, y = (synth.ACGT[rng.integers(0, 4, size=(pairs, 130))] for _ in range(2))
        for i in range(pairs):
            k = 20 + i % 11
            y[i, 10:10 + k] = x[i, 120 - k:120]
        ctx.block_run(np.concatenate([g[:, at:at + 100] for g in (x, y) for at in (0, 10, 20, 30)]))
        per[pairs] = block_stats(ctx)["fm_meetings"]
    # and below some 8 bases, where most strings are met, a few offsets' worth
    assert 200 <= per[200] < 200 + 8 * 400 and 1500 <= per[1500] < 1500 + 8 * 3000, per
