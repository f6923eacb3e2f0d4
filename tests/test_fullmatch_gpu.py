"""The full match's listed form at its edges: list lengths around the
one-block limit (1024), several stages, runs of more than a warp, reads that
meet themselves, short and long reads, with and without N, against the oracle;
and against the pass form on reads with other letters, which both run by
passes.  Everything is whole numbers: results must be equal."""
import numpy as np
import pytest

from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS, stream_dtype, stream_names

pytestmark = pytest.mark.gpu


def reads_of(kind, n, L, with_n):
    rng = np.random.default_rng([n, L, with_n, len(kind)])
    r = synth.ACGT[rng.integers(0, 4, size=(n, L))]
    if kind == "tails":  # many suffixes and prefixes of one string: runs of hundreds at many offsets
        k = L // 3
        r[: n // 2, -k:] = ord("A")
        r[n // 4: 3 * n // 4, :k] = ord("A")
    elif kind == "periodic":  # reads that meet themselves and each other at every period
        for i in range(0, n, 3):
            p = 1 + i % 7
            r[i] = np.resize(r[i, :p], L)
    elif kind == "overlapping":  # fragments of one sequence, most overlaps short
        g = synth.ACGT[rng.integers(0, 4, size=n * L // 2)]
        r = np.lib.stride_tricks.sliding_window_view(g, L)[rng.integers(0, len(g) - L + 1, size=n)].copy()
    if with_n:
        r[np.arange(n), rng.integers(0, L, size=n)] = ord("N")
    return r


def results(ctx, seqs, **knobs):
    default = ctx.tuning()
    ctx.set_tuning(**dict(default, **knobs))
    ctx.block_run(seqs)
    ctx.set_tuning(**default)
    return {nm: ctx.get(nm, dt) for nm, dt in
            list(STAGE_RESULTS.items()) + [(s, stream_dtype(s)) for s in stream_names(seqs.shape[1])]}


@pytest.fixture(scope="module")
def ctx():
    from curc_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("with_n", [0, 1])
@pytest.mark.parametrize("kind,n,L", [
    ("random", 2, 40), ("random", 1023, 64), ("random", 1024, 64), ("random", 1025, 64), ("random", 6000, 48),
    ("tails", 900, 60), ("tails", 3000, 75), ("periodic", 700, 50), ("periodic", 2500, 90),
    ("overlapping", 2000, 100), ("overlapping", 1500, 12), ("overlapping", 1500, 16), ("overlapping", 1500, 17),
    ("overlapping", 1300, 511)])
def test_listed_form_at_its_edges(ctx, kind, n, L, with_n):
    seqs = reads_of(kind, n, L, with_n)
    ora = OracleBlock(seqs)
    got = results(ctx, seqs)
    bad = [nm for nm, v in got.items() if not np.array_equal(v, ora.get(nm, v.dtype.type))]
    assert not bad, bad


@pytest.mark.parametrize("kind,n", [("tails", 300), ("random", 1600)])
def test_other_letters_take_the_pass_form(ctx, kind, n):
    seqs = reads_of(kind, n, 60, 1)
    # one letter beyond A, C, G and N: the passes merge runs per first letter,
    # with T, R, ... as one run, so reads that mix those are not sorted by them
    # and which of their equal ends meet is not defined
    seqs[seqs == ord("T")] = ord("G")
    seqs[::5, 7] = ord("R")
    a, b = results(ctx, seqs), results(ctx, seqs, fm_loop=0)
    bad = [nm for nm in a if not np.array_equal(a[nm], b[nm])]
    assert not bad, bad
