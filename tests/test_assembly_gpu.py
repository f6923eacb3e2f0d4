"""Assembly around the one-block limit (8192 members) with chains and cycles,
and repeat removal around its limits (2048 hits walked by one thread, spans at
every byte alignment of the output).  Whole numbers: equal to the oracle."""
import numpy as np
import pytest

from curc_b200 import synth
from tests.oracle_lib import OracleBlock, STAGE_RESULTS, stream_dtype, stream_names

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from curc_b200 import Context
    with Context(0) as c:
        yield c


def same_as_oracle(ctx, seqs):
    ora = OracleBlock(seqs)
    ctx.block_run(seqs)
    names = list(STAGE_RESULTS.items()) + [(s, stream_dtype(s)) for s in stream_names(seqs.shape[1])]
    bad = [nm for nm, dt in names if not np.array_equal(ctx.get(nm, dt), ora.get(nm, dt))]
    assert not bad, bad


@pytest.mark.parametrize("n", [1, 2, 1023, 1025, 8191, 8192, 8193])
@pytest.mark.parametrize("step", [7, 20])
def test_circles_and_chains(ctx, n, step):
    """Reads along circles of different sizes (cycles) and lines (chains)."""
    rng = np.random.default_rng([n, step])
    L, parts, made = 60, [], 0
    while made < n:
        k = min(n - made, int(rng.integers(1, 700)))
        g = synth.ACGT[rng.integers(0, 4, size=k * step + (L if made % 2 else 0))]
        idx = np.arange(k)[:, None] * step + np.arange(L)
        parts.append(g[idx % len(g)])
        made += k
    seqs = np.concatenate(parts)
    same_as_oracle(ctx, seqs[rng.permutation(n)])


@pytest.mark.parametrize("copies,unit", [(3, 5000), (700, 400), (2500, 120)])
def test_reverse_complement_repeats(ctx, copies, unit):
    rng = np.random.default_rng([copies, unit])
    seg = synth.ACGT[rng.integers(0, 4, size=unit)]
    parts = []
    for i in range(copies):  # both strands of one segment between random spacers
        parts += [seg if i % 2 else synth.revcomp(seg), synth.ACGT[rng.integers(0, 4, size=int(rng.integers(60, 110)))]]
    g = np.concatenate(parts)
    starts = np.arange(0, len(g) - 100, 23)
    seqs = np.lib.stride_tricks.sliding_window_view(g, 100)[starts].copy()
    same_as_oracle(ctx, seqs[rng.permutation(len(seqs))])
