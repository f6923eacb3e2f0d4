"""Runs of reads that share their first 32 bases, up to the whole block: in
the oracle's order around the longest run a warp orders, and in a time that
does not grow with the run (one warp once flagged a run 32 rows a step, which
made the sort of a million such reads 14 times as long as one in runs of a
thousand)."""
import numpy as np
import pytest

from curc_b200 import synth

pytestmark = pytest.mark.gpu


def reads_of(n, L, heads, seed=1):
    rng = np.random.default_rng([n, L, heads, seed])
    r = synth.ACGT[rng.integers(0, 4, size=(n, L))]
    r[:, :32] = r[rng.integers(0, heads, size=n), :32]
    return np.ascontiguousarray(r)


@pytest.fixture(scope="module")
def ctx():
    from curc_b200 import Context
    with Context(0) as c:
        yield c


@pytest.mark.parametrize("run", [16, 17, 31, 32, 33, 34, 48, 49, 64, 65])
@pytest.mark.parametrize("at", ["first", "middle", "last"])
def test_a_run_anywhere_in_the_list(ctx, run, at):
    n, L = 5003, 50
    rng = np.random.default_rng(run)
    r = synth.ACGT[rng.integers(0, 4, size=(n, L))]
    r[:, 0] = ord("C")
    r[rng.permutation(n)[:run], :32] = {"first": ord("A"), "middle": ord("C"), "last": ord("T")}[at]
    ctx.block_run(r)
    assert np.array_equal(ctx.get("sorted_ids", np.uint32), np.argsort(r.view(f"S{L}").ravel(), kind="stable"))


def test_time_does_not_grow_with_the_run(ctx):
    import torch
    n, L = 1_000_000, 64
    ms = {}
    for heads in (1, 1000):
        r = reads_of(n, L, heads)
        d = torch.from_numpy(r.reshape(-1)).cuda()
        ms[heads] = []
        for _ in range(4):
            ctx.block_run_device(d.data_ptr(), n, L)
            ms[heads].append(ctx.stage_ms("sort_dedupe.radix"))
        assert np.array_equal(ctx.get("sorted_ids", np.uint32), np.argsort(r.view(f"S{L}").ravel(), kind="stable"))
    assert min(ms[1]) < 3 * min(ms[1000]), ms
