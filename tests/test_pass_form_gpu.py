"""The full match's pass form (fm_loop 0) on random blocks against the oracle
(tests/test_sweep_gpu.py draws the blocks and checks the listed form).  Whole
numbers: equal."""
import random

import numpy as np
import pytest

from tests.oracle_lib import OracleBlock, STAGE_RESULTS, stream_dtype, stream_names
from tests.test_sweep_gpu import draw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [7, 8])
def test_random_blocks(seed):
    from curc_b200 import Context
    rnd = random.Random(seed)
    with Context(0) as ctx:
        ctx.set_tuning(**dict(ctx.tuning(), fm_loop=0))
        for _ in range(12):
            w, params = draw(rnd, 1500)
            seqs, pe = w.sequences(), w.mate2 is not None
            ora = OracleBlock(seqs, w.preserve_order, pe)
            ctx.block_run(seqs, w.preserve_order, pe)
            bad = [nm for nm, dt in list(STAGE_RESULTS.items()) + [(s, stream_dtype(s)) for s in stream_names(seqs.shape[1])]
                   if not np.array_equal(ctx.get(nm, dt), ora.get(nm, dt))]
            assert not bad, (params, bad)
