"""The autotuner runs each different setting twice, and none that is another's
alias: its launches are those of the runs that make sense."""
import pytest

from tests.cases import CASES

pytestmark = pytest.mark.gpu


def test_no_alias_is_timed():
    import torch
    from curc_b200 import Context, kernel_launches
    seqs, po, pe = CASES["se75_20k"]()
    n, L = seqs.shape
    d = torch.from_numpy(seqs.reshape(-1).copy()).cuda()

    def launches(f):
        k = kernel_launches()
        f()
        return kernel_launches() - k

    with Context(0) as ctx:
        default = ctx.tuning()
        ctx.keep_intermediates(False)
        run = lambda: ctx.block_run_device(d.data_ptr(), n, L, po, pe)
        run()
        listed = launches(run)
        ctx.set_tuning(**dict(default, fm_loop=0))
        passes = launches(run)
        ctx.set_tuning(**default)
        total = launches(lambda: ctx.autotune(d.data_ptr(), n, L, po, pe))
    # table_factor 4, bitmap_bits 3, check_every 3, map_threads 3, fm_loop 2
    assert total < 2 * (4 + 3 + 3 + 3) * listed + 2 * (passes + listed) + listed
