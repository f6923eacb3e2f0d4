"""The training kernels at the edges of their tiles (32 rows a block, stages of
32 rows, eight stages in flight): loss and gradients against the float64
restatement, at the tolerance of the gradient test."""
import numpy as np
import pytest

from tests.test_learned_gpu import HID, IN, NB, _numpy_loss_grads, _out

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 2, 31, 32, 33, 64, 255, 257, 1000])
def test_gradients_at_tile_edges(B):
    from curc_b200 import Learner, learn_param_count
    rng = np.random.default_rng(B)
    p = (rng.standard_normal(learn_param_count()) * 0.1).astype(np.float32)
    x = (rng.random((B, IN)) < 0.15).astype(np.float32)
    tb = rng.integers(-1, NB, B).astype(np.int8)
    tg = rng.integers(-1, _out() - NB, B).astype(np.int8)
    with Learner(0) as lrn:
        loss, g = lrn.grad(p, x, tb, tg)
    ref_loss, ref_g = _numpy_loss_grads(p, x, tb, tg)
    assert g.shape == (HID * IN + HID + HID * HID + HID + _out() * (HID + 1),)
    assert abs(loss - ref_loss) <= 1e-4 * max(1.0, abs(ref_loss))
    np.testing.assert_allclose(g, ref_g, rtol=1e-3, atol=1e-5)
