"""Training batches where a tile, a 64-sample chunk or a slice of the weight
gradients (k_layer, k_weight_grads, k_reduce_params) is not full: gradients
per parameter block against the oracle, within the tolerance of the other
training tests (3e-2 of the block's norm: a few BF16 roundings differ by one
unit); a training step is the Adam step of those gradients."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))
import mlp_oracle as M  # noqa: E402
from test_gpu_surrogate import _data, _net  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 63, 65, 128, 129, 1025, 2113, 4096])
def test_gradients_at_the_edges_of_tiles_and_slices(gpu, n):
    s = _net()
    x, t = _data(n, seed=n)
    loss, g = s.gradients(x, t)
    p0 = s.params().astype(np.float64)
    lo, go = M.loss_and_grad(p0, x, t, s.norm)
    step_loss = s.train_step(x, t, lr=1e-3)
    p1 = s.params().astype(np.float64)
    s.close()
    assert abs(loss - lo) <= 1e-2 * lo
    assert step_loss == loss  # the same pass, bit for bit
    o = 0
    for name, shape in M.SHAPES:
        k = int(np.prod(shape))
        a, b = g[o:o + k], go[o:o + k]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b) + 1e-12, name
        o += k
    # first Adam step from rest: m / bc1 = g, v / bc2 = g^2 (FP32 evaluation: 1e-6 of a step of 1e-3, and p's rounding)
    g = g.astype(np.float64)
    np.testing.assert_allclose(p1, p0 - 1e-3 * g / (np.abs(g) + 1e-8), rtol=1e-6, atol=2e-8 + 1e-3 * 1e-4)


def test_a_step_whose_wait_ran_out_changes_nothing(gpu):
    """A kernel whose wait runs out leaves its result unwritten, so the sums over
    the slices of such a pass hold older values: the step reports it and touches
    neither parameters, moments nor the step count. (The status is set from the
    host; no wait is made to run out.)"""
    from mercurydpm_fork_b200.surrogate import SurrogateError, lib
    s, twin = _net(), _net()
    batches = [_data(n, seed=n) for n in (300, 1024, 128)]
    for net in (s, twin):
        net.train_step(*batches[0])
    before = s.params()
    assert lib().dem_mlp_selftest_expire(s._h) == 0
    with pytest.raises(SurrogateError, match="2: "):
        s.train_step(*batches[1])
    np.testing.assert_array_equal(s.params(), before)
    for b in batches[1:]:
        assert s.train_step(*b) == twin.train_step(*b)
        np.testing.assert_array_equal(s.params(), twin.params())
    s.close()
    twin.close()
