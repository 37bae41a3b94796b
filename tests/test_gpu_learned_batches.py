"""The network's gradient at the batch sizes where its tiles and the reduction
over their partial sums can go wrong: one row, a row short of a tile and one
over, a second tile for one CTA alone (two CTAs an SM), a full round; and sums
that leave FP32's range."""
import numpy as np
import pytest

from imodel_gb300 import learned
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _problem(n, seed):
    rng = np.random.default_rng(seed)
    xb = learned.to_bf16_bits(rng.normal(size=(n, 24)).astype(np.float32))
    x = (xb.astype(np.uint32) << 16).view(np.float32)
    return xb, x, rng.normal(size=n).astype(np.float32)


@pytest.mark.parametrize("batch", [1, 127, 129, 304 * 128 + 1, 65536])
def test_gradient_at_the_edges_of_tiles(batch):
    """The bounds are those of the products in BF16 (8 bits) through three
    layers, 4e-3 in all and 8e-3 a parameter block, as for other batches; a
    single row has no averaging, so four times as much."""
    xb, x, t = _problem(batch, 3)
    p = mo.init_params(4)
    net = learned.Mlp(params=p)
    loss, g = net.grad(xb, t, batch=batch, seed=0)
    lo, gr = mo.loss_and_grad(p, x, t, None)
    scale = 4.0 if batch == 1 else 1.0
    assert abs(loss - lo) <= scale * 4e-3 * lo
    assert np.linalg.norm(g - gr) < scale * 4e-3 * np.linalg.norm(gr)
    # the same numbers from call to call
    loss2, g2 = net.grad(xb, t, batch=batch, seed=0)
    assert loss2 == loss and np.array_equal(g, g2)


def test_a_loss_beyond_fp32_is_infinite():
    xb, _, t = _problem(1000, 5)
    net = learned.Mlp(params=mo.init_params(4))
    loss, g = net.grad(xb, np.full_like(t, 3e19), batch=1000, seed=0)
    assert np.isposinf(loss) and np.all(np.isfinite(g))
