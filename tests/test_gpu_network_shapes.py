"""The network's kernels at batches and crops whose tiles are ragged at some level, and at one with more tiles than run
at once: the forward pass and every gradient against the f64 network with the same BF16 rounding of the convolutions'
operands.

The bound: the kernels accumulate in FP32, so an activation near a rounding boundary may round to the other BF16
neighbour. It then lies one spacing from the oracle's operand, twice the half spacing that a rounding moves an operand at
most, and every operand downstream may follow (the f64 network itself moves by 3.3e-3 at crop 88 when its biases move by
1e-6). So two such networks lie within twice the distance which the rounding itself puts between the network and the
unrounded one, for the output and for each layer's gradient; 1e-3, the suite's bound, where that is less."""
import numpy as np
import pytest

from oracle import unet
from sandbox_reactions_b200.engine import Learner

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("crop,n", [(16, 1), (40, 3), (88, 2), (136, 1), (360, 2)])
def test_the_network_at_ragged_tiles(crop, n):
    rng = np.random.default_rng(crop + n)
    theta = unet.init_params(3)
    theta = (theta + 0.02 * rng.normal(size=theta.shape)).astype(np.float32)
    feats = rng.normal(size=(n, 4, crop, crop))
    feats[:, 1:3] = rng.uniform(0.0, 0.25, size=(n, 2, crop, crop))
    feats[:, 3] = rng.uniform(size=(n, crop, crop))
    feats, target = feats.astype(np.float32), rng.normal(size=(n, crop, crop)).astype(np.float32)
    with Learner(crop=crop, capacity=4) as L:
        L.set_params(theta)
        loss, grad, out = L.loss_grad(feats, target)
        again = L.loss_grad(feats, target)
    assert loss == again[0] and np.array_equal(grad, again[1]) and np.array_equal(out, again[2])
    f64 = (theta.astype(np.float64), feats.astype(np.float64), target.astype(np.float64))
    e_loss, e_grad, e_out = unet.loss_and_grad(*f64, bf16=True)
    _, x_grad, x_out = unet.loss_and_grad(*f64, bf16=False)

    def bound(e, x):
        return max(1e-3, 2.0 * rel_l2(x, e))

    assert rel_l2(out, e_out) <= bound(e_out, x_out) and abs(loss - e_loss) <= 1e-3 * e_loss
    k = 0
    for ci, co, _, _ in unet.LAYERS:
        for size in (co * 9 * ci, co):
            at = slice(k, k + size)
            assert rel_l2(grad[at], e_grad[at]) <= bound(e_grad[at], x_grad[at]), (ci, co, size)
            k += size
