"""The weight gradients' sums over a large batch. With every parameter 0 but layer 13's biases (1, so that the head reads
ones) and no couplings in the features, the output is 0 and every pixel's output gradient is the same number g: the
head's bias gradient and its weights' at the middle tap are N g over N pixels. A partial sums at most 2,048 pixels in
FP32, 16 threads 128 each and their sums in turn, and the partials are summed in FP64, so the relative error is at most
144 · 2⁻²⁴, and 4 · 2⁻²⁴ for g itself, whatever the batch. (One run of additions as long as the batch allows, 2,048
and more a thread here, is past it for this target: 2.6e-5.)"""
import numpy as np
import pytest

from oracle import unet
from sandbox_reactions_b200.engine import Learner

pytestmark = pytest.mark.gpu


def test_the_sums_error_does_not_grow_with_the_batch():
    crop, n, c = 512, 16, 0.619
    sizes = [(co * 9 * ci, co) for ci, co, _, _ in unet.LAYERS]
    at = np.cumsum([0] + [w + b for w, b in sizes])
    theta = np.zeros(at[-1], np.float32)
    theta[at[13] + sizes[13][0]:at[14]] = 1.0
    feats = np.zeros((n, 4, crop, crop), np.float32)
    target = np.full((n, crop, crop), c, np.float32)
    with Learner(crop=crop, capacity=1) as L:
        L.set_params(theta)
        _, grad, out = L.loss_grad(feats, target)
    assert not out.any()
    energy = crop * crop * float(np.float32(c)) ** 2
    want = n * crop * crop * (-2.0 * float(np.float32(c)) / (n * energy * 1.001))
    head = grad[at[14]:].astype(np.float64)
    middle, bias = head[:72].reshape(9, 8)[4], head[72]
    assert np.abs(np.append(middle, bias) / want - 1.0).max() <= 148 * 2.0 ** -24
