"""The network's kernels tile by tile, at a batch with more tiles than CTAs (a convolution's CTAs take 8 x 16 pixels at a
time, 2,070 tiles on at most 1,480 CTAs here; a weight gradient's 16 x 8, on 128) and ragged ones on both axes. The output
is compared on every tile by itself, and the gradients are taken with the whole error δ on one tile, so that a tile
skipped, repeated or misplaced is the whole of what is compared and not one part in 2,070.

The bounds are tests/test_gpu_network_shapes.py's: two networks whose operands round to BF16 lie within twice the distance
which that rounding puts between them and the unrounded network, and 1e-3 where that is less."""
import numpy as np
import pytest
import torch

from oracle import unet
from sandbox_reactions_b200.engine import Learner

pytestmark = pytest.mark.gpu

CROP, N = 360, 2


def rel_l2(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def by_tile(v, w, h):
    """The rms of each tile of w x h pixels of (N, CROP, CROP), ragged ones over the pixels they have."""
    sq = np.zeros((N, -(-CROP // h) * h, -(-CROP // w) * w))
    sq[:, :CROP, :CROP] = v ** 2
    one = np.zeros_like(sq)
    one[:, :CROP, :CROP] = 1.0
    total = [a.reshape(N, a.shape[1] // h, h, a.shape[2] // w, w).sum((2, 4)) for a in (sq, one)]
    return np.sqrt(total[0] / total[1])


def test_every_tile_counts_once():
    rng = np.random.default_rng(11)
    # weights, biases and features above 0: no ReLU lies near its corner, so rounding moves every value by its own size only
    theta = np.concatenate([np.concatenate([rng.uniform(0.5, 1.5, co * 9 * ci) / (9 * ci), np.full(co, 0.05)])
                            for ci, co, _, _ in unet.LAYERS]).astype(np.float32)
    feats = rng.uniform(0.5, 1.5, size=(N, 4, CROP, CROP))
    feats[:, 1:3] = rng.uniform(0.0, 0.25, size=(N, 2, CROP, CROP))
    feats = feats.astype(np.float32)
    f = torch.tensor(feats, dtype=torch.float64)
    nets = []
    for bf16 in (True, False):
        t = torch.tensor(theta.astype(np.float64), requires_grad=True)
        nets.append((t, unet.forward(t, f, bf16)[:, 0]))
    e_out, x_out = (y.detach().numpy() for _, y in nets)
    # an error of 4 x 4 pixels each: in the first tile, in the ragged corner, in tiles of a CTA's second turn in the middle
    # and in the ragged last column, and across the corner of four weight-gradient tiles
    spots = [(0, 2, 2), (1, 356, 356), (1, 200, 100), (1, 8, 352), (0, 336, 8)]
    with Learner(crop=CROP, capacity=1) as L:
        L.set_params(theta)
        _, _, out = L.loss_grad(feats, np.ones((N, CROP, CROP), np.float32))
        got = []
        for img, y, x in spots:
            target = out.copy()
            target[img, y:y + 4, x:x + 4] += np.float32(4.0)
            got.append((target, L.loss_grad(feats, target)[1]))
    rms = np.sqrt((e_out ** 2).mean())
    assert by_tile(out - e_out, 8, 16).max() <= max(1e-3 * rms, 2.0 * by_tile(x_out - e_out, 8, 16).max())
    for (img, y, x), (target, grad) in zip(spots, got):
        tg = torch.tensor(target, dtype=torch.float64)
        energy = (tg * unet.scaled_operator(f, tg)).sum((1, 2))
        delta = tg - torch.tensor(out, dtype=torch.float64)
        assert int((delta != 0).sum()) == 16
        gy = -2.0 * unet.scaled_operator(f, delta) / (N * (energy + 1e-3 * energy.mean()))[:, None, None]
        e_grad, x_grad = (torch.autograd.grad(o, t, gy, retain_graph=True)[0].numpy() for t, o in nets)
        k = 0
        for ci, co, _, _ in unet.LAYERS:
            for size in (co * 9 * ci, co):
                at = slice(k, k + size)
                bound = max(1e-3, 2.0 * rel_l2(x_grad[at], e_grad[at]))
                assert rel_l2(grad[at], e_grad[at]) <= bound < 0.05, ((img, y, x), ci, co, size, bound)
                k += size
