"""P2 at every transform length (32 to 8192 points, each a radix plan of its own) and at row and column counts that do
not fill a CTA's group, against the oracle's f64 convolution. φ is held to rel L1 1e-5 as in the suite's gravity tests;
g is a central difference of an FP32 φ, so an ulp of the largest |φ| (2⁻²³ of it) over the mean |g| bounds what rounding
alone can do to it."""
import numpy as np
import pytest

import oracle as O
from sandbox_reactions_b200.abi import Config
from sandbox_reactions_b200.engine import Step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(16, 16), (24, 40), (40, 136), (136, 72), (264, 24), (24, 264), (520, 48), (48, 1032),
                                 (1032, 40), (2056, 16), (16, 2056)])
def test_the_field_at_every_transform_length(w, h):
    rng = np.random.default_rng(w * 7 + h)
    P = np.zeros((4, h, w), np.float32)
    P[0] = rng.random((h, w)) + 0.05
    P[0, : h // 4] = 1e-9  # not a source
    P[3] = 1.0
    cfg = Config(width=w, height=h, gravity=True)
    with Step(cfg) as s:
        s.upload(P)
        phi, gx, gy = s.gravity_field()
    ophi, ogx, ogy = O.grav_field(cfg, P[0].astype(np.float64))
    assert np.abs(phi - ophi).sum() <= 1e-5 * np.abs(ophi).sum()
    ulp = 2.0 ** -23 * np.abs(ophi).max()
    for g, o in ((gx, ogx), (gy, ogy)):
        assert np.abs(g - o).mean() <= 1e-5 * np.abs(o).mean() + 2 * ulp
