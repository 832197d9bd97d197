"""The gas step with gravity, and the gas-only step that carries the floors and Δt in its own kernel, at widths and
heights that end inside a tile, a warp's 128 columns or a thread's rows, with a vacuum block: one step against the
oracle from the same f32 start (rel L1 1e-5 per field, the per-step bar), and Δt_{n+1} against the oracle's rule on the
stepped state (FP32 speeds: 1e-5)."""
import numpy as np
import pytest

import oracle as O
from sandbox_reactions_b200.abi import Config
from sandbox_reactions_b200.engine import Step

pytestmark = pytest.mark.gpu


def state(w, h, gamma, seed):
    rng = np.random.default_rng(seed)
    sigma = 0.5 + rng.random((h, w))
    u, v = 0.3 * rng.standard_normal((2, h, w))
    P = np.zeros((4, h, w))
    P[0], P[1], P[2] = sigma, sigma * u, sigma * v
    P[3] = (1.0 + rng.random((h, w))) / (gamma - 1.0) + 0.5 * sigma * (u * u + v * v)
    P[:, : h // 3, w // 2:] = np.array([1e-9, 0.0, 0.0, 1e-9])[:, None, None]
    return P.astype(np.float32)


@pytest.mark.parametrize("gravity", [False, True])
@pytest.mark.parametrize("edge", ["bounce", "leave"])
@pytest.mark.parametrize("w,h", [(16, 16), (32, 24), (136, 40), (264, 16), (24, 136)])
def test_one_step_matches_the_oracle(w, h, edge, gravity):
    gamma = 5.0 / 3.0
    cfg = Config(width=w, height=h, edge=edge, gamma=gamma, gravity=gravity)
    P = state(w, h, gamma, 5 * w + h)
    with Step(cfg) as s:
        s.upload(P)
        s.run(1)
        gpu, rep = s.readback().astype(np.float64), s.read_dt()
        s.upload(P)
        s.run(1)
        assert np.array_equal(s.readback().astype(np.float64), gpu)
    D = P.astype(np.float64)
    g = None
    if gravity:
        _, gx, gy = O.grav_field(cfg, D[0])
        g = (gx, gy)
    assert abs(rep.dt - O.hydro_dt(cfg, D, g)) <= 1e-5 * rep.dt and rep.steps == 1 and rep.sim_time == rep.dt
    ref, _ = O.hydro_step(cfg, D, rep.dt, g)
    ref = O.floors(cfg, ref)
    for k in range(4):
        assert np.abs(gpu[k] - ref[k]).sum() <= 1e-5 * np.abs(ref[k]).sum(), k
    assert abs(rep.dt_next - O.hydro_dt(cfg, ref, g)) <= 1e-5 * rep.dt_next
