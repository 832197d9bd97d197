"""The multigrid's coarse tail and level smoothers over the level shapes where their code paths change: a world that is
its own tail (at most 64 cells a side), one row or column past it, odd-width levels, levels wider than tall and taller
than wide, and a mixed batch of worlds with tails of different sizes. The V-cycle is judged by what it is for: MG-PCG
reaches an FP64 residual of 1e-8, and the solution is the oracle's (its f64 Jacobi-PCG to 1e-12) within 1e-6 of the
largest value, the residual bar times the system's conditioning (the bar of the suite's first-system tests)."""
import numpy as np
import pytest

import oracle as O
from sandbox_reactions_b200 import scenes
from sandbox_reactions_b200.abi import Config
from sandbox_reactions_b200.engine import Batch, Step

pytestmark = pytest.mark.gpu


def world(w, h, seed):
    rng = np.random.default_rng(seed)
    kappa = (10.0 ** rng.uniform(-1.5, 1.5, (h, w))).astype(np.float32)
    T = 30.0 + 300.0 * rng.random((h, w))
    P = np.zeros((4, h, w), np.float32)
    P[0] = 1.0
    P[0, : h // 8, : w // 3] = 1e-9  # vacuum in a corner: masked cells in every level
    P[3] = (P[0] * T / (5.0 / 3.0 - 1.0)).astype(np.float32)
    cfg = Config(width=w, height=h, hydro=False, heat=True, opacity_plane=True, gamma=5.0 / 3.0)
    return cfg, P, kappa


@pytest.mark.parametrize("sweeps", [1, 4])
@pytest.mark.parametrize("w,h", [(16, 16), (64, 64), (72, 64), (64, 72), (104, 88), (264, 56), (56, 264), (328, 152),
                                 (1048, 16), (16, 1048)])
def test_the_v_cycle_solves_over_the_level_shapes(w, h, sweeps):
    cfg, P, kappa = world(w, h, 31 * w + h)
    dt = 1e-4
    with Step(cfg.replace(mg_pre=sweeps, mg_post=sweeps)) as s:
        s.upload(P)
        s.upload_opacity(kappa)
        _, rounds, rel, x = s.heat_first_solve(dt, "mg", want_x=True)
        _, plain, _, _ = s.heat_first_solve(dt, "jacobi")
    assert rel <= 1e-8 and 0 < rounds < plain, (rounds, plain)
    diag, rhs, kx, ky, gas = O.heat_system(cfg, P.astype(np.float64), dt, kappa.astype(np.float64))
    ref, _ = O.heat_pcg(diag, rhs, kx, ky, gas, rel=1e-12, max_rounds=200000)
    assert np.abs(x - ref).max() <= 1e-6 * np.abs(ref).max()


@pytest.mark.parametrize("sweeps", [1, 4])
@pytest.mark.parametrize("w,h", [(1048, 904), (2056, 1800)])
def test_levels_of_more_regions_than_fit_the_gpu_at_once(w, h, sweeps):
    """Level 0 (and, in the larger world, the weighted level 1) has more smoother regions than CTAs, so a CTA walks over
    several, and the SpMV's threads take several rows. Against the Jacobi-preconditioned solve, which has no smoother:
    each solution is within 1e-6 of the true one (above), so within 2e-6 of the other."""
    cfg, P, kappa = world(w, h, 31 * w + h)
    with Step(cfg.replace(mg_pre=sweeps, mg_post=sweeps)) as s:
        s.upload(P)
        s.upload_opacity(kappa)
        _, rounds, rel, x = s.heat_first_solve(1e-4, "mg", want_x=True)
        _, plain, plain_rel, ref = s.heat_first_solve(1e-4, "jacobi", want_x=True)
    assert rel <= 1e-8 and plain_rel <= 1e-8 and 0 < rounds < plain, (rounds, plain)
    assert np.abs(x - ref).max() <= 2e-6 * np.abs(ref).max()


def test_worlds_made_later_leave_the_larger_tails_of_earlier_ones_alone():
    specs = [(128, 128), (80, 40), (16, 24)]
    worlds = [world(w, h, 7 + w) for w, h in specs]
    with Batch([c.replace(dt_fixed=1e-4) for c, _, _ in worlds]) as b:
        for k, (_, P, kappa) in enumerate(worlds):
            b.upload(k, P, kappa)
        b.run(2)
        for k in range(len(worlds)):
            r = b.read_heat(k)
            assert r.converged and r.rel_residual <= 1e-8
            assert np.isfinite(b.readback(k)).all()
