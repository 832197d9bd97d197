"""The reports of a step against what the step did."""
import ctypes as C

import numpy as np
import pytest

from sandbox_reactions_b200 import scenes
from sandbox_reactions_b200.abi import sr_dt_report
from sandbox_reactions_b200.engine import Batch, Step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["mg", "jacobi"])
def test_the_heat_report_names_the_step_it_covers(precond):
    cfg, P, kappa = scenes.full_step(64)
    seen = []
    with Step(cfg) as s:
        s.set_heat_precond(precond)
        s.upload(P)
        s.upload_opacity(kappa)
        for _ in range(3):
            s.run(1)
            seen.append(s.read_heat().dt)
            assert seen[-1] == s.read_dt().dt > 0.0
        s.run(2)
        assert s.read_heat().dt == s.read_dt().dt
    assert len(set(seen)) == 3  # the CFL rule gave each step a Δt of its own


def test_the_heat_reports_of_a_batch_name_their_steps():
    worlds = [scenes.full_step(n, scene=k) for k, n in enumerate((64, 96))]
    with Batch([w[0] for w in worlds]) as b:
        for i, (_, P, kappa) in enumerate(worlds):
            b.upload(i, P, kappa)
        for _ in range(2):
            b.run(1)
            for i in range(2):
                dt = sr_dt_report()
                assert b.lib.sr_read_dt(b.lib.sr_batch_ctx(b._h, i), C.byref(dt)) == 0
                assert b.read_heat(i).dt == dt.dt > 0.0


def test_a_step_without_a_solve_reports_no_dt():
    cfg, P, kappa = scenes.full_step(64)
    with Step(cfg.replace(pin_temperature=True)) as s:
        s.upload(P)
        s.upload_opacity(kappa)
        s.run(1)
        assert s.read_heat().dt == 0.0 < s.read_dt().dt


def test_the_per_pass_times_of_a_gas_only_step():
    """Under the per-pass timing the floors and Δt are a pass of their own, and the state is the one-kernel step's."""
    cfg, P = scenes.sod(264)
    out = []
    for timing in (0, 2):
        with Step(cfg) as s:
            s.upload(P)
            s.set_timing(timing)
            s.run(20)
            cost = s.read_cost()
            out.append((s.readback(), s.read_dt()))
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
    assert cost.kernel_launches == 2 * 20 and cost.hydro_update_launches == 20
    assert 0.0 < cost.hydro_update_ms <= cost.hydro_ms and cost.dt_ms > 0.0


def test_the_gas_update_of_a_step_with_gravity_is_timed_whole():
    """P4 is the update's kernels and the half step's solve, which is P2's on another density: what the update leaves of
    P4 is P2's time, not P2's and the kick's (a third more at this size)."""
    cfg, P = scenes.disk(2048)
    with Step(cfg) as s:
        s.upload(P)
        s.set_timing(2)
        s.run(2)
        s.run(10)
        cost = s.read_cost()
    assert cost.hydro_ms - cost.hydro_update_ms <= 1.15 * cost.gravity_ms
