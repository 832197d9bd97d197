"""The reports of a step against what the step did."""
import ctypes as C

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
