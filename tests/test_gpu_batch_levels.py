"""A batch's worlds against the same worlds alone, with several multigrid levels above the coarse tail: alone, a round's
kernels start before the one ahead has ended, in a batch they do not, and the state is the same bit for bit. One step
before and two after a readback, with MG and with Jacobi (whose rounds have no multigrid)."""
import numpy as np
import pytest

from sandbox_reactions_b200 import scenes
from sandbox_reactions_b200.engine import Batch, Step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["mg", "jacobi"])
def test_a_batch_of_worlds_of_many_levels_matches_them_alone(precond):
    worlds = [scenes.full_step(n, scene=k) for k, n in enumerate((512, 264, 328) if precond == "mg" else (136, 64))]
    worlds = [(cfg.replace(precond=precond), P, kappa) for cfg, P, kappa in worlds]
    with Batch([w[0] for w in worlds]) as b:
        for i, (_, P, kappa) in enumerate(worlds):
            b.upload(i, P, kappa)
        first = (b.run(1), [b.readback(i) for i in range(len(worlds))])[1]
        b.run(2)
        last = [b.readback(i) for i in range(len(worlds))]
        rounds = [b.read_heat(i).rounds for i in range(len(worlds))]
    for i, (cfg, P, kappa) in enumerate(worlds):
        with Step(cfg) as s:
            s.upload(P)
            s.upload_opacity(kappa)
            s.run(1)
            assert np.array_equal(first[i], s.readback()), i
            s.run(2)
            assert np.array_equal(last[i], s.readback()), i
            assert rounds[i] == s.read_heat().rounds > 0
