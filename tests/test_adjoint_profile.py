"""A plan's profile counts evaluations, whatever launches a phase is."""

import pytest

from laser_polio_gb300 import ops
from oracle import incidence as I


@pytest.mark.gpu
@pytest.mark.parametrize("G", [20, 300])
def test_gpu_profile_counts_evaluations(G):
    inp = I.random_inputs(12, G, 2, seed=1)
    plan = ops.IncidencePlan(inp, I.incidence(inp)[0])
    try:
        plan.set_profiling(True)
        for _ in range(3):
            plan.evaluate(inp)
        for _ in range(2):
            plan.evaluate(inp, lam=True, grad=False)
        counts = [n for _, n in plan.profile().values()]
        assert counts == [5, 5, 5, 3, 3, 3]
    finally:
        plan.close()
