"""A product's wait that runs out (lpg_test_stall_products withholds loads):
the evaluation reports a timeout, the kernel leaves with its loads and
products finished, and the plan evaluates as before afterwards."""

import numpy as np
import pytest

from laser_polio_gb300 import _lib
from laser_polio_gb300 import ops
from oracle import incidence as I


@pytest.mark.gpu
@pytest.mark.parametrize("stages", [0, 1, 2, 3, 5])
def test_gpu_a_product_without_its_loads_times_out(stages):
    T, G = 365, 774  # every CTA has more than five loads to issue
    inp = I.random_inputs(T, G, 1, seed=stages)
    g = np.random.default_rng(1).normal(size=(T, G))
    plan = ops.IncidencePlan(inp)
    try:
        want = plan.evaluate(inp, g, lam=True)
        plan.test_stall_products(stages, 4096)
        with pytest.raises(_lib.LpgError, match="wait ran out"):
            plan.evaluate(inp, g, lam=True)
        plan.test_stall_products(-1)
        got = plan.evaluate(inp, g, lam=True)
        assert np.array_equal(got["lam"], want["lam"])
        scale = np.max(np.abs(want["grad"]["network"]))
        assert np.max(np.abs(got["grad"]["network"] - want["grad"]["network"])) <= 1e-12 * scale
    finally:
        plan.close()


@pytest.mark.gpu
def test_gpu_a_short_limit_without_a_stall_is_enough():
    """A good wait takes far fewer polls than the limit."""
    inp = I.random_inputs(60, 774, 3, seed=5)
    plan = ops.IncidencePlan(inp)
    try:
        plan.test_stall_products(-1, 1 << 16)
        lam = plan.evaluate(inp, lam=True, grad=False)["lam"]
        plan.test_stall_products(-1)
        assert np.array_equal(plan.evaluate(inp, lam=True, grad=False)["lam"], lam)
        with pytest.raises(ValueError):
            plan.test_stall_products(-1, 1 << 25)
    finally:
        plan.close()
