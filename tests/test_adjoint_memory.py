"""The device memory of an incidence plan, and the products of plans whose
digits are formed a part at a time (more than 2^22 elements of beta)."""

import numpy as np
import pytest

from laser_polio_gb300 import ops
from oracle import incidence as I


@pytest.mark.gpu
@pytest.mark.parametrize("T,G,S", [(60000, 129, 3), (2000, 1500, 2), (400, 300, 3)])
def test_gpu_a_plan_needs_no_more_than_its_arrays(T, G, S):
    """FP32 pairs of beta and dL/du, u and exp(-r) beside beta took 40 bytes
    an element, and 96 a pair of nodes; plans may take 200 MB beside that."""
    import torch

    n = T * G
    one = np.ones(1)
    inp = dict(srisk=np.ones((T, G)), beta=np.ones((T, G, S)), pop=np.ones((T, G)), doy=np.ones(T), year=np.full(T, 365.0),
               pops=np.ones(G), dist=np.broadcast_to(one, (G, G)))
    torch.cuda.synchronize()
    ops.IncidencePlan(I.random_inputs(4, 4, 1)).close()  # the library's own memory
    before = torch.cuda.mem_get_info()[0]
    plan = ops.IncidencePlan(inp)
    try:
        taken = before - torch.cuda.mem_get_info()[0]
    finally:
        plan.close()
    assert taken <= 40 * n * S + 40 * n + 96 * G * G + 200e6, taken
    if n * S > 1 << 24:
        assert taken <= 17 * n * S + 40 * n + 96 * G * G + 300e6, taken


@pytest.mark.gpu
@pytest.mark.parametrize("T,G,S", [(7100, 300, 2), (11000, 129, 3), (1450, 1500, 2)])
def test_gpu_products_in_parts(T, G, S):
    inp = I.random_inputs(T, G, S, seed=G)
    g = np.random.default_rng(T).uniform(0.5, 1.5, (T, G))
    g[:, ::2] = 0.0
    want_lam, want = I.incidence(inp, g)
    plan = ops.IncidencePlan(inp)
    try:
        lam = plan.evaluate(inp, lam=True, grad=False)["lam"]  # forward alone first
        for _ in range(2):
            got = plan.evaluate(inp, g, lam=True)
            assert np.array_equal(got["lam"], lam)
            assert np.max(np.abs(lam - want_lam)) <= 1e-12 * np.max(np.abs(want_lam))
            net, ref = got["grad"]["network"][::2], want["network"][::2]
            # a sum of T S terms in numpy's order is within T S 2^-53 of them
            assert np.all(np.abs(net - ref) <= (2.0**-38 + T * S * 2.0**-52) * np.abs(ref))
            assert np.max(np.abs(got["grad"]["r0s"] - want["r0s"])) <= 1e-12 * np.max(np.abs(want["r0s"]))
    finally:
        plan.close()
