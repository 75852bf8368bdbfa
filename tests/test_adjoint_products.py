"""The expected-incidence products on the tensor cores (csrc/lpg_ozaki.cuh):
sizes about their tiles (128 rows, 64 columns, depth 32, 512 per drain) and
about the line to the double-float products, against the numpy oracle.

Tolerance: eight digits of seven bits leave 2^-56 of an element against its
row's or column's largest, so a sum over K <= 1200 terms is within K 2^-55 =
3.4e-14 of the largest product; 1e-12 of an output's largest magnitude leaves
a factor of 30 for the passes around the products."""

import numpy as np
import pytest

from laser_polio_gb300 import ops
from oracle import incidence as I

TOL = 1e-12


def _close(got, want, what):
    scale = float(np.max(np.abs(want)))
    err = float(np.max(np.abs(np.asarray(got) - np.asarray(want))))
    assert err <= TOL * scale, (what, err, scale)


@pytest.mark.gpu
@pytest.mark.parametrize(
    "T,G,S,max_frac",
    [(244, 128, 1, 0.2), (245, 128, 1, 0.2), (16, 129, 1, 0.2), (43, 161, 3, 1e-5), (128, 192, 2, 0.2), (3, 33, 2, 0.2),
     (1, 256, 1, 1e-6), (2, 257, 1, 0.2),
     (129, 193, 1, 1e-6), (171, 255, 3, 0.2), (130, 257, 4, 0.2), (20, 545, 1, 0.2), (257, 300, 4, 0.2),
     (37, 1200, 2, 1e-5)],
)
def test_gpu_products_match_the_oracle(T, G, S, max_frac):
    inp = I.random_inputs(T, G, S, seed=T + G)
    inp["max_frac"] = max_frac
    g = np.random.default_rng(T).normal(size=(T, G))
    want_lam, want = I.incidence(inp, g)
    plan = ops.IncidencePlan(inp)
    try:
        for _ in range(2):  # the second evaluation reuses the plan's buffers
            got = plan.evaluate(inp, g, lam=True)
            _close(got["lam"], want_lam, "lam")
            _close(got["grad"]["r0s"], want["r0s"], "r0s")
            _close(got["grad"]["network"], want["network"], "network")
    finally:
        plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("G", [40, 600])
def test_gpu_a_nan_stays_in_its_own_tick(G):
    """A NaN infectivity reaches every node of its tick and strain and no
    other tick, in the FP64 sums and the sliced products alike."""
    inp = I.random_inputs(20, G, 2, seed=1)
    inp["beta"][7, 3, 1] = np.nan
    lam, _ = ops.expected_incidence(inp)
    assert np.all(np.isnan(lam[7])) and np.all(np.isfinite(np.delete(lam, 7, axis=0)))


@pytest.mark.gpu
@pytest.mark.parametrize("k,a,b,c", [(0.5, 0.0, 0.0, 0.0), (0.5, 1.0, 0.0, 2.0), (-0.3, 1.0, 1.0, 2.0),
                                     (0.5, 0.7, 1.3, -0.4), (1e-3, 55.0, 1.0, 2.0)])
def test_gpu_flows_equal_the_oracle_at_every_exponent(k, a, b, c):
    """Flows formed in integers and, beyond the fixed-point range (a = 55),
    in FP64; nodes without people and nodes at one place included."""
    inp = I.random_inputs(16, 30, 1, seed=2)
    inp["pops"][4] = 0.0
    inp["dist"][1, 2] = inp["dist"][2, 1] = 0.0
    inp.update(k=k, a=a, b=b, c=c, max_frac=1e-4)
    want = I.incidence(inp)[0]
    got = ops.expected_incidence(inp)[0]
    _close(got, want, "lam")


@pytest.mark.gpu
@pytest.mark.parametrize("G", [30, 200])
def test_gpu_distances_at_the_edges_of_the_logarithm(G):
    """log2 of the distances in integers (normal ones) and in FP64: subnormal,
    next to one, powers of two and their neighbours, infinite; the diagonal,
    which is never read, may hold anything, and no other entry may be
    negative or NaN."""
    inp = I.random_inputs(12, G, 1, seed=4)
    edges = [1e-310, 2.0**-1022, 0.5, 1 - 2.0**-53, 1.0, 1 + 2.0**-52, 2 - 2.0**-52, 2.0, 1e300, np.inf]
    for j, d in enumerate(edges):
        inp["dist"][0, j + 1] = inp["dist"][j + 1, 0] = d
    inp.update(k=0.5, a=0.7, b=1.1, c=0.3, max_frac=1e-3)
    _close(ops.expected_incidence(inp)[0], I.incidence(inp)[0], "lam")
    lam = ops.expected_incidence(inp)[0]
    odd = dict(inp, dist=inp["dist"].copy())
    np.fill_diagonal(odd["dist"], [np.nan, -1.0] * (G // 2))
    assert np.array_equal(ops.expected_incidence(odd)[0], lam)
    for bad in (-1.0, np.nan):
        odd = dict(inp, dist=inp["dist"].copy())
        odd["dist"][3, G - 1] = bad
        with pytest.raises(Exception):
            ops.expected_incidence(odd)
