"""Every element of the expected incidence and of dL/dN on its own, where
elements of one row or column lie many decades apart: waves that do not
overlap, one infected node, one large node above a tiny background, distances
over three and a half decades.  Against the numpy oracle, elementwise; upstream
gradients are positive and vanish at the nodes whose rows are compared, so
that neither the sums nor the diagonal's subtraction cancel.

Tolerance: FP32 pairs carry each term to 3 2^-48 and a sum of K <= 900 terms
to K 2^-48 more, 2^-38 of the element; lam = srisk sum(1 - exp(-r)) adds the
cancellation of 1 - exp, 2^-51 of srisk a strain."""

import numpy as np
import pytest

from laser_polio_gb300 import ops
from oracle import incidence as I

TOL = 2.0**-38


def _elements(got, want, floor, what):
    err = np.abs(got - want)
    bad = err > TOL * np.abs(want) + floor
    rel = np.max(np.where(want != 0, err / np.where(want != 0, np.abs(want), 1.0), 0.0))
    assert not bad.any(), (what, int(bad.sum()), float(rel))


def _spread(T, G, S, c, seed):
    """Nodes along a line at log-uniform places, 1 to 3000 km."""
    inp = I.random_inputs(T, G, S, seed=seed)
    x = 10.0 ** np.random.default_rng(seed).uniform(0.0, 3.5, G)
    dist = np.abs(x[:, None] - x[None, :])
    dist[dist == 0] = 1.0
    np.fill_diagonal(dist, 0.0)
    inp.update(dist=dist, c=c, max_frac=0.2)
    return inp


def _scale_to_see(inp):
    """R so that the smallest rate is about 1e-3: lam shows every u."""
    N = I.network(inp["pops"], inp["dist"], inp["k"], inp["a"], inp["b"], inp["c"], inp["max_frac"])[0]
    _, mid = I.forward(inp["srisk"], inp["beta"], inp["pop"], inp["doy"], inp["year"], inp["r0s"], 1.0, inp["amp"],
                       inp["peak"], N)
    r = mid["u"] * mid["q"][:, :, None]
    inp["R"] = 1e-3 / float(r[r > 0].min())


def _lam(inp):
    _scale_to_see(inp)
    want = I.incidence(inp)[0]
    got = ops.expected_incidence(inp)[0]
    _elements(got, want, inp["srisk"] * inp["beta"].shape[2] * 2.0**-51, "lam")


@pytest.mark.gpu
@pytest.mark.parametrize("c", [2.0, 4.0])
@pytest.mark.parametrize("T,G,S", [(9, 160, 1), (20, 300, 2), (33, 333, 3)])
def test_gpu_one_infected_node(T, G, S, c):
    inp = _spread(T, G, S, c, seed=G)
    only = np.zeros_like(inp["beta"])
    only[:, G // 3, :] = 1.0 + inp["beta"][:, G // 3, :]
    inp["beta"] = only
    _lam(inp)


@pytest.mark.gpu
@pytest.mark.parametrize("c", [2.0, 4.0])
@pytest.mark.parametrize("T,G,S", [(9, 160, 1), (40, 774, 1)])
def test_gpu_one_large_node_above_a_background(T, G, S, c):
    inp = _spread(T, G, S, c, seed=G + 1)
    inp["beta"] = 1e-6 * (0.1 + inp["beta"])
    inp["beta"][:, 5, :] = 3e5
    _lam(inp)


@pytest.mark.gpu
@pytest.mark.parametrize("few", [False, True])
@pytest.mark.parametrize("T,G,S", [(200, 160, 2), (365, 300, 1), (301, 257, 3)])
def test_gpu_waves_that_do_not_overlap(T, G, S, few):
    """dL/dN of node pairs whose waves are up to T days apart.  few: only
    some nodes' waves come late, so that a tile has a handful of such pairs."""
    inp = I.random_inputs(T, G, S, seed=T)
    rng = np.random.default_rng(G)
    peak = rng.uniform(0.0, T, G)
    if few:
        peak = np.where(rng.uniform(size=G) < 0.02, T - 1.0, 0.1 * peak)
    t = np.arange(T)[:, None]
    wave = np.exp(-0.5 * ((t - peak[None, :]) / 22.0) ** 2)
    inp["beta"] = wave[:, :, None] * rng.gamma(2.0, 20.0, (T, G, S))
    g = wave * rng.uniform(0.5, 1.5, (T, G))
    g[:, ::2] = 0.0
    want = I.incidence(inp, g)[1]["network"]
    got = ops.expected_incidence(inp, g)[1]["network"]
    assert np.ptp(np.log10(want[::2, 1::2])) > 5.0
    _elements(got[::2], want[::2], 0.0, "network")


@pytest.mark.gpu
def test_gpu_an_element_of_cancelling_terms_and_an_empty_one():
    """A sum whose terms cancel is left as it is, a row or column without
    any term is exactly zero."""
    T, G = 64, 192
    inp = I.random_inputs(T, G, 2, seed=9)
    inp["beta"][:, 7, :] = 0.0
    g = np.random.default_rng(3).normal(size=(T, G))
    g[:, 11] = 0.0
    want = I.incidence(inp, g)[1]["network"]
    got = ops.expected_incidence(inp, g)[1]["network"]
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
    assert np.all(got[7] == 0.0)
