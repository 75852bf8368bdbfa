"""The initialisation's FP32 forms of the timers and the heterogeneity
(csrc/lpg_init_fast.cuh) give the FP64 definitions' bits: every kind that has
such a form, the ranges next to the ones that do not, and sizes about the
kernels' tiles, against the oracle's restatement of lpg_init.h."""

import numpy as np
import pytest

from laser_polio_gb300 import _abi
from laser_polio_gb300 import init as dinit
from laser_polio_gb300.core import LaserFrame

GAMMA, LOGNORMAL, POISSON, CONSTANT, EXPONENTIAL = 2, 3, 5, 0, 1
TIMERS = [
    ((POISSON, 3.0, 0.0), (GAMMA, 4.51, 5.32), (LOGNORMAL, 12.5, 3.5)),
    ((GAMMA, 1.0, 3.0), (GAMMA, 64.0, 2.0), (LOGNORMAL, 200.0, 90.0)),
    ((CONSTANT, 3.0, 0.0), (CONSTANT, 200.0, 0.0), (POISSON, 9.99, 0.0)),
    ((GAMMA, 3.0, 90.0), (POISSON, 0.01, 0.0), (CONSTANT, 24.0, 0.0)),
    ((GAMMA, 0.9, 3.0), (GAMMA, 4.0, 6.0), (LOGNORMAL, 12.5, 0.0)),  # no FP32 form
    ((EXPONENTIAL, 3.0, 0.0), (GAMMA, 4.0, 6.0), (LOGNORMAL, 12.5, 3.5)),  # no FP32 form
]
HET = [(4.0, 0.8), (float(np.exp(0.64) - 1.0), -0.9), (0.0, 0.5), (1e-3, 1.0), (1e8, 0.3)]


def _both(capacity, parts, fields, pops=None):
    from oracle_backend import oracle_fill

    out = []
    for fill in (dinit.fill, oracle_fill):
        node_pop = np.array([capacity]) if pops is None else np.asarray(pops)
        count = int(node_pop.sum())
        people = LaserFrame(capacity=capacity, initial_count=count)
        spec = dinit.InitSpec(7, node_pop, count, capacity)
        for k, v in fields.items():
            setattr(spec, k, v)
        fill(people, spec, parts)
        out.append({n: np.asarray(getattr(people, n)) for n in dinit.part_columns(parts)})
    for name in out[0]:
        np.testing.assert_array_equal(out[0][name].view(np.uint8), out[1][name].view(np.uint8), err_msg=name)


@pytest.mark.gpu
@pytest.mark.parametrize("capacity", [1, 1023, 1025, 16385, 150_001])
@pytest.mark.parametrize("exp,inf,par", TIMERS)
def test_gpu_timers_equal_the_fp64_definition(exp, inf, par, capacity):
    _both(capacity, _abi.INIT_TIMERS, {"dur_exp": exp, "dur_inf": inf, "t_to_paralysis": par})


@pytest.mark.gpu
@pytest.mark.parametrize("capacity", [1, 1023, 1025, 16385, 150_001])
@pytest.mark.parametrize("var,corr", HET)
def test_gpu_heterogeneity_equals_the_fp64_definition(var, corr, capacity):
    _both(capacity, _abi.INIT_HETEROGENEITY, {"risk_mult_var": var, "corr_risk_inf": corr, "r0": 14.0,
                                              "dur_inf": (GAMMA, 4.51, 5.32), "heterogeneity": 1})


@pytest.mark.gpu
@pytest.mark.parametrize("pops", [[1], [31, 0, 1, 32, 33], [8191, 1, 8193], [40_000, 7, 0, 60_001], [300] * 200])
def test_gpu_choices_and_node_ids(pops):
    """Tiles of 8192 agents, words of 32, windows that cover a whole small
    node; none, one, all but one and all of a node."""
    n = np.asarray(pops)
    cap = int(n.sum()) + 21
    rng = np.random.default_rng(len(pops))
    for k in (np.zeros_like(n), np.minimum(n, 1), np.maximum(n - 1, 0), n, rng.integers(0, n + 1)):
        _both(cap, _abi.INIT_BASE | _abi.INIT_IMMUNITY, {"immune_k": k}, pops)
    for k in (0, 1, int(n.sum()) // 3, int(n.sum())):
        _both(cap, _abi.INIT_BASE | _abi.INIT_MISSED, {"missed_k": k}, pops)


@pytest.mark.gpu
@pytest.mark.parametrize("bins,deaths", [(1, 1), (17, 101), (256, 256), (257, 400)])
def test_gpu_dates(bins, deaths):
    """Tables within and beyond shared memory's 256 entries, empty bins and
    years, totals of more than 2^31 deaths."""
    rng = np.random.default_rng(bins)
    lo = np.cumsum(rng.integers(1, 90, bins)).astype(np.int32)
    w = rng.integers(0, 3, bins).astype(np.int64)
    w[-1] = 1
    fields = {"age_lo": lo, "age_hi": lo + rng.integers(1, 400, bins).astype(np.int32), "age_weight": w,
              "km_max_year": 300}
    for scale in (1, 10**8):
        fields["km"] = np.cumsum(rng.integers(0, 2, deaths) * scale).astype(np.int64)
        _both(50_021, _abi.INIT_BASE | _abi.INIT_AGES | _abi.INIT_DEATHS | _abi.INIT_RI, fields, [30_000, 20_000])
