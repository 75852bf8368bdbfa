"""The disease-state events of a tick against the oracle, bit for bit, with
infectivities and strain scalars at the edges of the integer form of the
infectivity sums: zero, subnormal and huge values, products that round at
either of its two steps, and scalars without a short binary form.  Integer
state and float columns are identical on both sides, so there is no
tolerance.
"""

import numpy as np
import pytest

import laser_polio_gb300 as lp
from laser_polio_gb300.core import PropertySet
from oracle_backend import assert_same
from oracle_backend import run_spec_gpu
from oracle_backend import run_spec_oracle
from oracle_backend import snapshot

pytestmark = pytest.mark.gpu

EDGES = np.array(
    [0.0, 1e-45, 1.1754944e-38, 2.0**-100, 2.0**-53, 2.0**-41, 3 * 2.0**-42, 2.0**-40, 1.5 * 2.0**-40, 2.0**-9,
     1 - 2.0**-24, 1.0, 1 + 2.0**-23, 14.0, 2.0**12, 2.0**13, 2.0**21],
    np.float32,
)


@pytest.mark.parametrize("scalars", [(1.0, 0.25, 0.125), (1.0 / 3.0, 0.3, 1.0 - 2.0**-53)])
def test_infectivity_sums_at_the_edges(scalars):
    pops = np.array([20_000, 5_000, 129])
    d = np.abs(np.arange(3)[:, None] - np.arange(3)[None, :]) * 20.0
    pars = PropertySet(
        {
            "seed": 14,
            "start_date": lp.date("2019-01-01"),
            "dur": 60,
            "init_pop": pops,
            "cbr": np.full(3, 40.0),
            "init_immun": np.zeros(3),
            "init_prev": np.array([300, 40, 3]),
            "r0": 4,
            "r0_scalars": np.ones(3),
            "strain_r0_scalars": dict(enumerate(scalars)),
            "distances": d,
            "migration_method": "gravity",
            "gravity_k": 0.5,
            "max_migr_frac": 0.3,
            "stop_if_no_cases": False,
            "verbose": 0,
        }
    )
    sim = lp.SEIR_ABM(pars)
    sim.components = [lp.VitalDynamics_ABM, lp.DiseaseState_ABM, lp.Transmission_ABM]
    n = sim.people.count
    rng = np.random.default_rng(8)
    # the infectious carry the edge values from the start; the rest some of them
    inf = sim.people.daily_infectivity
    at = np.concatenate([np.flatnonzero(sim.people.disease_state[:n] > 0), rng.integers(0, n, 300)])
    inf[at] = rng.choice(EDGES[:13], len(at))
    few = rng.choice(at, 6, replace=False)
    inf[few] = rng.choice(EDGES[13:], 6)
    sim.people.strain[:n] = rng.integers(0, 3, n).astype(sim.people.strain.dtype)
    spec, cols_o, res_o = snapshot(sim)
    _, cols_g, res_g = snapshot(sim)
    so = run_spec_oracle(spec, cols_o, res_o, sim.nt - 1)
    sg = run_spec_gpu(spec, cols_g, res_g, sim.nt - 1, check=True)
    assert (sg.t, sg.stopped, sg.count, sg.error) == (so.t, so.stopped, so.count, so.error)
    assert_same(res_o, res_g, "result")
    assert_same(cols_o, cols_g, "column", count=so.count)
    assert res_o["new_exposed"].sum() > 0
