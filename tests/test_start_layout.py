"""The engine's start (node histogram, node-major scatter, recount, first
events) against the oracle at node sizes around the scatter's 512-slot runs
and the 2048-slot chunks, which put the nodes' runs of the input at every
byte alignment; the columns read back must be the input's, bit for bit, and
a few ticks and the invariant check follow.  No tolerance.
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


@pytest.mark.parametrize(
    "pops",
    [
        [512, 511, 513, 1, 2048, 2047, 2049, 1535, 3, 4097],
        [5, 7, 8, 9, 255, 256, 257, 2],  # less than one run of the scatter, histogram groups of eight
        [6000],
    ],
)
def test_start_keeps_every_column(pops):
    n = len(pops)
    pars = PropertySet(
        {
            "seed": 23,
            "start_date": lp.date("2019-01-01"),
            "dur": 30,
            "init_pop": np.array(pops),
            "cbr": np.full(n, 40.0),
            "init_immun": np.full(n, 0.3),
            "init_prev": np.full(n, 0.1),
            "r0": 14,
            "r0_scalars": np.ones(n),
            "distances": np.abs(np.arange(n)[:, None] - np.arange(n)[None, :]) * 20.0,
            "migration_method": "gravity",
            "gravity_k": 0.5,
            "max_migr_frac": 0.2,
            "vx_prob_ri": np.full(n, 0.6),
            "stop_if_no_cases": False,
            "verbose": 0,
        }
    )
    sim = lp.SEIR_ABM(pars)
    sim.components = [lp.VitalDynamics_ABM, lp.DiseaseState_ABM, lp.RI_ABM, lp.Transmission_ABM]
    for n_ticks in (0, 15):
        spec, cols_o, res_o = snapshot(sim)
        _, cols_g, res_g = snapshot(sim)
        so = run_spec_oracle(spec, cols_o, res_o, n_ticks)
        sg = run_spec_gpu(spec, cols_g, res_g, n_ticks, check=True)
        assert (sg.t, sg.count, sg.error) == (so.t, so.count, so.error)
        assert_same(res_o, res_g, "result")
        assert_same(cols_o, cols_g, "column", count=so.count)
