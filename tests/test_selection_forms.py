"""The selection's forms against the oracle, bit for bit: rounds made by the
whole grid (many targets, nodes that still lack hundreds after a round),
weights beyond 32 bits (risks from 256 on), zero weights, and target offsets
beyond the shared-memory table (8192 nodes and more).  Integer state and
float columns are identical on both sides, so there is no tolerance.
"""

import numpy as np
import pytest

import laser_polio_gb300 as lp
from laser_polio_gb300 import synthetic
from laser_polio_gb300.core import PropertySet
from oracle_backend import assert_same
from oracle_backend import run_spec_gpu
from oracle_backend import run_spec_oracle
from oracle_backend import snapshot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "pops,prev,risks",
    [
        ([200_000, 30_000, 300], 400, ()),  # one node far above the rest: rounds of the grid, then of its CTA
        ([60_000, 60_000, 60_001, 2_049], 2_000, (0.0, 255.99998, 256.0, 300.0, 5000.0)),
    ],
)
def test_selection_rounds_of_the_grid(pops, prev, risks):
    n = len(pops)
    d = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :]) * 20.0
    pars = PropertySet(
        {
            "seed": 91,
            "start_date": lp.date("2019-01-01"),
            "dur": 16,
            "init_pop": np.array(pops),
            "cbr": np.full(n, 30.0),
            "init_immun": np.zeros(n),
            "init_prev": np.full(n, prev),
            "r0": 200,
            "risk_mult_var": 9.0,
            "r0_scalars": np.ones(n),
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
    if risks:
        rng = np.random.default_rng(5)
        at = rng.integers(0, sim.people.count, 400)
        sim.people.acq_risk_multiplier[at] = rng.choice(np.array(risks, np.float32), 400)
    spec, cols_o, res_o = snapshot(sim)
    _, cols_g, res_g = snapshot(sim)
    so = run_spec_oracle(spec, cols_o, res_o, sim.nt - 1)
    sg = run_spec_gpu(spec, cols_g, res_g, sim.nt - 1, check=True)
    assert (sg.t, sg.stopped, sg.count, sg.error) == (so.t, so.stopped, so.count, so.error)
    assert_same(res_o, res_g, "result")
    assert_same(cols_o, cols_g, "column", count=so.count)
    assert res_o["new_exposed"].sum(1).max() > 16_384


def test_selection_of_more_nodes_than_the_offset_table():
    from laser_polio_gb300._lib import Handle

    sims = [synthetic.nigeria_like(n_agents=20_000, n_nodes=774, dur=25, seed=60 + k) for k in range(11)]
    snaps_o = [snapshot(s) for s in sims]
    snaps_g = [snapshot(s) for s in sims]
    assert sum(spec.desc.n_nodes for spec, _, _ in snaps_g) > 8192
    states_o = [run_spec_oracle(spec, cols, res, s.nt - 1) for s, (spec, cols, res) in zip(sims, snaps_o)]
    h = Handle([spec.desc for spec, _, _ in snaps_g])
    for i, (_, cols, _) in enumerate(snaps_g):
        h.bind_columns(i, cols)
    h.start()
    h.step(sims[0].nt - 1)
    h.sync()
    for i, ((_, cols_o, res_o), (_, cols_g, res_g), so) in enumerate(zip(snaps_o, snaps_g, states_o)):
        sg = h.state(i)
        assert (sg.t, sg.stopped, sg.count, sg.error) == (so.t, so.stopped, so.count, so.error), i
        h.read_results(i, res_g)
        h.read_columns(i, cols_g)
        assert_same(res_o, res_g, f"replicate {i} result")
        assert_same(cols_o, cols_g, f"replicate {i} column", count=so.count)
    assert sum(res_o["new_exposed"].sum() for _, _, res_o in snaps_o) > 0
    h.close()
