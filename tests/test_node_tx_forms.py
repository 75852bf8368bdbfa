"""The exposure counts with several nodes a CTA (nodes spread over the SMs, at
most 32 a CTA) against the oracle, bit for bit: CTAs whose nodes belong to
different replicates, last CTAs that are partly filled, zero-inflated and
overdispersed seeding beside local infectivity, more nodes than 32 an SM.
No tolerance: integer state and float columns are identical on both sides.
"""

import pytest

from laser_polio_gb300 import synthetic
from oracle_backend import assert_same
from oracle_backend import run_spec_oracle
from oracle_backend import snapshot
from test_parity_gpu import _busy_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "nodes,zis",
    [
        ((139, 14), (0.4,)),  # 157 nodes: two a CTA, the last CTA with one
        ((774,) * 6 + (300,), (0.0, 0.4)),  # 4952 nodes: more than 32 for each of 152 SMs
    ],
)
def test_nodes_of_several_replicates_share_a_cta(nodes, zis):
    from laser_polio_gb300._lib import Handle

    sims = [synthetic.nigeria_like(n_agents=60 * n, n_nodes=n, dur=20, seed=70 + k) for k, n in enumerate(nodes)]
    for k, zi in enumerate(zis):
        sims.insert(1 + 2 * k, _busy_sim(seed=40 + k, dur=20 + 5 * k, zi=zi, disp=2))
    snaps_o = [snapshot(s) for s in sims]
    snaps_g = [snapshot(s) for s in sims]
    states_o = [run_spec_oracle(spec, cols, res, s.nt - 1) for s, (spec, cols, res) in zip(sims, snaps_o)]
    h = Handle([spec.desc for spec, _, _ in snaps_g])
    for i, (_, cols, _) in enumerate(snaps_g):
        h.bind_columns(i, cols)
    h.start()
    h.step(max(s.nt for s in sims) - 1)
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
