"""lpg_init_columns beside other work on the device: its scratch is ordered on
its own stream, so a call does not wait for another stream's kernels."""

import threading
import time

import numpy as np
import pytest

from laser_polio_gb300 import synthetic
from laser_polio_gb300.engine import build_sim_spec


def _fill_seconds(stream):
    """A build of a table whose choices need more scratch than the thread's
    workspace, on `stream`."""
    import torch

    import laser_polio_gb300 as lp

    pars, immun, _ = synthetic.nigeria_like_pars(40_000_000, 60, 30, 3)
    pars.update({"init_immun": list(immun), "age_pyramid_path": None})
    with torch.cuda.stream(stream):
        t = time.perf_counter()
        sim = lp.SEIR_ABM(lp.PropertySet(pars))
        sim.components = [lp.VitalDynamics_ABM, lp.DiseaseState_ABM, lp.RI_ABM, lp.SIA_ABM, lp.Transmission_ABM]
        stream.synchronize()
        t = time.perf_counter() - t
        out = {k: v.clone() for k, v in sim.people.device_columns().items()}
        sim.components = []
    return t, out


@pytest.mark.gpu
def test_gpu_a_table_is_built_while_another_stream_works():
    import torch

    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    _, want = _fill_seconds(mine)
    torch.cuda.synchronize()
    quiet = min(_fill_seconds(mine)[0] for _ in range(2))
    torch.cuda.synchronize()
    begun, done = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with torch.cuda.stream(other):
        begun.record()
        for _ in range(20):
            torch.cuda._sleep(200_000_000)  # about a tenth of a second each, on one SM
        done.record()
    t, got = _fill_seconds(mine)
    still = not done.query()
    torch.cuda.synchronize()
    assert still, (t, quiet, begun.elapsed_time(done))
    for k in want:
        assert torch.equal(got[k], want[k]), k


@pytest.mark.gpu
def test_gpu_threads_build_tables_at_once():
    """A workspace is a thread's own, and goes with it."""
    import torch

    def build(seed, out):
        sim = synthetic.zamfara_like(n_agents=30_000, dur=10, seed=seed)
        spec = build_sim_spec(sim)
        cols = {k: (v.cpu().numpy() if hasattr(v, "cpu") else np.array(v)) for k, v in spec.columns.items()}
        out[seed] = cols

    want, got = {}, {}
    for s in range(4):
        build(s, want)
    for _ in range(3):
        ts = [threading.Thread(target=build, args=(s, got)) for s in range(4)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        torch.cuda.synchronize()
        for s in want:
            for k in want[s]:
                assert np.array_equal(want[s][k], got[s][k]), (s, k)
