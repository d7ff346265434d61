"""Batched pulses whose range weight reaches more gates than the gate window
(a triangle four gates wide a side, and a table of another shape), in every
form of the batch, against the FP64 oracle (compensated: 1e-5 of the largest
gate) and its sum of the FP32 contributions (plain: check() of
test_gpu_nodes)."""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_nodes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("interval", [0, 128])
@pytest.mark.parametrize("form", ["graph", "stream", "persistent"])
@pytest.mark.parametrize("triangle", [True, False])
def test_wide_range_weight(backend, oracle_lib, triangle, form, interval, precision):
    O = oracle_lib
    S = synth.make_scene(num_rain=3001, gates=77, gate_spacing=7.5, les_count=1, seed=5)
    if not triangle:
        S.range_w = np.array([0.0, 0.5, 1.0, 0.5, 0.0], np.float32)
        S.range_desc = np.array([2.0 / 30.0, 2.0, 4.0, 0.0], np.float32)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_sort_interval(interval)
    B = backend.Batch([W])
    B.set_populations([synth.population(S)])
    B.set_precision(precision)
    B.set_persistent(form == "persistent")
    st = O.OracleState(S.state)
    sims = np.stack([synth.pulse_sim_desc(S, 48 + k) for k in range(3)])
    for _ in range(2):   # the second run finds the accumulators the first one left
        got = B.run(sims[:, None, :], use_graph=form == "graph")
        for k, sd in enumerate(sims):
            g = got[k, 0]
            if precision == 0:
                direct, ab = O.make_pulse_direct(st, S, sd, return_abs=True)
                check(g, direct, ab, 4, "pulse %d" % k)
            else:
                r64 = O.make_pulse_f64(st, S, sd)
                assert (np.abs(g - r64) <= 1.0e-5 * np.abs(r64).max()).all() and np.abs(r64).max() > 0.0
            O.advance_time(st, S, S.counts, S.les[0], sd)
    B.close()
    W.close()
