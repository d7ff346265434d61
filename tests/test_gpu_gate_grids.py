"""Plain pulses on gate grids that FP32 does not hold, where the running sum of
the gate origins drifts from the spacing (and, last, on one it does hold):
the weights are pass 1's on every route, in spatial order, out of it and from
the caller's own buffers, against the oracle's exact sum of the reference's
FP32 contributions.

A few scatterers far apart, so that a gate has one or two in its reach and no
sum hides a weight.  Tolerance: check() of test_gpu_nodes.
"""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_nodes import check
from test_gpu_nodes_any import own_buffers_pulse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0.0, 30000.0])
@pytest.mark.parametrize("spacing,gates,n", [
    (30.0 / 9.0, 120, 9),
    (29.979 / 2.0, 38, 2),
    (1.2, 400, 25),
    (0.6, 512, 50),
    (2.5, 128, 12),
])
def test_weights_on_drifting_grids(backend, oracle_lib, spacing, gates, n, offset):
    O = oracle_lib
    num, rng = 300, np.random.default_rng(11)
    S = synth.make_scene(num_rain=num, gates=gates, gate_spacing=spacing, range_offset=offset, les_count=1, seed=5,
                         concept=0, tau=n * spacing / 1.5e8)
    start, reach = 1850.0 + offset, gates * spacing
    pos = S.state["pos"]
    r = start + rng.uniform(-30.0, reach + 30.0, num)
    few = np.arange(0, num, 17)
    r[few] = start + (np.arange(len(few)) + rng.uniform(0.0, 0.3, len(few))) * reach / len(few)
    pos[:, 0], pos[:, 2] = rng.uniform(-40.0, 40.0, num), rng.uniform(5.0, 60.0, num)
    pos[:, 1] = np.sqrt(r ** 2 - pos[:, 0].astype(np.float64) ** 2 - pos[:, 2].astype(np.float64) ** 2)
    rcs = np.zeros((num, 4), np.float32)
    rcs[few] = rng.standard_normal((len(few), 4))
    sd = synth.pulse_sim_desc(S, 50)
    sd[11] = 0.0
    sd[0], sd[1], sd[2] = synth.beam_unit(0.0, 0.8 if offset == 0.0 else 0.05)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.advance_time(synth.population(S), 0, sd)   # a step of no length: sorted, nothing moves
    W.upload(0, rcs=rcs)
    S.state["rcs"] = rcs
    direct, ab = O.make_pulse_direct(O.OracleState(S.state), S, sd, return_abs=True)
    assert (ab > 0.0).any()
    W.make_pulse(sd)
    check(W.download_pulse(1.0), direct, ab, n, "in order")
    U = backend.Worker(0)
    synth.load_worker(U, S)
    U.set_sort_interval(0)
    U.make_pulse(sd)
    check(U.download_pulse(1.0), direct, ab, n, "caller's order")
    B = backend.Batch([W])
    B.set_populations([synth.population(S)])
    check(B.run(sd.reshape(1, 1, 16))[0, 0], direct, ab, n, "batch")
    B.close()
    if gates <= 128:
        check(own_buffers_pulse(backend, S, pos, rcs, sd), direct, ab, n, "own buffers")
    W.close()
    U.close()
