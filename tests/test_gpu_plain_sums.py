"""Plain sums of many equal terms that reach the nodes one by one: a state out
of spatial order, on more gates than the warps' sums hold, whose neighbours
lie in different gates.  150,000 additions of one value in FP32 are off by up
to 1e-2 of the sum, in FP64 by nothing to speak of.

Tolerance: check() of test_gpu_nodes."""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_nodes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num", [65, 300007])
def test_many_equal_terms(backend, oracle_lib, num):
    O = oracle_lib
    S = synth.make_scene(num_rain=num, gates=512, gate_spacing=1.5, les_count=1, seed=7)
    pos = S.state["pos"]
    pos[:, :3] = 0.0, 1900.0, 100.0
    pos[1::2, :3] = 0.0, 2100.0, 110.0
    S.state["rcs"][:] = 0.7, 0.1, 0.9, -0.3
    sd = synth.pulse_sim_desc(S, 50)
    direct, ab = O.make_pulse_direct(O.OracleState(S.state), S, sd, return_abs=True)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_sort_interval(0)
    for _ in range(2):   # the second finds the sums the first one left
        W.make_pulse(sd)
        check(W.download_pulse(1.0), direct, ab, 20, "worker")
    B = backend.Batch([W])
    B.set_populations([synth.population(S)])
    check(B.run(sd.reshape(1, 1, 16))[0, 0], direct, ab, 20, "batch")
    B.close()
    W.close()


@pytest.mark.parametrize("warps", [1, 2, 8])
def test_blocks_of_few_warps(backend, oracle_lib, warps):
    """The last block's sums of the nodes fit its shared memory whatever the
    number of warps."""
    O = oracle_lib
    S = synth.make_scene(num_rain=20001, gates=77, gate_spacing=7.5, les_count=1, seed=9)
    sd = synth.pulse_sim_desc(S, 50)
    st = O.OracleState(S.state)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_pulse_shape(warps, 1)
    for k in range(2):   # out of spatial order, and in it
        W.make_pulse(sd)
        direct, ab = O.make_pulse_direct(st, S, sd, return_abs=True)
        check(W.download_pulse(1.0), direct, ab, 4, "pulse %d" % k)
        W.advance_time(synth.population(S), 0, sd)
        O.advance_time(st, S, S.counts, S.les[0], sd)
    W.close()
