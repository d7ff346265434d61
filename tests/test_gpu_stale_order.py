"""Pulses of a state whose last sort is long past (the sort interval set by
hand): the routes for a state out of order, on arrays that are permuted, and
a batch of the same, against the oracle on the downloaded state."""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_nodes import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing,gates,n", [(15.0, 40, 2), (7.5, 77, 4), (2.5, 240, 12)])
@pytest.mark.parametrize("precision", [0, 1])
def test_pulses_long_after_the_sort(backend, oracle_lib, precision, spacing, gates, n):
    O = oracle_lib
    S = synth.make_scene(num_rain=3000, debris=[(synth.OBJ_LEAF, 200)], gates=gates, gate_spacing=spacing, les_count=1,
                         seed=71)
    pop = synth.population(S)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_sort_interval(1000)
    W.set_precision(precision)
    B = backend.Batch([W])
    B.set_populations([pop])
    B.set_precision(precision)

    def same(g, sd, state, where):
        st = O.OracleState(state)
        if precision == 0:
            direct, ab = O.make_pulse_direct(st, S, sd, return_abs=True)
            check(g, direct, ab, n, where)
        else:
            r64, ab = O.make_pulse_f64(st, S, sd, return_abs=True)
            assert (np.abs(g - r64) <= 5.0e-9 * ab + 6.0e-8 * np.abs(r64) + 1e-30).all(), where

    for k in range(300):
        W.advance_time(pop, 0, synth.pulse_sim_desc(S, k % 90))
        if k in (254, 255, 256, 299):
            sd = synth.pulse_sim_desc(S, 48)
            state = W.download()
            W.make_pulse(sd)
            same(W.download_pulse(1.0), sd, state, "%d steps" % (k + 1))
    assert W.sort_count == 1
    state, sd = W.download(), synth.pulse_sim_desc(S, 49)
    same(B.run(sd.reshape(1, 1, 16))[0, 0], sd, state, "batch")
    B.close()
    W.close()
