"""aux and sig are those of the latest pulse (scat_sig_aux), or what was
uploaded since, however many steps and downloads follow it: bit for bit
against the oracle, whose steps do not touch them."""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_parity import assert_state_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("materialize", [False, True])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("interval", [0, 2, 128])
def test_sig_aux_of_the_latest_pulse(backend, oracle_lib, interval, fused, materialize):
    O = oracle_lib
    S = synth.make_scene(num_rain=2000, debris=[(synth.OBJ_LEAF, 100)], les_count=1, seed=41)
    pop = synth.population(S)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_sort_interval(interval)
    W.set_fused_step(fused)
    W.set_materialize(materialize)
    st = O.OracleState(S.state)

    def same(where):
        assert_state_equal(W.download(("aux", "sig")), st.s, fields=("aux", "sig"), where=where)

    def advance(k):
        sd = synth.pulse_sim_desc(S, k, tic=k * 1e-3)
        W.advance_time(pop, 0, sd)
        O.advance_time(st, S, S.counts, S.les[0], sd)

    for r in range(3):
        sd = synth.pulse_sim_desc(S, 40 + r)
        W.make_pulse(sd)
        O.make_pulse(st, S, sd)
        if r == 1:
            # new debris backscatter is not in the pulse that went before
            W.update_debris_rcs(pop, sd)
            W.upload(0, rcs=st.s["rcs"])
        for k in range(4):
            advance(41 + r)
            if k != 1:
                same("pulse %d, %d steps later " % (r, k + 1))
    # uploaded ones stay until the next pulse
    aux = np.random.default_rng(2).standard_normal(st.s["aux"].shape).astype(np.float32)
    W.upload(0, aux=aux)
    st.s["aux"][:] = aux
    for k in range(3):
        advance(50 + k)
        same("uploaded, %d steps later " % (k + 1))
    W.close()
