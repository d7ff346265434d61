"""The batched background advance is compiled per concept and LES spacing when
the instances share them, and chooses per instance when they do not: every
combination, with the concept changing from run to run (which replaces the
captured graph), bit for bit against the oracle; and aux / sig, which no run
forms for the pulses of an earlier one, as the last pulse leaves them.
"""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_parity import STATE_FIELDS, assert_state_equal, push_to_edges

pytestmark = pytest.mark.gpu

BG, EL, EL_BOUNDED, FP = 0, synth.CONCEPT_DRAGGED, synth.CONCEPT_DBU, synth.CONCEPT_FIXED_POS


@pytest.fixture(scope="module")
def pair():
    A = synth.make_scene(num_rain=1500, debris=[(synth.OBJ_BRICK, 40)], les_count=2, seed=21)
    B = synth.make_scene(num_rain=257, with_tables=False, seed=22)
    B.les, B.les_cfg, B.les_desc = A.les, A.les_cfg, A.les_desc
    for S in (A, B):
        push_to_edges(S, n_rain=40, n_deb=0)
    return A, B


@pytest.mark.parametrize("threads", [64, 128, 256])
@pytest.mark.parametrize("uniform", [(False, False), (True, True), (False, True)])
def test_advance_forms_match_oracle(backend, oracle_lib, pair, uniform, threads):
    O = oracle_lib
    stretched = pair[0].les_desc
    flat = np.zeros(16, np.float32)      # spacing code 0: index = pos * scale + offset
    flat[0:3] = 0.1, 0.09, 0.06
    flat[4:7] = 80.0, -100.0, 0.5
    try:
        ws, sts = [], []
        for S, u in zip(pair, uniform):
            S.les_desc = flat if u else stretched
            W = backend.Worker(0)
            synth.load_worker(W, S)
            ws.append(W)
            sts.append(O.OracleState(S.state))
        Bt = backend.Batch(ws)
        Bt.set_populations([synth.population(S) for S in pair])
        Bt.set_advance_shape(threads)
        k = 0
        for concepts in ((EL, EL), (BG, BG), (EL_BOUNDED, EL), (EL, BG), (FP, FP), (FP, EL_BOUNDED), (BG, BG)):
            sims = np.zeros((2, 2, 16), np.float32)
            les = np.array([[k & 1, 0], [1, k & 1]], np.int32)
            for j in range(2):
                for i, S in enumerate(pair):
                    sims[j, i] = synth.pulse_sim_desc(S, 3 * k + j + i, tic=(2 * k + j) * 1e-3)
                    sims[j, i, 5] = synth.fbits(concepts[i])
            Bt.run(sims, les, use_graph=True)
            for j in range(2):
                for i, S in enumerate(pair):
                    O.make_pulse(sts[i], S, sims[j, i])
                    O.advance_time(sts[i], S, S.counts, S.les[les[j, i]], sims[j, i])
            k += 1
        for i, W in enumerate(ws):
            assert_state_equal(W.download(STATE_FIELDS), sts[i].s, where="instance %d " % i)
            assert_state_equal(W.download(("aux", "sig")), sts[i].s, fields=("aux", "sig"), where="instance %d " % i)
        Bt.close()
        for W in ws:
            W.close()
    finally:
        for S in pair:
            S.les_desc = stretched


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("form", ["graph", "stream", "persistent", "unsorted"])
def test_long_run_equals_short_ones(backend, pair, form, precision):
    """A run long enough to be sorted on its way (300 steps: five parts of 60)
    against the same steps as runs of 77 and 69 (parts and a shorter last
    one): states bit for bit, each
    pulse within the two sums' order (2e-5 of the sums of |w x| a side; those are at most
    3 times the pulse's largest value here, so 1.2e-4 of that)."""
    results = []
    for cuts in ([300], [77, 77, 77, 69]):
        ws = []
        for S in pair:
            W = backend.Worker(0)
            synth.load_worker(W, S)
            W.set_precision(precision)
            if form == "unsorted":
                W.set_sort_interval(0)
            ws.append(W)
        Bt = backend.Batch(ws)
        Bt.set_populations([synth.population(S) for S in pair])
        Bt.set_precision(precision)
        Bt.set_persistent(form == "persistent")
        pulses, k = [], 0
        for c in cuts:
            sims = np.stack([[synth.pulse_sim_desc(S, (k + j) % 60 + i, tic=(k + j) * 1e-3) for i, S in enumerate(pair)]
                             for j in range(c)]).astype(np.float32)
            les = np.array([[((k + j) // 50) & 1] * 2 for j in range(c)], np.int32)
            pulses.append(np.array(Bt.run(sims, les, use_graph=form != "stream")))
            k += c
        results.append((np.concatenate(pulses), [W.download(STATE_FIELDS + ("aux", "sig")) for W in ws]))
        Bt.close()
        for W in ws:
            W.close()
    (pa, sa), (pb, sb) = results
    for a, b in zip(sa, sb):
        assert_state_equal(a, b, fields=STATE_FIELDS + ("aux", "sig"))
    scale = np.abs(pb).max(axis=(2, 3), keepdims=True)
    assert (scale > 0).all() and (np.abs(pa - pb) <= 1.2e-4 * scale).all()
