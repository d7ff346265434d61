"""Queued pulse copies (rsc_download_pulse_async): a pulse that would overwrite
one still on its way to the host is formed elsewhere, so every buffer and every
blocking read has to hold the pulse that was the latest when it was asked for.

Tolerance: the same pulse formed twice differs by the order of its FP32 sums,
2e-5 of the sums of |w x| a side; those are at most 2.9 times the pulse's
largest value here, so 1.2e-4 of that covers both, and the pulses of different
beams differ by more than a tenth of it.
"""
import numpy as np
import pytest

from simradar_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("reads", [
    "a" * 11,          # more copies under way than pulses are kept
    "aab-a--ba-a",     # copies, blocking reads (b), pulses nobody reads (-)
    "-2-2b2aa2b2",     # two copies of one pulse (2)
])
def test_reads_hold_their_own_pulse(backend, precision, reads):
    torch = pytest.importorskip("torch")
    S = synth.make_scene(num_rain=3000, debris=[], gates=40, les_count=1, seed=3)
    A, B = backend.Worker(0), backend.Worker(0)
    for W in (A, B):
        synth.load_worker(W, S)
        W.set_precision(precision)
    out = torch.zeros((2 * len(reads), S.range_count, 4), dtype=torch.float32).pin_memory().numpy()
    want, got = [], []
    for k, r in enumerate(reads):
        sd = synth.pulse_sim_desc(S, 9 * k)
        A.make_pulse(sd)
        B.make_pulse(sd)
        B.synchronize()
        want.append(B.download_pulse(1.0))
        if r == "b":
            got.append((k, A.download_pulse(1.0)))
        for j in range({"a": 1, "2": 2}.get(r, 0)):
            A.download_pulse_async(out[2 * k + j])
            got.append((k, out[2 * k + j]))
    A.synchronize()
    for k, g in got:
        scale = float(np.abs(want[k]).max())
        assert scale > 0.0
        np.testing.assert_allclose(g, want[k], rtol=0, atol=1.2e-4 * scale, err_msg="read of pulse %d" % k)
    differ = [float(np.abs(want[k] - want[k - 1]).max()) / float(np.abs(want[k]).max()) for k in range(1, len(want))]
    assert min(differ) > 0.1
    A.close()
    B.close()
