"""rsc_batch_run_async returns once a run is queued, however many parts it
has: the calls' host time against the time the device takes for the work."""
import time

import numpy as np
import pytest

from simradar_gb300 import synth

pytestmark = pytest.mark.gpu


def queued(backend, persistent, runs, steps=500, instances=4):
    torch = pytest.importorskip("torch")
    S = synth.make_scene(num_rain=500000, les_count=1, seed=61)
    ws = []
    for _ in range(instances):
        W = backend.Worker(0)
        synth.load_worker(W, S)
        ws.append(W)
    B = backend.Batch(ws)
    B.set_populations([synth.population(S)] * instances)
    B.set_persistent(persistent)
    sims = np.stack([np.stack([synth.pulse_sim_desc(S, 40 + k % 40)] * instances) for k in range(steps)])
    out = [torch.zeros((steps, instances, B.max_gates, 4), pin_memory=True).numpy() for _ in range(runs)]
    for _ in range(2):   # buffers and graphs are there
        for o in out:
            B.run(sims, out=o, wait=False)
        B.synchronize()
    calls = []
    t0 = time.perf_counter()
    for o in out:
        t = time.perf_counter()
        B.run(sims, out=o, wait=False)
        calls.append(time.perf_counter() - t)
    B.synchronize()
    total = time.perf_counter() - t0
    assert all(np.isfinite(o).all() and (o != 0.0).any(axis=(1, 2, 3)).all() for o in out)
    B.close()
    for W in ws:
        W.close()
    return calls, total


def test_persistent_run_is_queued(backend):
    calls, total = queued(backend, True, 1)
    assert calls[0] < 0.5 * total, (calls, total)


@pytest.mark.parametrize("instances,steps", [(4, 500), (40, 100)])
def test_second_run_is_queued_behind_the_first(backend, instances, steps):
    """One run may wait in the queue behind the one under way: the call that
    queues it does not wait for parts of the first."""
    calls, total = queued(backend, False, 2, steps, instances)
    assert sum(calls) < 0.5 * total, (calls, total)
