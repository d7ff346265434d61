"""A tuned launch shape is the one launched, for the kernel it was timed for and
no other."""
import numpy as np
import pytest

from simradar_gb300 import synth

pytestmark = pytest.mark.gpu


def scene(seed=51, rain=400000):
    return synth.make_scene(num_rain=rain, les_count=1, seed=seed)


@pytest.mark.parametrize("precision", [0, 1])
def test_worker_shape_is_of_the_timed_kernel(backend, precision):
    S = scene()
    pop, sd = synth.population(S), synth.pulse_sim_desc(S, 50)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_precision(precision)
    W.make_pulse(sd)
    before = W.pulse_shape
    W.advance_time(pop, 0, sd)
    W.make_pulse(sd)
    ordered = W.pulse_shape
    assert min(before) > 0 and min(ordered) > 0
    # timed out of order: pulses in order keep their default
    W.upload(0, pos=S.state["pos"])
    unsorted = W.autotune(sd)
    W.make_pulse(sd)
    assert W.pulse_shape == unsorted
    W.advance_time(pop, 0, sd)
    W.make_pulse(sd)
    assert W.pulse_shape == ordered
    # timed in order
    tuned = W.autotune(sd)
    W.advance_time(pop, 0, sd)
    W.make_pulse(sd)
    assert W.pulse_shape == tuned
    # set by hand: for all
    W.set_pulse_shape(4, 2)
    W.make_pulse(sd)
    assert W.pulse_shape == (4, 2)
    W.upload(0, pos=S.state["pos"])
    W.make_pulse(sd)
    assert W.pulse_shape == (4, 2)
    W.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("interval,steps", [(128, 3), (128, 150), (0, 3), (600, 200)])
def test_batch_shape_is_the_launched_one(backend, interval, steps, precision):
    """Tuned before the first run, on a state not yet sorted: the runs launch
    that shape, whichever form their pulses take (600: parts too long for the
    node sums), and tuning changes neither state nor aux / sig."""
    scenes = [scene(52, 300000), scene(53, 70000)]
    ws = []
    for S in scenes:
        W = backend.Worker(0)
        synth.load_worker(W, S)
        W.set_sort_interval(interval)
        W.make_pulse(synth.pulse_sim_desc(S, 40))
        ws.append(W)
    B = backend.Batch(ws)
    B.set_populations([synth.population(S) for S in scenes])
    B.set_precision(precision)
    fields = ("pos", "vel", "rcs", "rnd", "aux", "sig")
    sims = np.stack([np.stack([synth.pulse_sim_desc(S, 40 + k % 40) for S in scenes]) for k in range(steps)])
    before = ws[0].download(fields)
    tuned = B.autotune(sims[0])
    after = ws[0].download(fields)
    assert all(np.array_equal(before[f].view(np.uint32), after[f].view(np.uint32)) for f in fields)
    assert min(tuned) > 0
    for _ in range(2):
        B.run(sims)
        assert B.pulse_shape == tuned
    B.close()
    for W in ws:
        W.close()
