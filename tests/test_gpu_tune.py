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
