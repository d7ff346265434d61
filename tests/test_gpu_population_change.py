"""Populations that change from call to call: the spatial order, made for one
population's ranges, is invisible to another whose ranges cut through them, or
which do not follow one another.  Every state is bit for bit that of a worker
that keeps the caller's order, given the same calls."""
import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_parity import STATE_FIELDS, assert_state_equal

pytestmark = pytest.mark.gpu

RAIN, LEAF, BRICK = 3000, 700, 500


def populations(backend, S):
    make = lambda counts, origins: backend.Population.make(counts, origins=origins)  # noqa: E731
    return [
        synth.population(S),
        make([RAIN, LEAF // 2, 0], [0, RAIN, 0]),                      # the first half of the leaves
        make([RAIN, LEAF - 100, BRICK], [0, RAIN + 100, RAIN + LEAF]),  # leaves and drops that do not follow
        make([RAIN // 3, LEAF, BRICK], [500, RAIN, RAIN + LEAF]),      # some of the drops
        make([0, 0, BRICK], [0, 0, RAIN + LEAF]),                      # bricks alone
        make([RAIN, 300, BRICK + 400], [0, RAIN, RAIN + 300]),         # some leaves as bricks
    ]


@pytest.mark.parametrize("fused", [False, True])
def test_ranges_cut_through_the_order(backend, fused):
    S = synth.make_scene(num_rain=RAIN, debris=[(synth.OBJ_LEAF, LEAF), (synth.OBJ_BRICK, BRICK)], les_count=1, seed=31)
    pops = populations(backend, S)
    results = []
    for interval in (2, 0):
        W = backend.Worker(0)
        synth.load_worker(W, S)
        W.set_sort_interval(interval)
        W.set_fused_step(fused)
        got = []
        for k, i in enumerate((0, 0, 1, 0, 2, 2, 3, 4, 1, 0, 0, 5, 5, 0)):
            sd = synth.pulse_sim_desc(S, 40 + k, tic=k * 1e-3)
            W.make_pulse(sd)
            W.advance_time(pops[i], 0, sd)
            if k % 3 == 2:
                W.update_debris_rcs(pops[(i + 1) % len(pops)], sd)
            got.append(W.download(STATE_FIELDS + ("aux", "sig")))
        assert (W.sort_count > 3) == (interval > 0)
        results.append(got)
        W.close()
    for k, (a, b) in enumerate(zip(*results)):
        assert_state_equal(a, b, fields=STATE_FIELDS + ("aux", "sig"), where="step %d " % k)


def test_batch_of_another_population(backend):
    S = synth.make_scene(num_rain=RAIN, debris=[(synth.OBJ_LEAF, LEAF), (synth.OBJ_BRICK, BRICK)], les_count=1, seed=32)
    pops = populations(backend, S)
    results = []
    for interval in (128, 0):
        W = backend.Worker(0)
        synth.load_worker(W, S)
        W.set_sort_interval(interval)
        sd = synth.pulse_sim_desc(S, 45)
        W.advance_time(pops[0], 0, sd)
        B = backend.Batch([W])
        for i in (1, 2, 0):
            B.set_populations([pops[i]])
            B.run(np.stack([synth.pulse_sim_desc(S, 45 + k) for k in range(3)])[:, None, :])
        B.close()
        results.append(W.download(STATE_FIELDS + ("aux", "sig")))
        W.close()
    assert_state_equal(results[0], results[1], fields=STATE_FIELDS + ("aux", "sig"))
