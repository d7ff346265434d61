"""The compensated pulse where its interval sums are delicate, against the FP64
pulse of the same state: scatterers within a rounding of a node of the gate
grid, gates fine beside the range's own spacing, and values near the end of
FP32's range.
"""
import numpy as np
import pytest

from simradar_gb300 import synth

pytestmark = pytest.mark.gpu


def still_worker(backend, S, one_warp=False):
    """A worker whose state has been sorted by a step of no length: positions
    are the scene's, in spatial order."""
    S.concept = 0
    S.sim_desc[5] = synth.fbits(0)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_precision(1)
    if one_warp:
        W.set_pulse_shape(1, 1)
    sd = synth.pulse_sim_desc(S, 50)
    sd[11] = 0.0
    W.advance_time(synth.population(S), 0, sd)
    assert W.sort_count == 1
    assert np.array_equal(W.download(("pos",))["pos"], S.state["pos"])
    return W, sd


def both(W, sd):
    W.make_pulse(sd)
    comp = W.download_pulse(1.0).astype(np.float64)
    W.set_precision(2)
    W.make_pulse(sd)
    ref = W.download_pulse(1.0).astype(np.float64)
    W.set_precision(1)
    return comp, ref


@pytest.mark.parametrize("start,spacing,node", [
    (1850.1, 7.5, 27),         # a start FP32 does not hold on the ranges' grid
    (1850.0, 30.0 / 7.0, 39),  # a spacing it does not hold
    (1850.0, 15.0, 12),        # both held
])
def test_scatterers_just_below_a_node(backend, start, spacing, node):
    """Scatterers 1e-8 to 6e-7 m below the node that ends a warp's window of two
    intervals: their offset from its start is the spacing in FP32, yet they
    belong to it.  The rest of the scatterers, without backscatter, bring the
    windows there; the pulse is that of the few.

    Tolerance: that of the documented form, 1e-5 of a gate, taken of the
    largest; a scatterer left out is 1 / sqrt(count) of it."""
    n, rng = 40000, np.random.default_rng(3)
    S = synth.make_scene(num_rain=n, gates=int(570 / spacing), gate_spacing=spacing, range_start=start, les_count=1, seed=5)
    R = float(np.float32(start)) + node * float(np.float32(spacing))
    few = rng.choice(np.arange(n // 2, n), 1500, replace=False)
    x0 = rng.uniform(15.0, 25.0, n)
    r = np.empty(n)
    r[:n // 2] = R - spacing - rng.uniform(0.01, 0.3, n // 2)
    r[n // 2:] = R - rng.uniform(0.01, 0.3, n - n // 2)   # one shell of the order
    r[few] = R - rng.uniform(1e-8, 6e-7, len(few))
    pos = S.state["pos"]
    pos[:, 2] = 1.0
    pos[:, 1] = np.sqrt(r ** 2 - x0 ** 2 - 1.0)
    y = pos[:, 1].astype(np.float64)
    pos[:, 0] = np.sqrt(r ** 2 - y ** 2 - 1.0)          # the range to 2e-8 m
    assert np.isfinite(pos).all()
    W, sd = still_worker(backend, S, one_warp=True)
    sd[0], sd[1], sd[2] = synth.beam_unit(0.5, 0.0)
    rcs = np.zeros((n, 4), np.float32)
    rcs[few] = rng.standard_normal((len(few), 4))
    W.upload(0, rcs=rcs)
    comp, ref = both(W, sd)
    top = np.abs(ref).max()
    assert top > 0.0
    assert (np.abs(comp - ref) <= 1.0e-5 * top).all(), np.abs(comp - ref).max() / top
    W.close()


def test_gates_fine_beside_the_range(backend):
    """Gates 1/16 m apart at 31,850 m, where FP32 ranges are 1/512 m apart: the
    tail of a scatterer's offset in its interval is then a hundredth of the
    gate, and what a term's tail times it leaves out shows in the gate.

    Tolerance: FP32 output, 2^-24 of the gate, and the range's 2^-48 (1.1e-10 m:
    1.4e-8 rad of phase, 2e-9 of the gate) added at random; 2^-23 of the
    largest gate covers both."""
    n, rng = 4096, np.random.default_rng(4)
    S = synth.make_scene(num_rain=n, gates=64, gate_spacing=0.0625, range_offset=30000.0, les_count=1, seed=5,
                         tau=0.125 / 1.5e8)
    r = rng.uniform(31849.9, 31854.1, n)
    x, z = rng.uniform(-200.0, 200.0, n), rng.uniform(1.0, 300.0, n)
    pos = S.state["pos"]
    pos[:, 0], pos[:, 2] = x, z
    pos[:, 1] = np.sqrt(r ** 2 - pos[:, 0].astype(np.float64) ** 2 - pos[:, 2].astype(np.float64) ** 2)
    W, sd = still_worker(backend, S)
    sd[0], sd[1], sd[2] = synth.beam_unit(0.0, 0.25)
    W.upload(0, rcs=rng.standard_normal((n, 4)).astype(np.float32))
    comp, ref = both(W, sd)
    top = np.abs(ref).max()
    assert (np.abs(comp - ref) <= 2.0 ** -23 * top).all(), np.abs(comp - ref).max() / top
    W.close()


@pytest.mark.parametrize("word,value", [(0, np.nan), (1, np.inf), (4, np.nan), (4, np.inf)])
def test_beam_that_is_not_finite(backend, word, value):
    """A wave number that is not finite makes every scatterer's term NaN, and NaN
    times a weight of 0 reaches every gate: also when no scatterer is in a
    gate's reach, as in the FP64 pulse and the sums gate by gate.  (A beam that
    is not finite leaves the terms finite, on the antenna table's end.)"""
    n = 1024
    S = synth.make_scene(num_rain=n, gates=10, les_count=1, seed=5)
    rng = np.random.default_rng(6)
    az, el = np.radians(rng.uniform(-7.0, 7.0, n)), np.radians(rng.uniform(1.0, 15.0, n))
    pos = S.state["pos"]
    pos[:, 0], pos[:, 1] = 2300.0 * np.cos(el) * np.sin(az), 2300.0 * np.cos(el) * np.cos(az)
    pos[:, 2] = 2300.0 * np.sin(el)                    # gates up to 2,015 m
    W, sd = still_worker(backend, S)
    comp, ref = both(W, sd)
    assert (comp == 0.0).all() and (ref == 0.0).all()
    sd[word] = value
    comp, ref = both(W, sd)
    W.set_moments(False)
    gates, _ = both(W, sd)
    assert np.array_equal(np.isnan(comp), np.isnan(gates))
    if word == 4:
        assert np.isnan(ref).all() and np.isnan(comp).all()
    W.close()


@pytest.mark.parametrize("r,x", [(20.0, 3.0e38), (10.0, 1.0e38), (20.0, 1.0e-33)])
def test_sums_at_the_ends_of_fp32(backend, r, x):
    """512 equal terms whose sums, or moments, pass FP32's largest value, and
    whose tails are below its smallest normal: a gate is the FP64 one, to 1e-5
    and to 2^-23 of the terms (the triangle's ends are where its FP32 scale
    puts them, 2^-24 of a weight off the nodes), or not finite where a sum on
    the way cannot be held, never another finite value."""
    n = 512
    S = synth.make_scene(num_rain=n, gates=3, range_start=10.0, les_count=1, seed=5,
                         box=(-50.0, 1.0, -50.0, 100.0, 100.0, 100.0))
    pos = S.state["pos"]
    pos[:, :3] = 0.0, r, 0.0
    pos[:, 0] = np.linspace(-1e-3, 1e-3, n)
    W, sd = still_worker(backend, S)
    sd[0], sd[1], sd[2] = 0.0, 1.0, 0.0
    W.upload(0, rcs=np.tile(np.array([x, 0.0, x, 0.0], np.float32), (n, 1)))
    with np.errstate(over="ignore"):
        comp, ref = both(W, sd)
    ok = np.isfinite(comp)
    fits = np.isfinite(ref)
    lim = 1.0e-5 * np.abs(ref) + 2.0 ** -23 * n * x / r ** 2
    bad = ok & ~(fits & (np.abs(comp - np.where(fits, ref, 0.0)) <= lim))
    assert not bad.any(), (comp, ref)
    if x < 1.0:
        assert ok.all()
    W.close()


@pytest.mark.parametrize("spacing,gates", [(7.5, 89), (7.5, 90), (3.75, 44), (3.75, 45)])
def test_out_of_order_on_fine_gates(backend, oracle_lib, spacing, gates):
    """A state out of spatial order on gates too fine for moments, on both sides
    of the line from which its scatterers go to their intervals one by one:
    the bound of test_compensated_node_sums, 5e-9 of the sum of |w x| and the
    output's rounding."""
    O = oracle_lib
    S = synth.make_scene(num_rain=20011, gates=gates, gate_spacing=spacing, les_count=1, seed=5)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_precision(1)
    sd = synth.pulse_sim_desc(S, 50)
    r64, ab = O.make_pulse_f64(O.OracleState(S.state), S, sd, return_abs=True)
    for _ in range(2):
        W.make_pulse(sd)
        g = W.download_pulse(1.0).astype(np.float64)
        assert (np.abs(g - r64) <= 5.0e-9 * ab + 6.0e-8 * np.abs(r64) + 1e-30).all()
    W.close()
