"""The plain pulse summed on the nodes of the gate grid (rsc_nodes.cuh): every
half width of the triangle, in gate spacings, that takes this path, at sizes
around its runs of 64, against the oracle's exact sum of the reference's FP32
contributions.

Tolerance.  As everywhere 2e-5 of the gate's sum of |w x| for the order of
the FP32 additions; and, because the interpolated weight is not the lerp's
bit pattern, 2.5e-7 of the sum of |x| in the triangle's reach: the lerp's
index (at most 2) is rounded at 2^-24 x 2, its mix and the interpolation's
two roundings each at 2^-24.  The gates' sums of |w x| over the reach add up
to at least that sum of |x|.
"""
import numpy as np
import pytest

from simradar_gb300 import synth

pytestmark = pytest.mark.gpu


def check(g, direct, ab, n, where):
    pad = np.pad(ab, ((n, n), (0, 0)))
    reach = sum(pad[k:k + len(ab)] for k in range(2 * n + 1))
    lim = 2.0e-5 * ab + 2.5e-7 * reach + 1e-30
    d = np.abs(g.astype(np.float64) - direct.astype(np.float64))
    assert np.isfinite(g).all() and (d <= lim).all(), "%s: worst %g of the bound" % (where, (d / lim).max())


@pytest.mark.parametrize("spacing,gates,rain,debris", [
    (30.0, 20, 256, 0),       # n = 1; the smallest state that is sorted
    (15.0, 40, 5000, 100),    # n = 2; sparse debris
    (7.5, 77, 4097, 3000),    # n = 4; debris dense enough to be a range of its own
    (2.5, 240, 20001, 0),     # n = 12: more gates than the window of the gate sums holds
    (1.5, 512, 1999, 33),     # n = 20, as many gates as there can be
    (15.0, 1, 777, 0),        # one gate
])
def test_node_sums_match_oracle(backend, oracle_lib, spacing, gates, rain, debris):
    O = oracle_lib
    objs = [(synth.OBJ_LEAF, debris), (synth.OBJ_BRICK, debris // 2 + 1)] if debris else []
    S = synth.make_scene(num_rain=rain, debris=objs, gates=gates, gate_spacing=spacing, les_count=1, seed=5)
    n = int(round(30.0 / spacing))
    pop = synth.population(S)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    st = O.OracleState(S.state)
    rng = np.random.default_rng(6)
    for k in range(4):
        sd = synth.pulse_sim_desc(S, 40 + k)
        if k == 3:
            # positions replaced in slots that stay in the earlier order: no
            # run of 64 lies together
            cur = W.download(("pos",))["pos"]
            cur[:rain] = cur[rng.permutation(rain)]   # drops among drops: debris has no radius
            W.upload(0, pos=cur)
            st.s["pos"][:] = cur
        W.make_pulse(sd)
        g = W.download_pulse(1.0)
        direct, ab = O.make_pulse_direct(st, S, sd, return_abs=True)
        check(g, direct, ab, n, "pulse %d" % k)
        W.advance_time(pop, 0, sd)
        O.advance_time(st, S, S.counts, S.les[0], sd)
    got = W.download(("pos", "vel", "ori", "tum", "rcs", "rnd"))
    for f, a in got.items():
        assert np.array_equal(a.view(np.uint32), st.s[f].view(np.uint32)), f
    W.close()


def test_node_sums_far_off_the_beam(backend, oracle_lib):
    """Scatterers beyond 60 degrees off the beam (and one behind it) take the
    general signal inside the node form."""
    O = oracle_lib
    S = synth.make_scene(num_rain=3000, les_count=1, seed=8)
    pop = synth.population(S)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    st = O.OracleState(S.state)
    sd = synth.pulse_sim_desc(S, 50)
    W.advance_time(pop, 0, sd)
    O.advance_time(st, S, S.counts, S.les[0], sd)
    for az in (61.0, 68.0, 180.0):
        sd = synth.pulse_sim_desc(S, 50)
        sd[0], sd[1], sd[2] = synth.beam_unit(az, 3.0)
        # an antenna table that is not zero out there
        W.set_angular_weight(np.array([1.0, 0.5, 0.25], np.float32), np.array([0.6, 0.0, 2.0, 0.0], np.float32))
        S.ang_w, S.ang_desc = np.array([1.0, 0.5, 0.25], np.float32), np.array([0.6, 0.0, 2.0, 0.0], np.float32)
        W.make_pulse(sd)
        g = W.download_pulse(1.0)
        direct, ab = O.make_pulse_direct(st, S, sd, return_abs=True)
        assert ab.max() > 0.0
        check(g, direct, ab, 2, "azimuth %g" % az)
    W.close()


def test_mid_range_roots_and_quotients(backend):
    """rsc_mid.cuh's roots and quotients are the correctly rounded ones."""
    rng = np.random.default_rng(9)
    m = rng.integers(0, 1 << 23, 1 << 20, dtype=np.uint32)
    e = rng.integers(87, 168, (2, 1 << 20), dtype=np.uint32) << np.uint32(23)
    m[:4] = (0, 1, 0x7fffff, 0x7ffffe)
    a = (m | e[0]).view(np.float32)
    b = (np.roll(m, 1) | e[1]).view(np.float32)
    assert np.array_equal(backend.eval_math(13, a), np.sqrt(a))
    assert np.array_equal(backend.eval_math(14, a, b), a / b)
    assert np.array_equal(backend.eval_math(14, np.ones_like(b), b), np.float32(1.0) / b)


@pytest.mark.parametrize("spacing,gates,rain,debris", [
    (30.0, 20, 256, 0), (7.5, 77, 4097, 3000), (2.5, 240, 9001, 0), (1.5, 512, 1999, 33), (15.0, 1, 777, 0),
])
def test_compensated_node_sums(backend, oracle_lib, spacing, gates, rain, debris):
    """The compensated pulse of every half width of the triangle against FP64:
    5e-9 of the sum of |w x| for the terms (the range to 2e-14 in the phase of
    2.5e5 rad; the sine and cosine add 1e-10), and the output's own
    rounding of its component."""
    O = oracle_lib
    objs = [(synth.OBJ_LEAF, debris), (synth.OBJ_BRICK, debris // 2 + 1)] if debris else []
    S = synth.make_scene(num_rain=rain, debris=objs, gates=gates, gate_spacing=spacing, les_count=1, seed=5)
    pop = synth.population(S)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_precision(1)
    st = O.OracleState(S.state)
    for k in range(3):
        sd = synth.pulse_sim_desc(S, 40 + k)
        W.make_pulse(sd)
        g = W.download_pulse(1.0).astype(np.float64)
        r64, ab = O.make_pulse_f64(st, S, sd, return_abs=True)
        lim = 5.0e-9 * ab + 6.0e-8 * np.abs(r64) + 1e-30
        assert (np.abs(g - r64) <= lim).all(), "pulse %d: worst %g of the bound" % (k, (np.abs(g - r64) / lim).max())
        W.advance_time(pop, 0, sd)
        O.advance_time(st, S, S.counts, S.les[0], sd)
    W.close()
