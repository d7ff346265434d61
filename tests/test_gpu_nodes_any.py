"""The plain pulse of a state in the caller's order, each scatterer added to its
two nodes of the gate grid by itself (k_pulse_nodes_any): a worker that does
not sort, and the pulse from the caller's own buffers, against the oracle's
exact sum of the reference's FP32 contributions; at sizes around a warp's 64
scatterers, from one gate to more than the warps' sums hold (which take the
gates' own sums), with scatterers off the beam and one that is not finite.

Tolerance: check() of test_gpu_nodes (the same weights, and FP32 sums per warp
and node of fewer terms than the bound's 2e-5 allows for).
"""
import ctypes

import numpy as np
import pytest

from simradar_gb300 import synth

from test_gpu_nodes import check

pytestmark = pytest.mark.gpu


def own_buffers_pulse(backend, S, pos, rcs, sd):
    torch = pytest.importorskip("torch")
    lib = backend.load_library()
    f = ctypes.POINTER(ctypes.c_float)
    fn = lib.rsc_make_pulse_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, f, ctypes.c_uint32, f, f, ctypes.c_uint32, f,
                   ctypes.c_float, ctypes.c_float, ctypes.c_uint32, f, ctypes.c_void_p, ctypes.c_void_p]
    fn.restype = ctypes.c_int
    p = lambda a: a.ctypes.data_as(f)  # noqa: E731
    tabs = [np.ascontiguousarray(a, np.float32) for a in (S.range_w, S.range_desc, S.ang_w, S.ang_desc, sd)]
    rw, rd, aw, ad, sim = tabs
    dp, dx = torch.from_numpy(pos).cuda(), torch.from_numpy(rcs).cuda()
    out = torch.full((S.range_count, 4), np.nan, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(2):   # the second call finds the scratch the first one left
        assert fn(dp.data_ptr(), dx.data_ptr(), len(pos), p(rw), rw.size, p(rd), p(aw), aw.size, p(ad),
                  float(S.range_start), float(S.range_delta), int(S.range_count), p(sim), out.data_ptr(), stream) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("spacing,gates", [
    (30.0, 20),     # n = 1: the gates' own sums
    (15.0, 40),     # n = 2
    (15.0, 1),      # one gate
    (7.5, 77),      # n = 4: wider than the window of the gate sums
    (2.5, 240),     # n = 12
    (1.5, 400),     # n = 20: the warps' sums no longer fit
])
@pytest.mark.parametrize("num", [2, 63, 64, 65, 20001])
def test_callers_order(backend, oracle_lib, spacing, gates, num):
    O = oracle_lib
    S = synth.make_scene(num_rain=num, gates=gates, gate_spacing=spacing, les_count=1, seed=7)
    n = int(round(30.0 / spacing))
    rng = np.random.default_rng(8)
    S.state["pos"] = np.ascontiguousarray(S.state["pos"][rng.permutation(num)])
    if num > 64:
        S.state["pos"][num // 2, :3] *= np.float32(-1.0)      # behind the beam
        S.state["pos"][num - 1, 0] += np.float32(5000.0)      # beyond every gate, far off the beam
    S.state["rcs"] = rng.standard_normal((num, 4)).astype(np.float32)
    sd = synth.pulse_sim_desc(S, 12)
    st = O.OracleState(S.state)
    direct, ab = O.make_pulse_direct(st, S, sd, return_abs=True)
    W = backend.Worker(0)
    synth.load_worker(W, S)
    W.set_sort_interval(0)
    for _ in range(2):
        W.make_pulse(sd)
    check(W.download_pulse(1.0), direct, ab, n, "worker")
    if gates <= 128:
        check(own_buffers_pulse(backend, S, S.state["pos"], S.state["rcs"], sd), direct, ab, n, "own buffers")
    # a value that is not finite reaches every gate, as in pass 1 (0 x NaN is NaN)
    S.state["rcs"][num // 2, 2] = np.nan
    W.upload(0, rcs=S.state["rcs"])
    W.make_pulse(sd)
    g = W.download_pulse(1.0)
    assert np.isnan(g[:, 2:]).all() and np.isfinite(g[:, :2]).all()
    if gates <= 128:
        g = own_buffers_pulse(backend, S, S.state["pos"], S.state["rcs"], sd)
        assert np.isnan(g[:, 2:]).all() and np.isfinite(g[:, :2]).all()
    W.close()
