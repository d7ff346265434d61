"""What the emulation loop is timed on: calls as a user's program makes them.

Every case goes through the package's public entry points (the ctypes mirror
of include/rsc.h) on synthetic, seeded scenes of the shapes the tests and the
benchmark use: the default box (range 1850-2420 m, azimuth +-8 degrees,
elevation 0-18 degrees), Marshall-Palmer drops, a stretched LES grid with a
vortex and turbulence, and leaf / board / brick debris.

Kinds of case:
  loop      make_pulse, the pulse to the host, advance_time, `steps` times on
            one worker: a dwell of the radar.  `read` says how a pulse reaches
            the host: "blocking" as rs.c reads it, "queued" into page-locked
            memory with one wait at the end of the dwell.  With `state` the
            whole scatterer state is read back after the dwell.
  batch     a run of `steps` steps of several instances, every pulse copied.
  noalloc   a pulse from the caller's own device buffers.
  start     the initial state of a run: generated, uploaded and read back.
"""
import ctypes
import gc
import math

import numpy as np
import torch

from simradar_gb300 import rsc, synth

OBJECTS = (synth.OBJ_LEAF, synth.OBJ_WOODBOARD_2X4, synth.OBJ_BRICK)
CONCEPTS = {
    "dbu": synth.CONCEPT_DBU,                            # dragged, bounded, uniform DSD: the default
    "bg": 0,                                             # drops follow the wind
    "dbu+c": synth.CONCEPT_DBU | synth.CONCEPT_CROSS_POL,
}
FORMS = {"plain": rsc.PULSE_PLAIN, "compensated": rsc.PULSE_COMPENSATED}
LES_SIZES = {"small": (88, 88, 40), "readme": (176, 176, 80), "large": (352, 352, 160)}


def _loop(**kw):
    c = dict(kind="loop", rain=0, debris=0, gates=40, spacing=15.0, offset=0.0, form="plain", concept="dbu",
             read="queued", les="readme", scan="ppi", steps=8, state=False)
    c.update(kw)
    return c


def listed():
    return [
        # The first look at a scene, and the smallest call: a handful of
        # scatterers, each pulse waited for as rs.c does.
        _loop(name="first_look_4k", rain=4096, debris=64, les="small", read="blocking", steps=2),
        # The case the reference can run on a CPU: 131,072 drops, a PPI.
        _loop(name="ppi_131k", rain=131072, steps=25),
        # The README's emulation, the everyday size.
        _loop(name="readme_2m", rain=1998848, debris=1024, steps=10),
        # The same with every pulse waited for and compensated sums.
        _loop(name="readme_2m_compensated", rain=1998848, debris=1024, form="compensated", read="blocking", steps=8),
        # A distant storm, where the two-way phase needs the compensated form.
        _loop(name="far_8m_compensated", rain=8388608, offset=30000.0, form="compensated", steps=3),
        # The largest scene the benchmark runs, on its LES grid, as a batch of one.
        dict(kind="batch", name="large_33m_batch", instances=1, lo=33554432, hi=33554432, debris=43691, gates=40,
             form="compensated", les="large", steps=2),
        # An ensemble of unequal instances, as one run.
        dict(kind="batch", name="ensemble_12", instances=12, lo=65536, hi=1048576, debris=4096, gates=40,
             form="plain", les="small", steps=10),
        # A debris storm: as much debris as rain, with cross-polar returns.
        _loop(name="debris_storm_393k", rain=196609, debris=65537, concept="dbu+c", steps=10),
        # Range oversampling: a 30 m pulse sampled every 2.5 m.
        _loop(name="oversampled_500k", rain=500000, gates=240, spacing=2.5, steps=4),
        # An odd size with four gates to the pulse, no drag, an RHI, and the
        # state read back after the dwell (RS_download).
        _loop(name="rhi_state_77k", rain=77777, gates=77, spacing=7.5, concept="bg", form="compensated",
              read="blocking", scan="rhi", steps=12, state=True),
        # A pulse from device buffers another program owns, in its order.
        dict(kind="noalloc", name="own_buffers_300k", rain=300007, gates=40, spacing=15.0),
        # The start of a run: RS_populate's state on the device, read back.
        dict(kind="start", name="start_1m", rain=1000003, debris=1000),
    ]


def _log_int(rng, lo, hi):
    """A whole number log-uniform in [lo, hi]: odd ones and round ones alike."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.3:
        n = n // 1024 * 1024 if n >= 2048 else n
    return max(lo, min(hi, n))


def draw(rng):
    kind = rng.choice(["loop", "loop", "loop", "loop", "far", "debris", "fine", "state", "batch", "noalloc", "start"])
    if kind == "loop":
        rain = _log_int(rng, 4096, 2000000)
        return _loop(rain=rain, debris=rng.choice([0, 0, _log_int(rng, 16, 1024)]),
                     form=rng.choice(["plain", "compensated"]), concept=rng.choice(["dbu", "dbu", "bg"]),
                     read=rng.choice(["blocking", "queued"]), les=rng.choice(["small", "readme"]),
                     spacing=rng.choice([15.0, 30.0, 20.0]), gates=rng.randint(20, 64),
                     scan=rng.choice(["ppi", "rhi"]), steps=rng.randint(2, 12))
    if kind == "far":
        return _loop(rain=_log_int(rng, 1000000, 8000000), offset=float(rng.choice([8000, 15000, 30000])),
                     form="compensated", gates=rng.randint(30, 60), steps=rng.randint(2, 3))
    if kind == "debris":
        return _loop(rain=_log_int(rng, 1024, 400000), debris=_log_int(rng, 4096, 65537),
                     concept=rng.choice(["dbu", "dbu+c"]), form=rng.choice(["plain", "compensated"]),
                     steps=rng.randint(3, 10))
    if kind == "fine":
        spacing = rng.choice([1.5, 2.5, 3.0, 3.75, 5.0, 6.0])
        return _loop(rain=_log_int(rng, 16384, 500000), spacing=spacing, gates=rng.randint(64, min(512, int(600 / spacing))),
                     form=rng.choice(["plain", "plain", "compensated"]), steps=rng.randint(2, 4))
    if kind == "state":
        return _loop(rain=_log_int(rng, 4097, 200000), concept=rng.choice(["dbu", "bg"]), spacing=rng.choice([7.5, 15.0]),
                     gates=rng.randint(38, 77), form=rng.choice(["plain", "compensated"]), read="blocking",
                     scan="rhi", steps=rng.randint(2, 12), state=True)
    if kind == "batch":
        hi = _log_int(rng, 131072, 1048576)
        return dict(kind="batch", instances=rng.randint(2, 12), lo=_log_int(rng, 16384, 131072), hi=hi,
                    debris=rng.choice([0, 1024, 4096]), gates=rng.randint(30, 48),
                    form=rng.choice(["plain", "compensated"]), les="small", steps=rng.randint(2, 10))
    if kind == "noalloc":
        spacing = rng.choice([15.0, 30.0, 7.5])
        return dict(kind="noalloc", rain=_log_int(rng, 1000, 2000000), gates=rng.randint(20, 100), spacing=spacing)
    return dict(kind="start", rain=_log_int(rng, 10000, 1000003), debris=rng.choice([0, 100, 1000]))


# ---------------------------------------------------------------- scenes
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _les(name, seed):
    """(config, uvwt) of one LES volume: a Burgers-Rott vortex (50 m/s at
    100 m) with a weak inflow and updraft, plus 3 m/s of turbulence."""
    nx, ny, nz = LES_SIZES[name]
    grow = {"small": (1.0212 ** 2, 1.05 ** 2), "readme": (1.0212, 1.05), "large": (1.0105, 1.025)}[name]
    cfg = synth.LESConfig(nx=nx, ny=ny, nz=nz, rx=grow[0], ry=grow[0], rz=grow[1])
    x, y, z = (torch.from_numpy(np.asarray(v)).cuda().float() for v in cfg.node_positions())
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    rho2 = (X * X + Y * Y).clamp_min(1e-6)
    core = 100.0
    swirl = 50.0 * 1.398 * core / rho2 * (1.0 - torch.exp(-1.25643 * rho2 / core ** 2))
    uvwt = 3.0 * torch.randn((nz, ny, nx, 4), generator=_generator(seed + 77), device="cuda")
    uvwt[..., 0] += -swirl * Y - 0.02 * X
    uvwt[..., 1] += swirl * X - 0.02 * Y
    uvwt[..., 2] += torch.clamp(0.04 * Z, max=15.0) * torch.exp(-rho2 / (9.0 * core ** 2))
    uvwt[..., 3] = 0.0
    return cfg, uvwt


def _scene(c, seed, rain, debris):
    """Tables and descriptors of a scene (synth's), without its state."""
    types = [(o, 1) for o in OBJECTS] if debris else []
    scan = synth.rhi_positions(2.0, 0.5, 18.0, 0.25) if c.get("scan") == "rhi" else None
    S = synth.make_scene(num_rain=1, debris=types, gates=c["gates"], gate_spacing=c.get("spacing", 15.0),
                         range_offset=c.get("offset", 0.0), concept=CONCEPTS[c.get("concept", "dbu")],
                         with_tables=False, scan=scan)
    S.counts = [rain] + ([debris] * 3 if debris else [])
    S.num_scats = sum(S.counts)
    sd = S.sim_desc
    sd[3] = np.float32(S.num_scats)
    vol = float(sd[12]) * float(sd[13]) * float(sd[14])
    sd[6] = np.float32(math.sqrt(vol * S.dsd_nd / rain))
    S.ell, S.ell_desc = synth.ellipsoid_rcs_table(sd[4], sd[6], S.concept, S.dsd_r, S.dsd_pdf)
    S.beam0 = int(seed) % len(S.scan)
    return S


def _state(S, seed, vel=True):
    """Positions uniform in the box, drop sizes over the DSD's bins, drops
    falling in a breeze, unit backscatter and random respawn seeds (GPU)."""
    n, rain = S.num_scats, S.counts[0]
    g = _generator(seed)
    sd = S.sim_desc
    pos = torch.rand((n, 4), generator=g, device="cuda")
    pos[:, :3] = pos[:, :3] * torch.tensor([float(v) for v in sd[12:15]], device="cuda")
    pos[:, :3] += torch.tensor([float(v) for v in sd[8:11]], device="cuda")
    bins = torch.randint(len(S.dsd_r), (n,), generator=g, device="cuda")
    pos[:, 3] = torch.from_numpy(np.asarray(S.dsd_r)).cuda()[bins]
    pos[rain:, 3] = 0.0
    rcs = torch.zeros((n, 4), device="cuda")
    rcs[:, 0] = 1.0
    rcs[:, 2] = 1.0
    if not vel:
        return {"pos": pos, "rcs": rcs}
    v = 12.0 * torch.randn((n, 4), generator=g, device="cuda")
    v[:, 2] = 0.25 * v[:, 2] - 4.0
    v[:, 3] = 0.0
    v[rain:] = 0.0
    rnd = torch.randint(2 ** 31 - 1, (n, 4), generator=g, device="cuda", dtype=torch.int32)
    return {"pos": pos, "vel": v, "rcs": rcs, "rnd": rnd}


def _worker(c, S, state, seed, les):
    W = rsc.Worker(0)
    W.malloc(S.num_scats, S.range_start, S.range_delta, S.range_count)
    W.set_range_weight(S.range_w, S.range_desc)
    W.set_angular_weight(S.ang_w, S.ang_desc)
    W.set_rcs_ellipsoid(S.ell, S.ell_desc)
    cfg, uvwt = les
    W.set_les(0, uvwt, None, cfg.desc())
    for t, (cd, cm, ad) in enumerate(S.adm):
        W.set_adm(t, cd, cm, ad)
    for t, (re, im, rd) in enumerate(S.rcs_tables):
        W.set_rcs(t, re, im, rd)
    arrays = {k: v.cpu().numpy() for k, v in state.items()}
    arrays["rnd"] = arrays["rnd"].view(np.uint32)
    if len(S.counts) > 1:
        n = S.num_scats
        arrays["ori"] = np.broadcast_to(np.array([0.5, -0.5, -0.5, 0.5], np.float32), (n, 4))
        arrays["tum"] = np.broadcast_to(np.array([0.0, 0.0, 0.0, 1.0], np.float32), (n, 4))
    W.upload(0, **arrays)
    W.set_precision(FORMS[c["form"]])
    return W


def _sizes(c, seed):
    """Rain count of each instance of a batch: log-uniform, set by the case."""
    if c["instances"] == 1:
        return [c["hi"]]
    lo, hi = math.log(min(c["lo"], c["hi"])), math.log(max(c["lo"], c["hi"]))
    return [int(math.exp(lo + (hi - lo) * ((0.61803398875 * (i + 1)) % 1.0))) for i in range(c["instances"])]


def _batch_scenes(c, seed):
    out = []
    for i, rain in enumerate(_sizes(c, seed)):
        S = _scene(dict(c, scan="rhi" if i % 2 else "ppi"), seed + i, rain, c["debris"])
        out.append(S)
    return out


def _descs(S, steps):
    return np.stack([synth.pulse_sim_desc(S, S.beam0 + k) for k in range(steps)])


def prepare(case, seed):
    c = case
    gc.collect()
    if c["kind"] == "loop":
        S = _scene(c, seed, c["rain"], c["debris"])
        cfg, uvwt = _les(c["les"], seed)
        W = _worker(c, S, _state(S, seed), seed, (cfg, uvwt.cpu().numpy()))
        out = torch.empty((c["steps"], S.range_count, 4), pin_memory=True).numpy()
        return {"kind": "loop", "w": W, "pop": synth.population(S), "sim": _descs(S, c["steps"]), "out": out,
                "blocking": c["read"] == "blocking", "state": c["state"]}
    if c["kind"] == "batch":
        cfg, uvwt = _les(c["les"], seed)
        uvwt = uvwt.cpu().numpy()
        scenes = _batch_scenes(c, seed)
        workers = [_worker(c, S, _state(S, seed + 1000 * i), seed, (cfg, uvwt)) for i, S in enumerate(scenes)]
        B = rsc.Batch(workers)
        B.set_populations([synth.population(S) for S in scenes])
        B.set_precision(FORMS[c["form"]])
        sim = np.stack([_descs(S, c["steps"]) for S in scenes], axis=1)
        out = torch.empty((c["steps"], len(workers), B.max_gates, 4), pin_memory=True).numpy()
        return {"kind": "batch", "b": B, "sim": np.ascontiguousarray(sim), "out": out}
    if c["kind"] == "noalloc":
        S = _scene(c, seed, c["rain"], 0)
        st = _state(S, seed, vel=False)
        lib = rsc.load_library()
        f = ctypes.POINTER(ctypes.c_float)
        fn = lib.rsc_make_pulse_noalloc
        fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t, f, ctypes.c_uint32, f, f, ctypes.c_uint32, f,
                       ctypes.c_float, ctypes.c_float, ctypes.c_uint32, f, ctypes.c_void_p, ctypes.c_void_p]
        fn.restype = ctypes.c_int
        pulse = torch.empty((S.range_count, 4), device="cuda")
        tables = [rsc.f32(a) for a in (S.range_w, S.range_desc, S.ang_w, S.ang_desc, _descs(S, 1)[0])]
        return {"kind": "noalloc", "fn": fn, "pos": st["pos"], "rcs": st["rcs"], "pulse": pulse, "tables": tables,
                "gates": (float(S.range_start), float(S.range_delta), int(S.range_count))}
    S = _scene(dict(gates=40), seed, c["rain"], c["debris"])
    W = rsc.Worker(0)
    W.malloc(S.num_scats, S.range_start, S.range_delta, S.range_count)
    args = rsc.PopulateArgs.make(_start_seed(seed), S.concept, S.box[:3], S.box[3:], S.counts, S.dsd_r, S.dsd_cdf)
    return {"kind": "start", "w": W, "args": args}


def _start_seed(seed):
    return (int(seed) * 2654435761 + 12345) & 0x3FFFFFFF


def run(state):
    s = state
    if s["kind"] == "loop":
        W, pop, out = s["w"], s["pop"], s["out"]
        if s["blocking"]:
            for k, sd in enumerate(s["sim"]):
                W.make_pulse(sd)
                W.download_pulse(1.0, out=out[k])
                W.advance_time(pop, 0, sd)
        else:
            for k, sd in enumerate(s["sim"]):
                W.make_pulse(sd)
                W.download_pulse_async(out[k])
                W.advance_time(pop, 0, sd)
            W.synchronize()
        got = {"pulses": [out[k] for k in range(len(out))]}
        if s["state"]:
            got["state"] = W.download(("pos", "vel", "rcs", "rnd"))
            got["state"]["rnd"] = got["state"]["rnd"].view(np.int32)
        return got
    if s["kind"] == "batch":
        s["b"].run(s["sim"], out=s["out"])
        return {"pulses": [s["out"][k] for k in range(len(s["out"]))]}
    if s["kind"] == "noalloc":
        rw, rd, aw, ad, sim = s["tables"]
        p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))  # noqa: E731
        start, delta, gates = s["gates"]
        st = s["fn"](s["pos"].data_ptr(), s["rcs"].data_ptr(), s["pos"].shape[0], p(rw), rw.size, p(rd), p(aw), aw.size,
                     p(ad), start, delta, gates, p(sim), s["pulse"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st != 0:
            raise RuntimeError("rsc_make_pulse_noalloc: status %d" % st)
        return s["pulse"]
    bins = rsc.populate_upload(s["w"], s["args"])
    got = s["w"].download(("pos", "aux", "rnd"))
    got["rnd"] = got["rnd"].view(np.int32)
    got["bins"] = bins.view(np.int32)
    return got


def work(case):
    """Per step: every attribute that changes read and written once (rain:
    position, velocity, backscatter; debris also attitude and tumble), the
    gates written; about 160 operations for a scatterer's signal and sums
    (twice that compensated) and 250 (rain) or 700 (debris) for its step."""
    c = case
    if c["kind"] in ("loop", "batch"):
        rains = [c["rain"]] if c["kind"] == "loop" else _sizes(c, 0)
        rain, deb, k = sum(rains), 3 * c["debris"] * len(rains), c["steps"]
        per = 320 if c["form"] == "compensated" else 160
        b = k * (96 * rain + 160 * deb + 16 * c["gates"] * len(rains))
        f = k * ((per + 250) * rain + (per + 700) * deb)
        if c.get("state"):
            b += 64 * (rain + deb)
        return {"bytes": b, "flops": f}
    if c["kind"] == "noalloc":
        return {"bytes": 32 * c["rain"] + 16 * c["gates"], "flops": 160 * c["rain"]}
    n = c["rain"] + 3 * c["debris"]
    return {"bytes": (16 * 8 + 48) * n, "flops": 20 * n}


# ---------------------------------------------------------------- 64 bits
def _lerp64(table, desc, x):
    w = torch.from_numpy(np.asarray(table, np.float64)).cuda()
    m = float(desc[2])
    f = (float(desc[0]) * x + float(desc[1])).clamp(0.0, m)
    i = f.floor()
    a = f - i
    i0 = i.long()
    return w[i0] + (w[(i0 + 1).clamp(max=int(m))] - w[i0]) * a


def _pulse64(S, pos, rcs, sd):
    """The pulse of a state in 64 bits: signal, antenna and range weights,
    sums per gate."""
    G = S.range_count
    out = torch.zeros((G, 4), dtype=torch.float64, device="cuda")
    b = torch.tensor([float(v) for v in sd[:3]], dtype=torch.float64, device="cuda")
    start, delta = float(S.range_start), float(S.range_delta)
    reach = 1.0 / float(S.range_desc[0])                 # half width of the triangle
    span = int(math.ceil(2.0 * reach / delta)) + 2
    for at in range(0, pos.shape[0], 1 << 22):
        p = pos[at:at + (1 << 22), :3].double()
        x = rcs[at:at + (1 << 22)].double()
        r = p.square().sum(1).sqrt()
        ang = torch.atan2(torch.linalg.cross(b.expand_as(p), p).square().sum(1).sqrt(), p @ b)
        k = _lerp64(S.ang_w, S.ang_desc, ang) / (r * r)
        ph = float(sd[4]) * r
        s, q = torch.sin(ph), torch.cos(ph)
        sig = torch.stack([x[:, 0] * q + x[:, 1] * s, x[:, 1] * q - x[:, 0] * s,
                           x[:, 2] * q + x[:, 3] * s, x[:, 3] * q - x[:, 2] * s], dim=1) * k[:, None]
        first = torch.ceil((r - reach - start) / delta).long() - 1
        for j in range(span):
            g = first + j
            ok = (g >= 0) & (g < G)
            w = _lerp64(S.range_w, S.range_desc, r - (start + g.double() * delta))
            out.index_add_(0, g[ok], (sig * w[:, None])[ok])
    return out.cpu()


def _wind64(S, cfg, uvwt, pos):
    d = cfg.desc().astype(np.float64)
    sd = S.sim_desc.astype(np.float64)
    centre = (sd[8] + 0.5 * sd[12], sd[9] + 0.5 * sd[13], 0.0)
    dims = (cfg.nx, cfg.ny, cfg.nz)
    low, high, frac = [], [], []
    for a in range(3):
        rel = pos[:, a] - centre[a]
        u = torch.copysign(torch.full_like(rel, d[a]), rel) * torch.log1p(d[4 + a] * rel.abs()) + d[8 + a] - 0.5
        fl = u.floor()
        frac.append(u - fl)
        low.append(fl.long().clamp(0, dims[a] - 1))
        high.append((fl.long() + 1).clamp(0, dims[a] - 1))
    out = torch.zeros((pos.shape[0], 4), dtype=torch.float64, device="cuda")
    for corner in range(8):
        i = [high[a] if corner >> a & 1 else low[a] for a in range(3)]
        w = 1.0
        for a in range(3):
            w = w * (frac[a] if corner >> a & 1 else 1.0 - frac[a])
        out += w[:, None] * uvwt[i[2], i[1], i[0]].double()
    return out


def _advance64(S, cfg, uvwt, st):
    """One time step of drops in 64 bits (with or without drag; respawn of
    those that left the box)."""
    sd = S.sim_desc.astype(np.float64)
    o = torch.from_numpy(sd[8:11]).cuda()
    size = torch.from_numpy(sd[12:15]).cuda()
    dt = sd[11]
    pos, vel = st["pos"].clone(), st["vel"]
    pos[:, :3] += vel[:, :3] * dt
    gone = ((pos[:, :3] <= o) | (pos[:, :3] >= o + size)).any(1)
    bg = _wind64(S, cfg, uvwt, pos)
    if S.concept & synth.CONCEPT_DRAGGED:
        dv = bg - vel
        speed = dv[:, :3].square().sum(1).sqrt()
        re = 6.7308e4 * 2.0 * pos[:, 3] * speed
        cd = 24.0 / re + 6.0 / (1.0 + re.sqrt()) + 0.4
        k = 0.5 * 1.225 * cd * 0.003006012 / pos[:, 3] * speed
        new = vel.clone()
        new[:, :3] += k[:, None] * dv[:, :3] * dt
        new[:, 2] -= 9.8 * dt
        over = new.square().sum(1).sqrt() > (3.0 * bg.square().sum(1).sqrt()).clamp_min(1.0)
        fall = bg.clone()
        fall[:, 2] -= 9.8 * dt
        new[over] = fall[over]
    else:
        new = bg
    e = torch.from_numpy(S.ell.astype(np.float64)).cuda()
    at = (pos[:, 3] * float(S.ell_desc[0]) + float(S.ell_desc[1])).float().clamp(0.0, float(S.ell_desc[2])).long()
    t = e[at]
    h2 = pos[:, 0].square() + pos[:, 1].square()
    c2 = (h2 / (h2 + pos[:, 2].square()))[:, None]
    rcs = torch.cat([t[:, :2], t[:, :2] + (t[:, 2:] - t[:, :2]) * c2], dim=1)
    seed = (st["rnd"] * 16807) & 0x7FFFFFFF
    born = seed[:, :3].double() / 2147483647.0 * size + o
    pos[gone, :3] = born[gone]
    new[gone] = 0.0
    rcs[gone] = st["rcs"][gone]
    return {"pos": pos, "vel": new, "rcs": rcs, "rnd": torch.where(gone[:, None], seed, st["rnd"])}


def _start64(S, seed, n, rain):
    """The C library's rand() (r[i] = r[i - 3] + r[i - 31]) in the order the
    initial state draws it."""
    def sequence(s, count):
        r = [s if s else 1]
        for _ in range(30):
            r.append(16807 * r[-1] % 2147483647)
        r += r[:3]
        for _ in range(310 + count):
            r.append((r[-31] + r[-3]) & 0xFFFFFFFF)
        return np.array(r[-count:], np.uint32) >> 1
    u = sequence(seed, 8 * n).reshape(n, 8)
    unit = u[:, :4].astype(np.float64) / 2147483647.0
    pos, aux = np.zeros((n, 4)), np.zeros((n, 4))
    for a in range(3):
        pos[:, a] = unit[:, a] * (10.0 if a == 2 else float(np.float32(S.box[3 + a]))) + float(np.float32(S.box[a]))
    aux[:, 1] = unit[:, 3]
    aux[:, 3] = 1.0
    d = sequence(2 * seed & 0xFFFFFFFF, rain).astype(np.float32) / np.float32(2147483647)
    bins = (d * np.float32(len(S.dsd_r))).astype(np.int64)
    pos[:rain, 3] = np.asarray(S.dsd_r)[bins]
    aux[:rain, 2] = (bins + 0.5) / len(S.dsd_r)
    return {"pos": pos, "aux": aux, "rnd": u[:, 4:].astype(np.int32),
            "bins": np.bincount(bins, minlength=len(S.dsd_r)).astype(np.int32)}


def exact(case, seed):
    """The first pulse of a run in 64 bits (the later ones follow a state that
    has been rounded to 32 bits in between), the state after the dwell where
    it holds drops only, and the whole initial state."""
    c = case
    if c["kind"] == "loop":
        S = _scene(c, seed, c["rain"], c["debris"])
        st = _state(S, seed)
        first = _pulse64(S, st["pos"], st["rcs"], _descs(S, 1)[0])
        got = {"pulses": [first] + [None] * (c["steps"] - 1)}
        if c["state"]:
            cfg, uvwt = _les(c["les"], seed)
            st = {k: v.double() if v.is_floating_point() else v.long() for k, v in st.items()}
            if c["debris"]:
                got["state"] = {k: None for k in st}
            else:
                for _ in range(c["steps"]):
                    st = _advance64(S, cfg, uvwt, st)
                got["state"] = {k: v.cpu() for k, v in st.items()}
        return got
    if c["kind"] == "batch":
        scenes = _batch_scenes(c, seed)
        first = []
        for i, S in enumerate(scenes):
            st = _state(S, seed + 1000 * i)
            first.append(_pulse64(S, st["pos"], st["rcs"], _descs(S, 1)[0]))
        return {"pulses": [torch.stack(first)] + [None] * (c["steps"] - 1)}
    if c["kind"] == "noalloc":
        S = _scene(c, seed, c["rain"], 0)
        st = _state(S, seed, vel=False)
        return _pulse64(S, st["pos"], st["rcs"], _descs(S, 1)[0])
    S = _scene(dict(gates=40), seed, c["rain"], c["debris"])
    return _start64(S, _start_seed(seed), S.num_scats, c["rain"])
