"""The calls that programs built on this package make, for measuring them.

A case is one call of a driver: a coupler's arrays through the order-9 WENO
dycore (``time_step`` of a number of SSPRK3 cycles), through the TKE closure,
through the boundary-layer driver's whole chain of modules, or a number of
training steps of the learned limiter weights.  ``listed`` gives the cases,
``draw`` more of the same ranges; ``prepare`` builds what a program holds
before the call, ``run`` makes the call, ``exact`` evaluates the same call in
64 bits with plain torch operations (section "64-bit evaluation" below).

Grids, spacings and flows are those of this repository's generators
(porturb_b200/cases.py): the warm bubble, the neutral boundary layer, the urban
canopy and the open stratified box of the tests, built here on the device with
resolved eddies on top of the generators' noise, as the flows hold after their
first minutes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from porturb_b200 import (Coupler, Dycore, Dynamics_Euler_Stratified_WenoFV, LES_Closure, Time_Averager,
                          apply_surface_fluxes, capi, geostrophic_wind_forcing, sponge_layer)
from porturb_b200.cases import Tracer, default_options

STATE = ("density_dry", "uvel", "vvel", "wvel", "temp")
HALOS = ("immersed_proportion_halos", "immersed_roughness_halos", "immersed_temp_halos")
ETIME, ELAPSED = 600.0, 3600.0
AVERAGES = (9.0, 0.2, 0.0, 0.1, 0.5, 0.0, -0.1, 0.4, 0.0, 0.3, 9.5, 0.1, 0.0)   # in the order of capi.TAVG_NAMES
LATITUDE = 43.289340204        # the boundary-layer driver's geostrophic forcing
CELLS_MOST = 512 * 512 * 128 * 2   # cell-steps of the largest listed call


# ---------------------------------------------------------------------------
# Cases.
# ---------------------------------------------------------------------------
def _case(kind, flow, nx, ny, nz, ntr, cycles=1, precision="f32", **kw):
    return dict(kind=kind, flow=flow, nx=nx, ny=ny, nz=nz, ntr=ntr, cycles=cycles, precision=precision, **kw)


def listed():
    return [
        # The smallest call: a thin bubble on a coarse grid, one cycle per call, as unit tests and
        # tutorials run it; launches and latency count.
        dict(name="bubble_small", **_case("step", "bubble", 64, 4, 32, 1)),
        # The warm-bubble verification run in FP64 (256x4x128), ten cycles per physics step.
        dict(name="bubble_f64", **_case("step", "bubble", 256, 4, 128, 1, 10, "f64")),
        # An ordinary small LES tile with the boundary-layer tracers, one physics step of ten cycles.
        dict(name="abl_small", **_case("step", "abl", 64, 64, 48, 2, 10)),
        # The neutral boundary layer (256x256x128, water vapour and TKE) on device arrays.
        dict(name="abl", **_case("step", "abl", 256, 256, 128, 2, 4)),
        # The urban canopy (512x512x128) with immersed buildings on device arrays: the largest call.
        dict(name="urban", **_case("step", "urban", 512, 512, 128, 1, 2)),
        # An open (precursor) box of odd sizes with Coriolis, three tracers and an immersed obstacle.
        dict(name="open_odd", **_case("step", "open", 101, 67, 53, 3, 3)),
        # The boundary layer in FP64: runs that check single precision, and users who want it throughout.
        dict(name="abl_f64", **_case("step", "abl", 128, 128, 96, 2, 2, "f64")),
        # A host program whose coupler arrays live in (pinned) host memory: copies in, steps, copies out.
        dict(name="abl_host", **_case("host", "abl", 256, 256, 128, 2, 4)),
        # Learned limiter weights in the reconstruction.
        dict(name="learned", **_case("learned", "abl", 128, 128, 64, 2, 2)),
        # The TKE closure alone on the boundary layer's arrays (FP64, every physics step).
        dict(name="les", **_case("les", "abl", 256, 256, 128, 2)),
        # The boundary-layer driver's whole physics step: forcing, dycore, sponge, surface fluxes,
        # closure, time averages.
        dict(name="abl_chain", **_case("chain", "abl", 128, 96, 64, 2, 10)),
        # Training of the learned weights on harvested stencils.
        dict(name="train", **_case("train", "abl", 64, 64, 48, 2, batch=65536, steps=20)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["host", "learned", "les", "les", "chain", "train"])
    if kind == "train":
        return _case("train", "abl", 64, 64, _log_int(rng, 24, 64), 2, batch=_log_int(rng, 1000, 65536),
                     steps=rng.randint(5, 20))
    flow = rng.choice(["abl", "abl", "urban", "open", "bubble"]) if kind == "step" else "abl"
    precision = rng.choice(["f32", "f32", "f32", "f64"]) if kind == "step" else "f32"
    cycles = 1 if kind == "les" else _log_int(rng, 1, 10)
    # A cell of FP64 or learned limiter costs about four of FP32.
    most = CELLS_MOST // cycles // (4 if precision == "f64" or kind == "learned" else 1)
    while True:
        nx = _log_int(rng, 24, 512)
        ny = rng.randint(1, 8) if flow == "bubble" else _log_int(rng, 24, 512)
        nz = _log_int(rng, 24, 160)
        if kind == "learned" or rng.random() < 0.5:   # sizes of a power-of-two grid beside ragged ones
            nx, nz = max(32, nx // 32 * 32), max(24, nz // 8 * 8)
            ny = ny if flow == "bubble" else max(32, ny // 16 * 16)
        if nx * ny * nz <= most // 4:
            break
    ntr = rng.choice([1, 2, 3, 4]) if kind == "step" else 2
    if flow == "abl":
        ntr = max(2, ntr)
    return _case(kind, flow, nx, ny, nz, ntr, cycles, precision)


# ---------------------------------------------------------------------------
# Grids and flows.
# ---------------------------------------------------------------------------
def _setup(case):
    """Options, tracers and spacings of a case."""
    flow = case["flow"]
    kw, d = {}, (10.0, 10.0, 10.0)
    if flow == "bubble":
        kw, d = dict(cfl=0.8), (20000.0 / case["nx"], 312.5 / case["ny"], 10000.0 / case["nz"])
    elif flow == "urban":
        d = (2.0, 2.0, 2.0)
    elif flow == "open":
        kw, d = dict(cfl=0.5, bc_x="precursor", bc_y="precursor", latitude=45.0), (100.0, 100.0, 100.0)
    tracers = [Tracer("water_vapor", "", True, True, True)]
    for t in range(1, case["ntr"]):
        tracers.append(Tracer("TKE", "", True, False, False) if t == 1 and flow == "abl"
                       else Tracer("tracer_%d" % t, "", t % 2 == 1, False, True))
    return default_options(**kw), tracers, d


def _eddies(gen, shape, dev, amp):
    """Resolved eddies: a few modes a few cells long, zero at the floor and the lid, and grid-scale noise."""
    nz, ny, nx = shape
    z = (torch.arange(nz, dtype=torch.float64, device=dev) + 0.5)[:, None, None] / nz
    y = torch.arange(ny, dtype=torch.float64, device=dev)[None, :, None] / ny
    x = torch.arange(nx, dtype=torch.float64, device=dev)[None, None, :] / nx
    r = torch.rand(6, 5, generator=gen, device=dev, dtype=torch.float64).cpu()
    f = torch.zeros(shape, dtype=torch.float64, device=dev)
    for q in range(6):
        kx, ky = 1 + int(r[q, 0] * (nx // 12)), int(r[q, 1] * (ny // 12 + 1))
        kz = 1 + int(r[q, 2] * (nz // 12))
        f += (0.5 + float(r[q, 3])) * torch.sin(2 * math.pi * (kx * x + ky * y + float(r[q, 4]))) * \
            torch.sin(math.pi * kz * z)
    noise = torch.rand(shape, generator=gen, device=dev, dtype=torch.float64) - 0.5
    return amp * (f / 2 + 0.05 * noise * torch.sin(math.pi * z))


def _flow(case, seed, dev):
    """(base arrays, perturbed arrays, immersed proportion): the horizontally uniform column that the
    dycore's init averages, and the flow that the call starts from, as dicts of FP64 (nz, ny, nx) tensors."""
    opts, tracers, (dx, dy, dz) = _setup(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shape = (nz, ny, nx)
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    f8 = dict(dtype=torch.float64, device=dev)
    zc = (torch.arange(nz, **f8) + 0.5) * dz
    ztop = nz * dz
    if case["flow"] == "abl":
        z_inv = min(500.0, 0.5 * ztop)
        theta = torch.where(zc < z_inv, 300.0, 300.0 + 0.01 * (zc - z_inv))
    elif case["flow"] == "open":
        theta = 300.0 + 0.003 * zc
    else:
        theta = torch.full((nz,), 300.0, **f8)
    # Hydrostatic Exner function from d(pi)/dz = -g / (cp theta), by the midpoint rule between centres.
    inv = 1.0 / theta
    steps = torch.cat([inv[:1] * dz / 2, 0.5 * (inv[1:] + inv[:-1]) * dz])
    pi = 1.0 - opts["grav"] / opts["cp_d"] * torch.cumsum(steps, 0)
    press = (opts["p0"] * pi ** (opts["cp_d"] / opts["R_d"]))[:, None, None].expand(shape)
    th = theta[:, None, None].expand(shape)

    def dry(theta3):
        rho = (press / opts["C0"]) ** (1.0 / opts["gamma_d"]) / theta3
        return rho, press / (opts["R_d"] * rho)

    prop = torch.zeros(shape, **f8)
    if case["flow"] == "urban":
        lot = 20
        r = torch.rand(ny // lot + 1, nx // lot + 1, 4, generator=gen, **f8).cpu()
        for jl in range(ny // lot):
            for il in range(nx // lot):
                occ, fx, fy, h = (float(v) for v in r[jl, il])
                wx, wy, hh = int(10 + 6 * fx), int(10 + 6 * fy), int((10 + 50 * h) / dz)
                if occ < 0.7:
                    i0, j0 = il * lot + (lot - wx) // 2, jl * lot + (lot - wy) // 2
                    prop[:max(1, min(hh, nz - 12)), j0:j0 + wy, i0:i0 + wx] = 1.0
    elif case["flow"] == "open":
        prop[:nz // 3, ny // 3:ny // 3 + max(2, ny // 8), nx // 3:nx // 3 + max(2, nx // 8)] = 1.0
        prop[nz // 2, ny // 2, (3 * nx) // 4] = 0.5
    fluid = (prop < 1).to(torch.float64)

    rho, T = dry(th)
    base = dict(zip(STATE, (rho, torch.zeros(shape, **f8), torch.zeros(shape, **f8), torch.zeros(shape, **f8), T)))
    amp = {"bubble": 0.0, "abl": 1.0, "urban": 0.5, "open": 1.0}[case["flow"]]
    wind = {"bubble": (0.0, 0.0), "abl": (10.0, 0.0), "urban": (10.0, 0.0), "open": (5.0, -3.0)}[case["flow"]]
    if case["flow"] == "bubble":
        xc = (torch.arange(nx, **f8) + 0.5) * dx
        x0 = 10000.0 + 500.0 * float(torch.rand(1, generator=gen, **f8).cpu())
        rad = torch.sqrt(((xc[None, None, :] - x0) / 2000.0) ** 2 + ((zc[:, None, None] - 2000.0) / 2000.0) ** 2)
        dth = torch.where(rad <= 1.0, 3.0 * torch.cos(math.pi * rad / 2) ** 2, 0.0) + 0.0 * th
        u, v, w = (torch.zeros(shape, **f8) for _ in range(3))
        # A bubble a minute old: a rising core and its return flow.
        bell = torch.exp(-2.0 * rad ** 2)
        w += 2.0 * bell
        u += 1.0 * bell * (xc - x0)[None, None, :] / 2000.0
        if ny > 1:
            v += 0.1 * bell
    else:
        u, v, w = (_eddies(gen, shape, dev, a) for a in (amp, amp, 0.5 * amp))
        top = 400.0 if case["flow"] == "abl" else ztop
        na = {"abl": 0.25, "urban": 0.1, "open": 0.5}[case["flow"]]
        dth = na * (2 * torch.rand(shape, generator=gen, **f8) - 1) * (zc <= top).to(torch.float64)[:, None, None]
        dth = dth + _eddies(gen, shape, dev, 0.2)
        u, v, w = ((c + a) * fluid for a, c in zip((u, v, w), wind + (0.0,)))
        if ny == 1:
            v = torch.zeros(shape, **f8)
    rho_p, T_p = dry(th + dth)
    flow = dict(zip(STATE, (rho_p, u, v, w, T_p)))
    for t, tr in enumerate(tracers):
        noise = torch.rand(shape, generator=gen, **f8)
        if tr.name == "TKE":
            base["TKE"] = torch.full(shape, 0.1, **f8)
            flow["TKE"] = 0.1 + 0.1 * noise
        elif t == 0:
            base[tr.name] = torch.zeros(shape, **f8)
            flow[tr.name] = rho_p * 5e-3 * torch.exp(-zc / 2000.0)[:, None, None] * (1 + 0.05 * noise)
        else:
            base[tr.name] = torch.zeros(shape, **f8)
            flow[tr.name] = 0.1 + 0.05 * noise
    return base, {k: x.contiguous() for k, x in flow.items()}, prop.contiguous()


def _halo(a, ground, fill):
    """A field with one halo cell per side: periodic x and y, the ground's value below, `fill` above."""
    h = torch.nn.functional.pad(a[None], (1, 1, 1, 1), mode="circular")[0]
    lid = torch.full_like(h[:1], fill)
    return torch.cat([torch.full_like(h[:1], ground), h, lid]).contiguous()


def _dt(case):
    opts, _, d = _setup(case)
    return (case["cycles"] - 0.05) * opts["cfl"] * min(d) / 450.0


def _coupler(case, base, prop, device):
    opts, tracers, d = _setup(case)
    c = Coupler(device=device)
    for k, v in opts.items():
        c.set_option(k, v)
    c.distribute_mpi_and_allocate_coupled_state(case["nz"], case["ny"], case["nx"])
    c.set_grid(d[0] * case["nx"], d[1] * case["ny"], d[2] * case["nz"])
    for t in tracers:
        c.add_tracer(t.name, t.desc, t.positive, t.adds_mass, t.diffuse)
    c.set_option("idWV", 0)
    for name in STATE + ("immersed_proportion",):
        c.register_and_allocate(name, "", (case["nz"], case["ny"], case["nx"]))
    _assign(c, base)
    _assign(c, {"immersed_proportion": prop})
    return c


def _assign(c, arrays):
    for name, a in arrays.items():
        dst = c.get(name)
        if isinstance(dst, np.ndarray):
            dst[...] = a.cpu().numpy()
        else:
            dst.copy_(a)


def _weights(seed):
    """Parameters of the 9-32-32-5 network as a program loads them: rows near the ideal weights."""
    rng = np.random.default_rng(seed)
    w1 = rng.uniform(-1, 1, (32, 9)) * math.sqrt(6 / 9)
    w2 = rng.uniform(-1, 1, (32, 32)) * math.sqrt(6 / 32)
    w3 = rng.uniform(-1, 1, (5, 32)) * 0.1
    b1, b2 = (0.1 * rng.uniform(-1, 1, 32) for _ in range(2))
    b3 = np.log(np.array([5, 40, 60, 20, 1]) / 126)
    return np.concatenate([a.ravel() for a in (w1, b1, w2, b2, w3, b3)]).astype(np.float32)


def _handle(case, base, flow):
    opts, tracers, d = _setup(case)
    h = Dycore(case["nx"], case["ny"], case["nz"], *d, tracers, opts, precision=case["precision"],
               stream=torch.cuda.current_stream().cuda_stream)
    names = [t.name for t in tracers]
    split = lambda a: [a[n].contiguous() for n in STATE] + [[a[n] for n in names]]
    h.init(*split({k: v.contiguous() for k, v in base.items()}))
    return h, split(flow)


def prepare(case, seed):
    kind = case["kind"]
    base, flow, prop = _flow(case, seed, "cuda")
    if kind in ("learned", "train"):
        h, arrays = _handle(case, base, flow)
        if kind == "learned":
            h.learned_set_weights(_weights(11))
            h.set_weno_mode("learned")
        else:
            h.load_state(*arrays)
            h.learned_harvest(1 << 20, seed=seed)
            h.learned_set_weights(_weights(seed))
        return dict(case=case, handle=h, arrays=arrays, dt=_dt(case))
    c = _coupler(case, base, prop, None if kind == "host" else "cuda:0")
    state = dict(case=case, coupler=c, dt=_dt(case))
    if kind == "host":   # the host program's arrays are pinned
        state["pinned"] = []
        for name in list(c.dm):
            t = torch.from_numpy(c.dm[name]).pin_memory()
            state["pinned"].append(t)
            c.dm[name] = t.numpy()
    if kind in ("les", "chain"):
        for name, a, ground, rest in zip(HALOS, (prop, 0.0, 0.0), (1.0, 0.1, 0.0), (None, 0.1, 0.0)):
            a = a if rest is None else torch.full_like(prop, rest)
            h = _halo(a, ground, 0.0)
            c.register_and_allocate(name, "", h.shape)
            c.get(name).copy_(h)
        state["les"] = LES_Closure()
    if kind != "les":
        state["dycore"] = Dynamics_Euler_Stratified_WenoFV(precision=case["precision"])
        state["dycore"].init(c)
    if kind == "chain":
        state["averager"] = Time_Averager()
        state["averager"].init(c)
        c.set_option("time_averager_etime", ETIME)   # an hour into the run, ten minutes into the averages
        c.set_option("elapsed_time", ELAPSED)
        for name, value in zip(capi.TAVG_NAMES, AVERAGES):
            c.get(name)[...] = value
    _assign(c, flow)
    return state


def run(state):
    case, dt = state["case"], state["dt"]
    kind = case["kind"]
    if kind == "train":
        r = state["handle"].learned_train(case["steps"], batch=case["batch"], lr=1e-3, seed=5)
        return {"weights": state["handle"].learned_get_weights(), "loss": r["loss_last"]}
    if kind == "learned":
        state["handle"].time_step(*state["arrays"], dt)
        return state["arrays"]
    c = state["coupler"]
    if kind == "les":
        state["les"].apply(c, dt)
    elif kind == "chain":
        geostrophic_wind_forcing(c, dt, LATITUDE, 10.0, 0.0)
        state["dycore"].time_step(c, dt)
        sponge_layer(c, dt, dt * 100, 0.1)
        apply_surface_fluxes(c, dt)
        state["les"].apply(c, dt)
        state["averager"].accumulate(c, dt)
        c.set_option("elapsed_time", c.get_option("elapsed_time") + dt)
    else:
        state["dycore"].time_step(c, dt)
    out = {n: c.get(n) for n in STATE + tuple(c.get_tracer_names())}
    if kind == "chain":
        out.update({n: c.get(n) for n in capi.TAVG_NAMES})
    return out


def work(case):
    """Bytes: each coupler array in and out once.  Operations: per cell, direction, field and stage one
    order-9 limiter (five smoothness indicators, two sets of mapped weights, ten edge values: about 400
    operations with a multiply-add as two)."""
    n = case["nx"] * case["ny"] * case["nz"]
    S = 5 + case["ntr"]
    dirs = 2 if case["ny"] == 1 else 3
    steps = 3 * case["cycles"]
    limiter = n * steps * dirs * (S + 1) * 400.0
    if case["kind"] == "train":
        b = case["steps"] * case["batch"]
        return {"bytes": b * 14 * 4.0, "flops": b * 6.0 * 1504}
    if case["kind"] == "les":
        return {"bytes": 8.0 * n * (2 * S - 2), "flops": 400.0 * n}
    if case["kind"] == "chain":
        return {"bytes": 8.0 * n * (2 * S + 26), "flops": limiter + 600.0 * n}
    return {"bytes": 8.0 * n * 2 * S, "flops": limiter}


def tolerance(case):
    """About four times the largest error against the 64-bit evaluation or, where there is none, four times
    what a change of the inputs by one FP32 rounding makes (measured: the vertical wind of the urban canopy
    3.6e-5, of the other FP32 flows 1e-5 to 2e-5; the horizontal wind of the FP64 bubble 4e-11; the closure
    2e-16; the learned form 5e-5; weights after training 7e-5)."""
    kind = case["kind"]
    if kind == "les":
        return {"rel": 1e-13}
    if kind == "train":
        return {"rel": 3e-4}
    if kind == "learned":
        return {"rel": 2e-4, "max": 0.02}
    if case["precision"] == "f64":
        return {"rel": 2e-10}
    return {"rel": 1.5e-4 if case["flow"] == "urban" else 8e-5, "max": 0.02}


# ---------------------------------------------------------------------------
# 64-bit evaluation with plain torch operations.
# ---------------------------------------------------------------------------
HS = 4
IDEAL = [5 / 126, 40 / 126, 60 / 126, 20 / 126, 1 / 126]


def _sub_stencils():
    """Per sub-stencil k (entries k..k+4 of a 9-cell stencil): the matrix from its five cell averages to
    the coefficients a_0..a_4 of its quartic about the centre cell."""
    out = []
    for k in range(5):
        A = np.zeros((5, 5))
        for row, o in enumerate(range(k - 4, k + 1)):
            for d in range(5):
                A[row, d] = ((o + 0.5) ** (d + 1) - (o - 0.5) ** (d + 1)) / (d + 1)
        out.append(np.linalg.inv(A))
    return out


SUB = _sub_stencils()


def _weno(s, do_map, imm_l, imm_r):
    """Left and right edge values of the centre cell of nine cell-average tensors s[0..8]."""
    tv, left, right = [], [], []
    for k in range(5):
        a = [sum(float(SUB[k][d, m]) * (s[k + m] - s[4]) for m in range(5) if k + m != 4) for d in range(5)]
        tv.append(a[1] ** 2 + 0.5 * a[1] * a[3] + 13 / 3 * a[2] ** 2 + 4.2 * a[2] * a[4] + 3129 / 80 * a[3] ** 2 +
                  625.8 * a[4] ** 2)
        even, odd = a[0] + a[2] / 4 + a[4] / 16, a[1] / 2 + a[3] / 8
        left.append(s[4] + even - odd)
        right.append(s[4] + even + odd)
    tot = sum(tv)
    scale = torch.where(tot > 1e-20, 1.0 / tot.clamp_min(1e-300), 1.0)
    tv = [t * scale for t in tv]
    if imm_l is not None:
        mx = torch.stack(tv).amax(0)
        tv[4], tv[0] = torch.where(imm_l, mx, tv[4]), torch.where(imm_r, mx, tv[0])
    rk = [1.0 / (t * t + 1e-20) for t in tv]
    out = []
    for ideal, vals in ((IDEAL, left), (IDEAL[::-1], right)):
        w = [i * r for i, r in zip(ideal, rk)]
        tot = sum(w)
        w = [x / tot for x in w]
        m = []
        for x, i in zip(w, ideal):
            t6, u = (x - i) ** 6, x * (1 - x)
            m.append(i + t6 * (x - i) / (t6 + 2000.0 * u * u * u))
        if do_map is not None:
            m = [torch.where(do_map, y, x) for x, y in zip(w, m)]
        out.append(sum(x * v for x, v in zip(m, vals)) / sum(m))
    return out


class _Exact:
    """The dycore and the modules beside it on FP64 coupler arrays."""

    def __init__(self, case, seed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.case = case
        self.o, self.tracers, self.d = _setup(case)
        self.base, self.a, self.prop = _flow(case, seed, dev)
        self.shape = (case["nz"], case["ny"], case["nx"])
        self.names = [t.name for t in self.tracers]
        self.dev = dev
        self.dt = _dt(case)

    # -- dycore -------------------------------------------------------------
    def total(self, a):
        o = self.o
        p = a["density_dry"] * o["R_d"] * a["temp"] + a["water_vapor"] * o["R_v"] * a["temp"]
        rho = a["density_dry"] + sum(a[t.name] for t in self.tracers if t.adds_mass)
        return rho, (p / o["C0"]) ** (1.0 / o["gamma_d"])

    def init(self):
        o, dz = self.o, self.d[2]
        g, C0, grav = o["gamma_d"], o["C0"], o["grav"]
        rho, rt = self.total(self.base)
        mean = lambda x: x.mean((1, 2))
        r, t, p = mean(rho), mean(rt / rho), mean(C0 * rt ** g)
        ext = [[], [], []]
        for below in (True, False):
            k0 = 0 if below else -1
            for kk in (range(HS, 0, -1) if below else range(1, HS + 1)):
                dg = grav * (g - 1) * dz * kk / (g * C0 * t[k0] ** g)
                rr = (r[k0] ** (g - 1) + (dg if below else -dg)) ** (1 / (g - 1))
                for q, x in zip(ext, (rr, t[k0], C0 * (rr * t[k0]) ** g)):
                    q.append(x)
        prof = [torch.cat([torch.stack(e[:HS]), x, torch.stack(e[HS:])]) for e, x in zip(ext, (r, t, p))]
        n = self.shape[0]
        edge = lambda x: (-x[HS - 2:HS + n - 1] + 7 * x[HS - 1:HS + n] + 7 * x[HS:HS + n + 1] -
                          x[HS + 1:HS + n + 2]) / 12
        self.rh, self.th, self.ph = (x[HS:-HS][:, None, None] for x in prof)
        self.re, self.te = edge(prof[0].log()).exp()[:, None, None], edge(prof[1])[:, None, None]
        self.imm = self.prop > 0
        self.has_imm = bool(self.imm.any())
        if self.has_imm:
            self.any10 = self.spread(self.imm, 10)
            tau = torch.full(self.shape, 1.0, dtype=torch.float64, device=self.dev)
            for reach, v in ((3, 2.0), (2, 4.0), (1, 8.0)):
                tau[self.spread(self.prop == 0, reach)] = v
            self.mult = self.prop ** o["immersed_power"] / tau

    def spread(self, mask, reach):
        """Cells with a set cell within `reach` in each index (x and y periodic)."""
        m = mask.clone()
        for dim in (0, 1, 2):
            acc = m.clone()
            for off in range(1, reach + 1):
                for s in (off, -off):
                    q = torch.roll(m, s, dim)
                    if dim == 0:
                        if off >= m.shape[0]:
                            continue
                        q[:off] = False if s > 0 else q[:off]
                        if s < 0:
                            q[-off:] = False
                    acc |= q
            m = acc
        return m

    def enforce(self, q):
        if self.has_imm:
            target = [self.rh, 0.0, 0.0, 0.0, self.rh * self.th] + [0.0] * len(self.tracers)
            q = [x + (t - x) * self.mult for x, t in zip(q, target)]
        for i, tr in enumerate(self.tracers):
            if tr.positive:
                q[5 + i] = q[5 + i].clamp_min(0.0)
        return q

    def tendency(self, q):
        o, F = self.o, 6 + len(self.tracers)
        rho = q[0]
        f = [rho - self.rh, q[1] / rho, q[2] / rho, q[3] / rho, q[4] / rho - self.th,
             o["C0"] * q[4] ** o["gamma_d"] - self.ph] + [x / rho for x in q[5:]]
        tend = [torch.zeros(self.shape, dtype=torch.float64, device=self.dev) for _ in q]
        nz, ny, nx = self.shape
        for dim in (2, 1, 0):
            n = self.shape[dim]
            if dim == 1 and ny == 1:
                continue
            idn = 3 - dim                      # the normal velocity among f
            bc = o[("bc_z", "bc_y", "bc_x")[dim]]
            i = torch.arange(-5, n + 5, device=self.dev)
            src = i % n if bc == "periodic" else i.clamp(0, n - 1)
            # Slabs of the other directions bound the memory of the stencil's temporaries.
            along = 1 if dim == 0 else 0
            m = self.shape[along]
            slab = max(1, int(4e6 // (self.shape[0] * ny * nx // m)))
            for lo in range(0, m, slab):
                cut = lambda x: x.narrow(along, lo, min(slab, m - lo)) if x.shape[along] > 1 else x
                E = []
                pos = lambda x, off, count: x.narrow(dim, off, count)
                imm = None
                if self.has_imm or dim == 0:
                    fl = cut(self.imm).index_select(dim, i % n)
                    if dim == 0:
                        out = (i < 0) | (i >= n)
                        fl = fl | out[:, None, None]
                    imm = [pos(fl, mm, n + 2) for mm in range(9)]
                do_map = ~pos(cut(self.any10).index_select(dim, i % n), 4, n + 2) if self.has_imm else None
                for l in range(F):
                    x = cut(f[l]).index_select(dim, src)
                    if bc == "solid_wall" and l in (3, 4):
                        x.narrow(dim, 0, 5).zero_()
                        x.narrow(dim, n + 5, 5).zero_()
                    s = [pos(x, mm, n + 2) for mm in range(9)]
                    if imm is not None and l in (1, 2, 3, 5) and l != idn:
                        s = self.der0(s, imm)
                    E.append(_weno(s, do_map, None if imm is None else imm[3], None if imm is None else imm[5]))
                L = [e[1].narrow(dim, 0, n + 1).clone() for e in E]
                R = [e[0].narrow(dim, 1, n + 1).clone() for e in E]
                del E
                if bc == "precursor":
                    for a, b in zip(L, R):
                        a.narrow(dim, 0, 1).copy_(b.narrow(dim, 0, 1))
                        b.narrow(dim, n, 1).copy_(a.narrow(dim, n, 1))
                if bc == "solid_wall":
                    for l, (a, b) in enumerate(zip(L, R)):
                        a.narrow(dim, 0, 1).copy_(b.narrow(dim, 0, 1))
                        b.narrow(dim, n, 1).copy_(a.narrow(dim, n, 1))
                        if l in (3, 4):
                            for y in (a, b):
                                y.narrow(dim, 0, 1).zero_()
                                y.narrow(dim, n, 1).zero_()
                hr, ht = (self.re, self.te) if dim == 0 else (cut(self.rh), cut(self.th))
                ruL, ruR = L[idn] * (L[0] + hr), R[idn] * (R[0] + hr)
                p = 0.5 * (L[5] + R[5] - 350.0 * (ruR - ruL))
                ru = 0.5 * (ruL + ruR - (R[5] - L[5]) / 350.0)
                up = ru > 0
                flux = [ru] + [ru * torch.where(up, L[l], R[l]) for l in (1, 2, 3)] + \
                    [ru * (torch.where(up, L[4], R[4]) + ht)] + [ru * torch.where(up, L[l], R[l]) for l in range(6, F)]
                flux[idn] = flux[idn] + p
                for x, fl in zip(tend, flux):
                    cut(x).sub_(torch.diff(fl, dim=dim) / self.d[2 - dim])
        if ny == 1:
            tend[2].zero_()
        tend[3] -= o["grav"] * f[0]
        fcor = 2 * 7.2921e-5 * math.sin(o["latitude"] / 180 * math.pi)
        if fcor and ny > 1:
            tend[1] += fcor * q[2]
            tend[2] -= fcor * q[1]
        return tend

    @staticmethod
    def der0(s, imm):
        """Values beyond the first immersed cell, outward from a fluid centre, repeat the last fluid one."""
        s = list(s)
        for order in ((5, 6, 7, 8), (3, 2, 1, 0)):
            hit, v = torch.zeros_like(imm[4]), s[4]
            for m in order:
                new = imm[m] & ~hit
                v = torch.where(new, s[m - 1 if m > 4 else m + 1], v)
                hit = hit | new
                s[m] = torch.where(hit & ~imm[4], v, s[m])
        return s

    def time_step(self):
        a, o = self.a, self.o
        dt = self.dt / self.case["cycles"]
        rho, rt = self.total(a)
        q = [rho, rho * a["uvel"], rho * a["vvel"], rho * a["wvel"], rt] + [a[n] for n in self.names]
        for _ in range(self.case["cycles"]):
            q0 = self.enforce(q)
            step = lambda x, c, t: [y + c * (z - y) + t * w for y, z, w in zip(x, q0, self.tendency(x))]
            q = self.enforce(step(q0, 0.0, dt))
            q = self.enforce(step(q, 0.75, dt / 4))
            q = self.enforce(step(q, 1 / 3, 2 * dt / 3))
        rho = q[0]
        dry = rho - sum(q[5 + t] for t, tr in enumerate(self.tracers) if tr.adds_mass)
        a["density_dry"] = dry
        for n, x in zip(STATE[1:4], q[1:4]):
            a[n] = x / rho
        a["temp"] = o["C0"] * q[4] ** o["gamma_d"] / (dry * o["R_d"] + q[5] * o["R_v"])
        for n, x in zip(self.names, q[5:]):
            a[n] = x

    # -- modules beside the dycore (periodic x and y, walls in z, no immersed cells but the ground) ---
    def geostrophic(self):
        fcor = 2 * 7.2921e-5 * math.sin(LATITUDE / 180 * math.pi)
        um, vm = (self.a[n].mean((1, 2), keepdim=True) for n in ("uvel", "vvel"))
        self.a["uvel"] = self.a["uvel"] + self.dt * fcor * vm
        self.a["vvel"] = self.a["vvel"] - self.dt * fcor * (um - 10.0)

    def sponge(self):
        nz, dz = self.shape[0], self.d[2]
        z = (torch.arange(nz, dtype=torch.float64, device=self.dev) + 0.5)[:, None, None] * dz
        z1, z2 = 0.9 * nz * dz, nz * dz
        fac = torch.where(z > z1, ((z - z1) / (z2 - z1)) ** 3 / 100.0, 0.0)
        for n in ("uvel", "vvel", "wvel", "temp"):
            m = 0.0 if n == "wvel" else self.a[n].mean((1, 2), keepdim=True)
            self.a[n] = fac * m + (1 - fac) * self.a[n]

    def surface(self):
        cd = (0.4 / math.log((self.d[2] / 2 + 0.1) / 0.1)) ** 2
        u, v = self.a["uvel"][0], self.a["vvel"][0]
        mag = torch.sqrt(u * u + v * v)
        for n, x in (("uvel", u), ("vvel", v)):
            y = self.a[n].clone()
            y[0] = x - self.dt * cd * x * mag / self.d[2]
            self.a[n] = y

    def les(self):
        a, o, dt = self.a, self.o, self.dt
        dx, dy, dz = self.d
        g, C0, grav = o["gamma_d"], o["C0"], o["grav"]
        diffused = [t.name for t in self.tracers if t.diffuse]
        rho = a["density_dry"]
        th = (rho * o["R_d"] * a["temp"] / C0) ** (1 / g) / rho
        f = [rho, a["uvel"], a["vvel"], a["wvel"], th, (a["TKE"] / rho).clamp_min(0.0)] + \
            [a[n] / rho for n in diffused]

        def halo(x, l):
            x = torch.nn.functional.pad(x[None], (1, 1, 1, 1), mode="circular")[0]
            lo, hi = x[:1].clone(), x[-1:].clone()
            if l == 3:
                lo, hi = torch.zeros_like(lo), torch.zeros_like(hi)
            if l == 0:
                t = torch.nn.functional.pad(th[None], (1, 1, 1, 1), mode="circular")[0]
                add = lambda tt: grav * (g - 1) * dz / (g * C0 * tt ** g)
                lo, hi = (lo ** (g - 1) + add(t[:1])) ** (1 / (g - 1)), (hi ** (g - 1) - add(t[-1:])) ** (1 / (g - 1))
            return torch.cat([lo, x, hi])

        H = [halo(x, l) for l, x in enumerate(f)]
        sp = {2: dx, 1: dy, 0: dz}
        delta = (dx * dy * dz) ** (1 / 3)
        inner = lambda x, dims: x[tuple(slice(1, -1) if q in dims else slice(None) for q in range(3))]
        tend = [torch.zeros(self.shape, dtype=torch.float64, device=self.dev) for _ in range(5 + len(diffused))]
        for dim in (2, 1, 0):
            others = [q for q in (0, 1, 2) if q != dim]
            c = 2 - dim
            normal = lambda l: inner(torch.diff(H[l], dim=dim), others) / sp[dim]
            avg = lambda x: 0.5 * (x.narrow(dim, 0, x.shape[dim] - 1) + x.narrow(dim, 1, x.shape[dim] - 1))

            def tang(l, e):
                n = H[l].shape[e]
                x = (H[l].narrow(e, 2, n - 2) - H[l].narrow(e, 0, n - 2)) / (2 * sp[e])
                return inner(avg(x), [q for q in others if q != e])

            G = {(v, e): (normal(1 + v) if 2 - e == dim else tang(1 + v, 2 - e))
                 for v in range(3) for e in range(3) if e == c or v == e or v == c}
            dtdz = normal(4) if dim == 0 else tang(4, 0)
            r, K, t = (inner(avg(H[l]), others) for l in (0, 5, 4))
            N = torch.where(dtdz >= 0, torch.sqrt((grav / t * dtdz).clamp_min(0.0)), 0.0)
            ell = (0.76 * K.sqrt() / (N + 1e-20)).clamp_max(delta)
            km = 0.1 * ell * K.sqrt()
            cap = 0.5 * 0.25 * sp[dim] ** 2 / dt
            nu, nut = km.clamp_max(cap), (km * (1 + 2 * ell) / delta).clamp_max(cap)
            div = G[0, 0] + G[1, 1] + G[2, 2]
            flux = []
            for v in range(3):
                flux.append(-r * nu * (2 * G[v, v] - 2 / 3 * div if v == c else G[v, c] + G[c, v]))
            flux += [-r * nut * normal(4), -2 * r * nu * normal(5)] + [-r * nu * normal(6 + q)
                                                                      for q in range(len(diffused))]
            if dim == 0:   # the ground is fully immersed: no flux through it
                for x in flux:
                    x[0] = 0.0
            for x, fl in zip(tend, flux):
                x.sub_(torch.diff(fl, dim=dim) / sp[dim])
        C = lambda l: inner(H[l], (0, 1, 2))
        shift = lambda l, e, s: inner(torch.roll(H[l], -s, e), (0, 1, 2))
        K, t = C(5), C(4)
        dtdz = (shift(4, 0, 1) - shift(4, 0, -1)) / (2 * dz)
        N = torch.where(dtdz >= 0, torch.sqrt((grav / t * dtdz).clamp_min(0.0)), 0.0)
        ell = (0.76 * K.sqrt() / (N + 1e-20)).clamp_max(delta)
        km = 0.1 * ell * K.sqrt()
        src = -grav * rho * km * (1 + 2 * ell) / delta / t * dtdz
        src = src - rho * (0.19 + 0.51 * ell / delta) / delta * K ** 1.5
        D = {}
        for e in range(3):
            for v in range(3):
                lo, hi = shift(1 + v, 2 - e, -1), shift(1 + v, 2 - e, 1)
                if e == 2 and v != 2:
                    lo = lo.clone()
                    lo[0] = C(1 + v)[0]     # the ground's tangential wind is the cell's own
                D[e, v] = (hi - lo) / (2 * sp[2 - e])
        src = src + rho * km * sum((D[e, v] + D[v, e]) * D[e, v] for e in range(3) for v in range(3))
        tend[4] += src
        for l, n in enumerate(STATE[1:4]):
            a[n] = a[n] + dt * tend[l] / rho
        a["temp"] = C0 * (th * rho + dt * tend[3]) ** g / (rho * o["R_d"])
        a["TKE"] = (f[5] * rho + dt * tend[4]).clamp_min(0.0)
        for q, n in enumerate(diffused):
            a[n] = a[n] + dt * tend[5 + q]

    def averages(self):
        a, dt = self.a, self.dt
        x = [a[n] for n in STATE[1:4]]
        inl, inn = ELAPSED / (ELAPSED + dt), ETIME / (ETIME + dt)
        long_avg = [inl * o + (1 - inl) * y for o, y in zip(AVERAGES[10:], x)]
        p = [y - m for y, m in zip(x, long_avg)]
        pairs = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
        samples = x + [a["TKE"]] + [p[i] * p[j] for i, j in pairs]
        return dict(zip(capi.TAVG_NAMES, [inn * o + (1 - inn) * y for o, y in zip(AVERAGES, samples)] + long_avg))


def exact(case, seed):
    kind = case["kind"]
    # The network's weights and activations are bfloat16 by definition: no 64-bit value.
    if kind in ("learned", "train"):
        return None
    e = _Exact(case, seed)
    if kind == "les":
        e.les()
        return e.a
    e.init()
    if kind != "chain":
        e.time_step()
        return e.a
    e.geostrophic()
    e.time_step()
    e.sponge()
    e.surface()
    e.les()
    return {**e.a, **{n: x for n, x in e.averages().items()}}
