"""Measured workloads of the time step: what a program that uses this
library asks of it, through its public entry points (lib.Solver, lib.Batch,
serve.RequestLoop), over the sizes, types and options it is used with.

Every pass starts from the state that `prepare` made (upload, or
submission to the batch) and ends with the state back in host memory, so a
pass can be repeated and gives the same answer each time.  The host arrays
are page-locked, as a program that moves states every output interval
keeps them.

The entry points exchange FP64 arrays in both forms.  The FP32 form's state
is FP32 on the device, so its results are kept here as FP32 arrays (every
value is an FP32 number: the narrowing loses nothing).

`exact` restates the step in FP64 tensors: finite-volume reconstruction,
Kurganov-Petrova fluxes, IMEX stages, implicit friction to convergence,
settling, entrainment, erosion, topography change and the ring inlet.
"""
import math

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
EPS = float(np.finfo(float).eps)

GRAV, PRES, R_AIR, CP_AIR, NU_AIR, T_AMB = 9.81, 101300.0, 287.051, 998.0, 1.48e-5, 300.0
RHO_L, CP_L, NU_L = 1000.0, 4186.0, 1.0e-6

# steps of the served jobs and of the ensemble's members whose FP64 answer
# `exact` gives (the others would take longer than it may)
EXACT_MEMBERS = 2


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    # FP32 currents run 20-32 steps a pass: over more of them the cells at an
    # inlet or a thin front carry the last bit of the state into the third
    # digit, in any FP32 arithmetic; the liquid flows do not
    return [
        # the Fortran driver's loop on the smallest served domain: one call
        # per solver routine of the reference, a few steps; latency counts
        {"name": "call_sites_64", "kind": "call_sites", "prec": 64, "nx": 64, "ny": 64, "ns": 1, "steps": 8},
        # the plain method's configuration: 200 x 200 dam break to t = 10 s
        {"name": "dam_break_200", "kind": "dam", "prec": 64, "nx": 200, "ny": 200, "ns": 1, "nrk": 2, "t_end": 10.0},
        # the second-order tableau (N_RK = 3), general stage kernels, FP32
        {"name": "dam_break_rk3", "kind": "dam", "prec": 32, "nx": 401, "ny": 263, "ns": 1, "nrk": 3, "steps": 96},
        # plain FP64 form of the pyroclastic current (the parity form)
        {"name": "current_512_fp64", "kind": "current", "prec": 64, "nx": 512, "ny": 512, "ns": 2, "settling": True,
         "entrain": False, "ring": True, "lim": 1, "spread": 0.68, "steps": 8},
        # the single-current configuration in the production form
        {"name": "current_1024", "kind": "current", "prec": 32, "nx": 1024, "ny": 1024, "ns": 2, "settling": False,
         "entrain": False, "ring": True, "lim": 1, "spread": 0.68, "steps": 24},
        # ragged rectangle, generalised minmod limiter, no inlet (a column
        # collapse started from a restart file), one class
        {"name": "collapse_ragged", "kind": "current", "prec": 32, "nx": 517, "ny": 333, "ns": 1, "settling": False,
         "entrain": False, "ring": False, "lim": 3, "spread": 0.8, "steps": 32},
        # up to the next output time, then every field that output reads
        {"name": "current_output", "kind": "output", "prec": 32, "nx": 640, "ny": 480, "ns": 2, "settling": True,
         "entrain": True, "ring": True, "lim": 1, "spread": 0.5, "steps": 32},
        # large single domain, 3 classes, entrainment: state far above L2
        {"name": "large_4096", "kind": "current", "prec": 32, "nx": 4096, "ny": 4096, "ns": 3, "settling": True,
         "entrain": True, "ring": True, "lim": 1, "spread": 0.45, "steps": 24},
        # erosion of the bed with topography change (sediment-laden flood)
        {"name": "eroding_flood", "kind": "flood", "prec": 64, "nx": 360, "ny": 180, "steps": 32},
        # a batched ensemble of debris floods from host buffers, FP32 form
        {"name": "ensemble_64", "kind": "ensemble", "prec": 32, "runs": 64, "lo": 96, "hi": 640, "steps": 80},
        # the same engine in the plain FP64 form: inlet currents
        {"name": "ensemble_fp64", "kind": "ensemble", "prec": 64, "runs": 8, "lo": 128, "hi": 512, "steps": 64},
        # the request loop: dam breaks and debris floods of 1-3 classes
        {"name": "served_16", "kind": "served", "prec": 32, "runs": 16, "lo": 64, "hi": 512, "steps": 120},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call_sites", "dam", "dam", "current", "current", "current", "current", "output", "flood",
                       "ensemble", "ensemble", "served"])
    prec = rng.choice([32, 32, 64])
    if kind == "call_sites":
        return {"kind": kind, "prec": prec, "nx": _log_int(rng, 64, 200), "ny": _log_int(rng, 64, 200),
                "ns": rng.randint(1, 3), "steps": rng.randint(4, 12)}
    if kind == "dam":
        return {"kind": kind, "prec": prec, "nx": _log_int(rng, 64, 700), "ny": _log_int(rng, 64, 400),
                "ns": rng.randint(1, 3), "nrk": rng.choice([2, 2, 3]), "steps": rng.randint(24, 96)}
    if kind in ("current", "output"):
        hi = 512 if prec == 64 else 2048
        # settling alone empties a front into films that hang on the last
        # bit: in FP32 it comes with entrainment
        settling = rng.random() < 0.6
        return {"kind": kind, "prec": prec, "nx": _log_int(rng, 160, hi), "ny": _log_int(rng, 160, hi),
                "ns": rng.randint(1, 3), "settling": settling,
                "entrain": settling and (prec == 32 or rng.random() < 0.5), "ring": rng.random() < 0.7,
                "lim": rng.choice([1, 1, 1, 3]), "spread": round(rng.uniform(0.4, 0.85), 3),
                "steps": rng.randint(4, 10) if prec == 64 else rng.randint(12, 24)}
    if kind == "flood":
        return {"kind": kind, "prec": 64, "nx": _log_int(rng, 96, 480), "ny": _log_int(rng, 64, 240),
                "steps": rng.randint(16, 40)}
    if kind == "ensemble":
        if prec == 64:
            return {"kind": kind, "prec": 64, "runs": rng.randint(2, 8), "lo": 128, "hi": rng.choice([256, 384, 512]),
                    "steps": rng.randint(16, 64)}
        return {"kind": kind, "prec": 32, "runs": rng.randint(4, 64), "lo": 96, "hi": rng.choice([384, 512, 640]),
                "steps": rng.randint(32, 80)}
    return {"kind": "served", "prec": 32, "runs": rng.randint(4, 16), "lo": 64, "hi": rng.choice([256, 384, 512]),
            "steps": rng.randint(48, 120)}


# ---------------------------------------------------------------------------
# inputs: parameters as plain values, topography and start state as tensors
# ---------------------------------------------------------------------------

def _base(nx, ny, dx, ns, prec):
    return dict(prec=prec, nx=nx, ny=ny, dx=dx, ns=ns, gas=1, energy=1, rheo=0, mu=0.0, xi=1.0, slope=0,
                rho_s=[], diam=[], cp_s=[1100.0] * ns, settling=0, entrain=0, ring=None, lim=1, nrk=2,
                erosion=None, dt0=1.0e-2, max_dt=10.0, cfl=0.24, t_end=1.0e9)


def _rand(seed, *shape):
    return torch.rand(*shape, generator=torch.Generator(device=DEV).manual_seed(seed & 0x7fffffff), device=DEV,
                      dtype=torch.float64)


def _centres(nx, ny, dx):
    return ((torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5) * dx,
            (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * dx)


def _cone(nx, ny, dx, seed, height=1500.0, sigma=2000.0, amp=20.0, modes=24):
    """A Gaussian cone with rough ground: random-phase cosines whose
    amplitudes fall with the wave number as a fractional surface's (Hurst
    0.8) do; cell centres, never below zero."""
    x, y = _centres(nx, ny, dx)
    r2 = (x[None, :] - 0.5 * nx * dx) ** 2 + (y[:, None] - 0.5 * ny * dx) ** 2
    B = height * torch.exp(-r2 / (2.0 * sigma * sigma))
    u = _rand(seed * 7 + 1, modes, 3).cpu().tolist()
    for a, b, c in u:
        k = 2.0 * math.pi / (40.0 * dx) * math.exp(-3.5 * a)      # wavelengths 40 dx and up
        th = 2.0 * math.pi * b
        w = amp * math.sqrt(2.0 / modes) * math.exp(-1.2 * 3.5 * (1.0 - a))
        fx, fy = k * math.cos(th) * x + 2.0 * math.pi * c, k * math.sin(th) * y
        B = B + w * (torch.cos(fx)[None, :] * torch.cos(fy)[:, None] - torch.sin(fx)[None, :] * torch.sin(fy)[:, None])
    return B.clamp_min(0.0)


def _rest(P, h, T, alphas, u=None, v=None):
    """Conservative state (nv, ny, nx) of a flow of thickness h, temperature
    T and solid volume fractions alphas."""
    at = sum(alphas)
    rho_c = PRES / (R_AIR * T) if P["gas"] else RHO_L
    rho_m = (1.0 - at) * rho_c + sum(a * r for a, r in zip(alphas, P["rho_s"]))
    xs = [a * r / rho_m for a, r in zip(alphas, P["rho_s"])]
    cm = sum(x * c for x, c in zip(xs, P["cp_s"])) + (1.0 - at) * rho_c / rho_m * (CP_AIR if P["gas"] else CP_L)
    q = torch.zeros(4 + P["ns"], P["ny"], P["nx"], dtype=torch.float64, device=DEV)
    q[0] = rho_m * h
    if u is not None:
        q[1], q[2] = q[0] * u, q[0] * v
    q[3] = q[0] * cm * T
    if P["energy"] and u is not None:
        q[3] += 0.5 * q[0] * (u * u + v * v)
    for i in range(P["ns"]):
        q[4 + i] = xs[i] * q[0]
    return q


def _dam(nx, ny, ns, prec, nrk, seed, t_end=1.0e9):
    """Dam break of a liquid on a flat bed, particle classes at zero
    concentration; the two depths vary a little with the seed."""
    P = _base(nx, ny, 1.0, ns, prec)
    P.update(gas=0, energy=0, rho_s=[2500.0] * ns, diam=[1.0e-4 * 10 ** i for i in range(ns)], nrk=nrk,
             dt0=1.0e-3, max_dt=1.0, t_end=t_end)
    a, b = _rand(seed, 2).cpu().tolist()
    x, _ = _centres(nx, ny, 1.0)
    h = torch.where(x < 0.5 * nx, 1.0 + 0.02 * a, 0.1 + 0.01 * b)[None, :].expand(ny, nx)
    return P, torch.zeros(ny, nx, dtype=torch.float64, device=DEV), _rest(P, h, T_AMB, [0.0] * ns)


def _current(c, seed, dx=10.0, source_r=50.0, mu=0.1, xi=1000.0, T_src=1000.0, alphas=None):
    """A gas-particle current spreading down a cone, minutes after its inlet
    opened: thickness falling with the radius to zero at the front, radial
    velocity, hot gas; with a ring inlet at the summit or without one.
    Without a spread the ground is empty and the inlet is about to open."""
    nx, ny, ns = c["nx"], c["ny"], c["ns"]
    P = _base(nx, ny, dx, ns, c["prec"])
    alphas = alphas or [0.01, 0.02, 0.01][:ns]
    P.update(rheo=1, mu=mu, xi=xi, slope=1, rho_s=[2500.0, 1500.0, 2500.0][:ns],
             diam=[1.0e-4, 1.0e-3, 1.0e-5][:ns], settling=int(c["settling"]), entrain=int(c["entrain"]),
             lim=c["lim"])
    xs, ys = 0.5 * nx * dx, 0.5 * ny * dx
    if c["ring"]:
        P["ring"] = dict(x=xs, y=ys, r=source_r, mfr=1.0e6, vel=20.0, T=T_src, alphas=alphas)
    B = _cone(nx, ny, dx, seed)
    if not c["spread"]:
        return P, B, torch.zeros(4 + ns, ny, nx, dtype=torch.float64, device=DEV)
    x, y = _centres(nx, ny, dx)
    ex, ey = x[None, :] - xs, y[:, None] - ys
    r = torch.sqrt(ex * ex + ey * ey)
    R = c["spread"] * 0.5 * min(nx, ny) * dx
    rr = (r / R).clamp_max(1.0)
    rough = 1.0 + 0.05 * (_rand(seed * 7 + 2, ny, nx) - 0.5)
    inner = source_r if c["ring"] else -1.0
    h = torch.where((r < R) & (r > inner), 3.0 * (1.0 - rr * rr) * rough, torch.zeros_like(r))
    ur = 15.0 * torch.sqrt(rr) / r.clamp_min(1.0e-9)
    return P, B, _rest(P, h, 0.95 * T_src, alphas, ur * ex, ur * ey)


def _flood(c, seed):
    """A column of sediment-laden water released over an erodible slope, the
    bed changing under it."""
    nx, ny, dx = c["nx"], c["ny"], 2.0
    P = _base(nx, ny, dx, 2, c["prec"])
    P.update(gas=0, energy=0, rheo=1, mu=0.05, xi=500.0, slope=1, rho_s=[2600.0, 2000.0], diam=[3.0e-4, 1.0e-4],
             cp_s=[900.0, 900.0], settling=1, dt0=1.0e-3, max_dt=1.0,
             erosion=dict(coeff=1.0e-3, porosity=0.4, T=290.0, depth=0.3, fract=[0.5, 0.5]))
    x, y = _centres(nx, ny, dx)
    a = _rand(seed, 1).item()
    B = (0.06 * (nx * dx - x))[None, :].expand(ny, nx).clone()
    r2 = (x[None, :] - 0.3 * nx * dx) ** 2 + (y[:, None] - 0.5 * ny * dx) ** 2
    h = torch.where(r2 <= (0.35 * ny * dx) ** 2, 2.0 + 0.2 * a, 0.0)
    return P, B, _rest(P, h, 290.0, [0.15, 0.1])


def _side(c, i):
    """Side of the i-th run: spread evenly over the range's logarithm, the
    sizes mixed in the order of the runs."""
    at = (i * 0.6180339887498949 + 0.25) % 1.0
    return int(round(c["lo"] * (c["hi"] / c["lo"]) ** at))


def _debris(side, dx, ns, prec, seed, u, settling):
    """A debris flood on an apron: a column of sediment-laden water released
    somewhere on gentle ground, with Voellmy friction."""
    P = _base(side, side, dx, ns, prec)
    P.update(gas=0, energy=0, rheo=1, mu=0.05 + 0.15 * u[0], xi=200.0 + 1800.0 * u[1], slope=1,
             rho_s=[2600.0, 2000.0, 1500.0][:ns], diam=[3.0e-4, 1.0e-4, 1.0e-3][:ns], settling=int(settling),
             max_dt=1.0)
    B = _cone(side, side, dx, seed, height=300.0, amp=4.0)
    x, y = _centres(side, side, dx)
    L = side * dx
    r2 = (x[None, :] - (0.35 + 0.3 * u[2]) * L) ** 2 + (y[:, None] - (0.35 + 0.3 * u[3]) * L) ** 2
    R2 = ((0.06 + 0.1 * u[4]) * L) ** 2
    h = torch.where(r2 < R2, (2.0 + 3.0 * u[5]) * (1.0 - 0.3 * r2 / R2), torch.zeros_like(r2))
    return P, B, _rest(P, h, 290.0, [0.05 + 0.15 * u[6], 0.1, 0.03][:ns])


def _ensemble_runs(c, seed):
    """Members of an ensemble, sides log-uniform, each its own ground, cell
    size and friction.  FP32: debris floods; FP64: gas currents from the
    opening of their inlets (inlet radius, temperature, particle fractions)."""
    out = []
    for i in range(c["runs"]):
        u = _rand(seed * 131 + i, 8).cpu().tolist()
        side = _side(c, i)
        dx = 5.0 + 15.0 * u[7]
        if c["prec"] == 32:
            out.append(_debris(side, dx, 2, 32, seed * 131 + i, u, True))
            continue
        out.append(_current(dict(nx=side, ny=side, ns=2, prec=64, settling=True, entrain=False, ring=True, lim=1,
                                 spread=0.0), seed * 131 + i, dx=dx, source_r=min(20.0 + 180.0 * u[2], 0.2 * side * dx),
                            mu=0.05 + 0.25 * u[0], xi=200.0 + 1800.0 * u[1], T_src=600.0 + 600.0 * u[3],
                            alphas=[0.005 + 0.045 * u[4], 0.005 + 0.045 * u[5]]))
    return out


def _served_runs(c, seed):
    """Jobs of a request stream: dam breaks and debris floods in turn, 1-3
    classes, step counts between a third of `steps` and `steps`."""
    out = []
    for i in range(c["runs"]):
        u = _rand(seed * 137 + i, 8).cpu().tolist()
        side = _side(c, i)
        ns, steps = 1 + (i // 2) % 3, int(c["steps"] * (1.0 + 2.0 * u[7]) / 3.0)
        if i % 2 == 0:
            run = _dam(side, side, ns, c["prec"], 2, seed * 137 + i)
        else:
            run = _debris(side, 10.0, ns, c["prec"], seed * 137 + i, u, False)
        out.append(run + (steps,))
    return out


def _one(case, seed):
    k = case["kind"]
    if k in ("call_sites", "dam"):
        return _dam(case["nx"], case["ny"], case["ns"], case["prec"], case.get("nrk", 2), seed,
                    case.get("t_end", 1.0e9))
    if k in ("current", "output"):
        return _current(case, seed)
    return _flood(case, seed)


def _host(t):
    """A tensor's values as an FP64 numpy array in page-locked memory."""
    out = torch.empty(t.shape, dtype=torch.float64, pin_memory=DEV == "cuda")
    out.copy_(t)
    return out.numpy().reshape(-1)


def _sflow(P):
    """The library's parameter block."""
    from imex_sflow2d_dev_gb300.params import MAX_VARS, PREC_FP32, PREC_FP64, default_params
    p = default_params()
    p.precision = PREC_FP32 if P["prec"] == 32 else PREC_FP64
    p.comp_cells_x, p.comp_cells_y, p.cell_size, p.n_solid = P["nx"], P["ny"], P["dx"], P["ns"]
    p.gas_flag, p.liquid_flag, p.energy_flag = P["gas"], 1 - P["gas"], P["energy"]
    p.rheology_flag, p.rheology_model, p.mu, p.xi, p.slope_correction_flag = P["rheo"], 1, P["mu"], P["xi"], P["slope"]
    p.grav, p.pres, p.sp_heat_a, p.sp_gas_const_a, p.kin_visc_a, p.T_ambient = GRAV, PRES, CP_AIR, R_AIR, NU_AIR, T_AMB
    p.rho_l, p.sp_heat_l, p.kin_visc_l, p.loss_rate = RHO_L, CP_L, NU_L, 0.0
    for i in range(P["ns"]):
        p.rho_s[i], p.diam_s[i], p.sp_heat_s[i] = P["rho_s"][i], P["diam"][i], P["cp_s"][i]
    for i in range(MAX_VARS):
        p.limiter[i] = P["lim"]
    p.settling_flag, p.entrainment_flag, p.n_rk = P["settling"], P["entrain"], P["nrk"]
    p.cfl, p.dt0, p.max_dt, p.t_start, p.t_end, p.dt_output = P["cfl"], P["dt0"], P["max_dt"], 0.0, P["t_end"], 2 * P["t_end"]
    p.set_bc_all(1, 0.0)
    if P["ring"]:
        s = P["ring"]
        p.radial_source_flag, p.x_source, p.y_source, p.r_source = 1, s["x"], s["y"], s["r"]
        p.mfr_source, p.vel_source, p.T_source = s["mfr"], s["vel"], s["T"]
        for i, a in enumerate(s["alphas"]):
            p.alphas_source[i] = a
    if P["erosion"]:
        e = P["erosion"]
        p.erosion_coeff, p.erodible_porosity, p.T_erodible = e["coeff"], e["porosity"], e["T"]
        p.initial_erodible_thickness, p.topo_change_flag = e["depth"], 1
        for i, f in enumerate(e["fract"]):
            p.erodible_fract[i] = f
    return p


# ---------------------------------------------------------------------------
# passes
# ---------------------------------------------------------------------------

class _Result:
    """Where a run's state comes back to: FP64 in page-locked memory, as the
    entry points write it, and for the FP32 form the FP32 array it is kept
    in."""

    def __init__(self, case, size):
        self.raw = _host(torch.zeros(size))
        self.kept = torch.from_numpy(self.raw) if case["prec"] == 64 else torch.zeros(size, dtype=torch.float32)

    def keep(self):
        if self.kept.dtype == torch.float32:
            self.kept.copy_(torch.from_numpy(self.raw))
        return self.kept


def prepare(case, seed):
    from imex_sflow2d_dev_gb300 import lib, serve
    st = {"case": case}
    if case["kind"] in ("ensemble", "served"):
        runs = _ensemble_runs(case, seed) if case["kind"] == "ensemble" else _served_runs(case, seed)
        jobs = [(_sflow(r[0]), r[1].cpu().numpy().reshape(-1), _host(r[2].permute(1, 2, 0)),
                 r[3] if len(r) > 3 else case["steps"]) for r in runs]
        cells = sum(r[0]["nx"] * r[0]["ny"] for r in runs)
        prec = jobs[0][0].precision
        if case["kind"] == "ensemble":
            st["batch"] = lib.Batch(prec, max_runs=len(jobs), max_cells=2 * cells + 65536)
            st["runs"], st["out"] = jobs, [_Result(case, q.size) for _, _, q, _ in jobs]
        else:
            # eight resident runs at most: the later ones wait for a slot
            st["loop"] = serve.RequestLoop(prec, max_runs=8, max_cells=2 * cells + 65536, keep_results=True)
            st["requests"] = [serve.Request(i, 0.0, p, B, q, n) for i, (p, B, q, n) in enumerate(jobs)]
        return st
    P, B, q = _one(case, seed)
    st["solver"] = lib.Solver(_sflow(P), B.cpu().numpy())
    st["q"] = _host(q.permute(1, 2, 0))
    st["out"] = _Result(case, q.numel())
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    keep = torch.float32 if case["prec"] == 32 else torch.float64
    if kind == "ensemble":
        b = st["batch"]
        ids = b.submit_many(st["runs"])
        b.advance(case["steps"])
        b.collect_many(ids, outs=[r.raw for r in st["out"]])
        return [r.keep() for r in st["out"]]
    if kind == "served":
        return [torch.from_numpy(r["q"]).to(keep) for r in st["loop"].run(st["requests"])]
    s = st["solver"]
    s.upload_q(st["q"])
    if kind == "call_sites":
        t, dt1, dt2 = 0.0, 1.0e-3, 1.0e-3
        for _ in range(case["steps"]):
            s.check_solve()
            dt = min(s.timestep(), 1.1 * 0.5 * (dt1 + dt2))      # the driver's clamps
            s.imex_rk_solver(t, dt)
            s.update_erosion_deposition_cell(dt)
            s.post_step()
            t, dt1, dt2 = t + dt, dt, dt1
    elif "t_end" in case:
        s.advance()
    else:
        s.advance(max_steps=case["steps"])
    s.download_q(st["out"].raw)
    out = {"q": st["out"].keep()}
    if kind == "output":
        out["qp"] = torch.from_numpy(s.download_qp()).to(keep)
        out["hmax"], out["pdynmax"], out["velmax"] = (torch.from_numpy(m).to(keep) for m in s.maps())
        out["deposit"] = torch.from_numpy(s.download_deposit()).to(keep)
    if kind == "flood":
        out["topography"], out["deposit"], out["erosion"] = (
            torch.from_numpy(f()) for f in (s.download_topography, s.download_deposit, s.download_erosion))
    return out


def work(case):
    """State read from and written back to host memory once (FP64), the
    topography read once; the operations of the flowing cells' faces,
    sources and stages."""
    def one(nx, ny, ns, wet, steps, nrk=2):
        nv = 4 + ns
        per_face = 2 * (12 * (nv + 2) + 16 * ns + 60) + 8 * nv
        per_cell = (nrk if nrk > 2 else 1) * (2 * per_face + 12 * nv) + (nrk - 1) * 90 + 60
        return nx * ny * (16.0 * nv + 8.0), float(nx * ny) * wet * steps * per_cell

    k = case["kind"]
    if k in ("ensemble", "served"):
        b = f = 0.0
        for i in range(case["runs"]):
            side = _side(case, i)
            dam = k == "served" and i % 2 == 0
            ns = 2 if k == "ensemble" else 1 + (i // 2) % 3
            wet = 1.0 if dam else 0.04 if case["prec"] == 32 else min(1.0, (40.0 / side) ** 2)
            x, y = one(side, side, ns, wet, case["steps"] * (1.0 if k == "ensemble" else 2.0 / 3.0))
            b, f = b + x, f + y
    else:
        nx, ny = case["nx"], case["ny"]
        wet = 1.0
        if k in ("current", "output"):
            wet = math.pi * (0.5 * case["spread"] * min(nx, ny)) ** 2 / (nx * ny)
        elif k == "flood":
            wet = math.pi * (0.35 * ny) ** 2 / (nx * ny)
        steps = case.get("steps") or case["t_end"] / 0.05
        b, f = one(nx, ny, case.get("ns", 2), wet, steps, case.get("nrk", 2))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the answers in FP64
# ---------------------------------------------------------------------------

def exact(case, seed):
    k = case["kind"]
    if k in ("ensemble", "served"):
        runs = _ensemble_runs(case, seed) if k == "ensemble" else _served_runs(case, seed)
        n = EXACT_MEMBERS if case["steps"] > 32 else len(runs)
        out = []
        for i, r in enumerate(runs):
            if i >= n:
                out.append(None)
                continue
            m = _Model(*r[:3])
            m.advance(r[3] if len(r) > 3 else case["steps"])
            out.append(m.aos(m.q))
        return out
    m = _Model(*_one(case, seed))
    if "t_end" in case:
        m.advance(1 << 30)
    else:
        m.advance(case["steps"])
    out = {"q": m.aos(m.q)}
    if k == "output":
        out["qp"] = m.aos(m.to_phys(m.q)[0])
        out["hmax"], out["pdynmax"], out["velmax"] = (a.reshape(-1) for a in m.maps)
        out["deposit"] = m.deposit.reshape(-1)
    if k == "flood":
        out["topography"], out["deposit"], out["erosion"] = m.B.reshape(-1), m.deposit.reshape(-1), m.erosion.reshape(-1)
    return out


def _quiet(num, den, ok):
    """num / den where ok, else 0."""
    return torch.where(ok, num / torch.where(ok, den, torch.ones_like(den)), torch.zeros_like(num))


class _Model:
    """The step on FP64 tensors.  Fields are (ny, nx); a state is (nv, ny,
    nx).  Cells that the solver leaves out of its active set are dry and
    get no flux, except the cells inside the ring inlet, which it never
    updates."""

    def __init__(self, P, B, q):
        self.P, self.B, self.q = P, B.clone(), q.clone()
        self.ns, self.nv = P["ns"], 4 + P["ns"]
        self.dx = P["dx"]
        self.eps_sing = min(self.dx ** 4, 1.0e-10)
        self.rho_amb = PRES / (R_AIR * T_AMB)
        z = torch.zeros_like(B)
        self.maps = [z.clone(), z.clone(), z.clone()]
        self.deposit = torch.zeros(self.ns, P["ny"], P["nx"], dtype=torch.float64, device=DEV)
        self.erosion = torch.zeros_like(self.deposit)
        e = P["erosion"]
        self.erodible = None
        if e:
            f = torch.tensor([x / sum(e["fract"]) for x in e["fract"]], dtype=torch.float64, device=DEV)
            self.fract = f.view(-1, 1, 1)
            self.erodible = (self.fract * (1.0 - e["porosity"]) * e["depth"]) * torch.ones_like(self.deposit)
        self.exchange = bool(P["settling"] or P["entrain"] or e)
        self.topography()
        self.ring()
        self.t, self.dt1, self.dt2 = 0.0, P["dt0"], P["dt0"]
        qp, pdyn = self.to_phys(self.q)
        self.post(qp, pdyn, self.q[0] > 0)

    def aos(self, a):
        return a.permute(1, 2, 0).reshape(-1).contiguous()

    # geometry ------------------------------------------------------------
    def topography(self):
        """Least-squares slopes and curvatures over 5 x 5 cells; the frame of
        two cells takes its neighbour's."""
        ny, nx, d = self.P["ny"], self.P["nx"], self.dx
        B = self.B
        c1, c2 = (-2.0, -1.0, 0.0, 1.0, 2.0), (2.0, -1.0, -2.0, -1.0, 2.0)
        jj = torch.arange(nx, device=DEV).clamp(2, nx - 3)
        kk = torch.arange(ny, device=DEV).clamp(2, ny - 3)

        def at(dj, dk):
            return B[2 + dk:ny - 2 + dk, 2 + dj:nx - 2 + dj]
        bx = sum(c1[m] * at(m - 2, 0) for m in range(5)) / (10.0 * d)
        by = sum(c1[m] * at(0, m - 2) for m in range(5)) / (10.0 * d)
        bxx = sum(c2[m] * at(m - 2, 0) for m in range(5)) / (7.0 * d * d)
        byy = sum(c2[m] * at(0, m - 2) for m in range(5)) / (7.0 * d * d)
        bxy = sum(c1[m] * c1[n] * at(m - 2, n - 2) for n in range(5) for m in range(5)) / (100.0 * d * d)
        bx, by, bxx, byy, bxy = (a[kk - 2][:, jj - 2] for a in (bx, by, bxx, byy, bxy))
        self.Bx, self.By = bx, by
        if self.P["slope"]:
            self.gc = 1.0 / (1.0 + bx * bx + by * by)
            self.gcx = -2.0 * self.gc ** 2 * (bx * bxx + by * bxy)
            self.gcy = -2.0 * self.gc ** 2 * (bx * bxy + by * byy)
        else:
            self.gc, self.gcx, self.gcy = torch.ones_like(bx), torch.zeros_like(bx), torch.zeros_like(bx)

    def ring(self):
        """The lateral ring inlet: cells inside the circle are left out, the
        cells around it feed the flow through their faces on the circle."""
        ny, nx, d = self.P["ny"], self.P["nx"], self.dx
        face = {f: np.zeros((ny, nx), dtype=bool) for f in "EWNS"}
        inside = np.zeros((ny, nx), dtype=bool)
        s = self.P["ring"]
        self.src = None
        if s:
            st = lambda i: i * d                                           # noqa: E731
            ce = lambda i: 0.5 * (st(i) + st(i + 1))                       # noqa: E731
            r2 = lambda x, y: (x - s["x"]) ** 2 + (y - s["y"]) ** 2        # noqa: E731
            normal = {f: {} for f in "EWNS"}
            R2 = s["r"] ** 2
            j0, j1 = max(1, int((s["x"] - s["r"]) / d) - 2), min(nx - 2, int((s["x"] + s["r"]) / d) + 2)
            k0, k1 = max(1, int((s["y"] - s["r"]) / d) - 2), min(ny - 2, int((s["y"] + s["r"]) / d) + 2)
            kind = {}
            for k in range(k0, k1 + 1):
                for j in range(j0, j1 + 1):
                    if r2(ce(j), ce(k)) > R2:
                        continue
                    kind[(k, j)] = 1
                    if r2(ce(j - 1), ce(k)) >= R2:
                        face["E"][k, j - 1], kind[(k, j - 1)] = True, 2
                        normal["E"][(k, j - 1)] = (st(j) - s["x"], ce(k) - s["y"])
                    elif r2(ce(j + 1), ce(k)) >= R2:
                        face["W"][k, j + 1], kind[(k, j + 1)] = True, 2
                        normal["W"][(k, j + 1)] = (st(j + 1) - s["x"], ce(k) - s["y"])
                    if r2(ce(j), ce(k - 1)) >= R2:
                        face["N"][k - 1, j], kind[(k - 1, j)] = True, 2
                        normal["N"][(k - 1, j)] = (ce(j) - s["x"], st(k) - s["y"])
                    elif r2(ce(j), ce(k + 1)) >= R2:
                        face["S"][k + 1, j], kind[(k + 1, j)] = True, 2
                        normal["S"][(k + 1, j)] = (ce(j) - s["x"], st(k + 1) - s["y"])
            perim, nxv, nyv = (np.zeros((ny, nx)) for _ in range(3))
            for (k, j), v in kind.items():
                if v == 1:
                    inside[k, j] = True
                    continue
                for f in "EWNS":
                    if (k, j) in normal[f]:
                        a, b = normal[f][(k, j)]
                        m = math.hypot(a, b)
                        if m > 0.0:
                            perim[k, j] += d
                            nxv[k, j] += d * a / m
                            nyv[k, j] += d * b / m
                m = math.hypot(nxv[k, j], nyv[k, j])
                if perim[k, j] > 0.0 and m > 0.0:
                    nxv[k, j], nyv[k, j] = nxv[k, j] / m, nyv[k, j] / m
            length = math.pi * 2.0 * s["r"]
            perim *= length / perim.sum()
            at = sum(s["alphas"])
            rho_c = PRES / (R_AIR * s["T"])
            rho_m = (1.0 - at) * rho_c + sum(a * r for a, r in zip(s["alphas"], self.P["rho_s"]))
            xs = [a * r / rho_m for a, r in zip(s["alphas"], self.P["rho_s"])]
            cm = sum(x * c for x, c in zip(xs, self.P["cp_s"])) + (1.0 - sum(xs)) * CP_AIR
            h_in = s["mfr"] / (length * rho_m * s["vel"])
            hd = torch.from_numpy(h_in * s["vel"] * perim / (d * d)).to(DEV)
            self.src = torch.stack([hd * rho_m, hd * rho_m * s["vel"] * torch.from_numpy(nxv).to(DEV),
                                    hd * rho_m * s["vel"] * torch.from_numpy(nyv).to(DEV), hd * rho_m * cm * s["T"]] +
                                   [hd * a * r for a, r in zip(s["alphas"], self.P["rho_s"])])
        self.face = {f: torch.from_numpy(a).to(DEV) for f, a in face.items()}
        self.inside = torch.from_numpy(inside).to(DEV)

    # closures --------------------------------------------------------------
    def to_phys(self, q):
        """h, hu, hv, T, h alpha_s, u, v and the dynamic pressure."""
        P, ns = self.P, self.ns
        wet = q[0] > EPS
        inv = _quiet(torch.ones_like(q[0]), q[0], wet)
        xs = q[4:] * inv
        tot = q[4:].sum(0)
        full = wet & (tot == q[0])
        xs = torch.where(full, _quiet(xs, xs.sum(0).expand_as(xs), full.expand_as(xs)), xs)
        xc = 1.0 - xs.sum(0)
        cm = sum(xs[i] * P["cp_s"][i] for i in range(ns)) + xc * (CP_AIR if P["gas"] else CP_L)
        e = q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) * inv if P["energy"] else q[3]
        T = _quiet(e, q[0] * cm, wet)
        T = torch.where((T <= 0) | (q[0] <= self.eps_sing), torch.full_like(T, T_AMB), T)
        inv_c = R_AIR * T / PRES if P["gas"] else torch.full_like(T, 1.0 / RHO_L)
        inv_m = sum(xs[i] / P["rho_s"][i] for i in range(ns)) + xc * inv_c
        rho_m = 1.0 / inv_m
        film = wet & (q[0] <= self.eps_sing)
        den = torch.sqrt(q[0] ** 4 + self.eps_sing ** 4)
        u = torch.where(film, math.sqrt(2.0) * q[0] * q[1] / den, q[1] * inv)
        v = torch.where(film, math.sqrt(2.0) * q[0] * q[2] / den, q[2] * inv)
        h = q[0] * inv_m
        al = [xs[i] * rho_m / P["rho_s"][i] for i in range(ns)]
        qp = torch.stack([h, h * u, h * v, T] + [a * h for a in al] + [u, v])
        dry = torch.zeros_like(qp)
        dry[3] = T_AMB
        qp = torch.where(wet, qp, dry)
        return qp, torch.where(wet, 0.5 * rho_m * (u * u + v * v), torch.zeros_like(u))

    def mixture(self, qp):
        """Volume fractions, carrier and mixture density, reduced gravity."""
        ok = qp[0] > EPS
        al = _quiet(qp[4:4 + self.ns], qp[0].expand_as(qp[4:4 + self.ns]), ok.expand_as(qp[4:4 + self.ns]))
        at = al.sum(0)
        rho_c = PRES / (R_AIR * qp[3]) if self.P["gas"] else torch.full_like(at, RHO_L)
        rho_m = (1.0 - at) * rho_c + sum(al[i] * self.P["rho_s"][i] for i in range(self.ns))
        return ok, al, rho_c, rho_m, (rho_m - self.rho_amb) / rho_m * GRAV

    # fluxes ------------------------------------------------------------------
    def limited(self, a, b):
        """Limited slope from the forward and backward slopes (uniform cells)."""
        def minmod(x, y):
            return torch.where(x * y > 0, torch.sign(x) * torch.minimum(x.abs(), y.abs()), torch.zeros_like(x))
        m = minmod(a, b)
        return m if self.P["lim"] == 1 else minmod(0.5 * (a + b), m)      # theta = 1

    def faces(self, qp, n_axis):
        """Reconstructed states below and above every face along x (axis 0)
        or y (axis 1); fields turned so that the direction is the last."""
        nv, d = self.nv, self.dx
        mom = 1 + n_axis
        turn = (lambda a: a) if n_axis == 0 else (lambda a: a.transpose(-1, -2))
        w = turn(qp)
        hi_f, lo_f = turn(self.face["E" if n_axis == 0 else "N"]), turn(self.face["W" if n_axis == 0 else "S"])
        use_hi = hi_f if n_axis == 0 else hi_f & ~lo_f
        use_lo = lo_f & ~hi_f if n_axis == 0 else lo_f
        diff = (w[..., 1:] - w[..., :-1]) / d
        sl = torch.zeros_like(w)
        sl[..., 1:-1] = self.limited(diff[..., 1:], diff[..., :-1])
        if n_axis == 0 and self.P["ring"]:
            # ring cells with a face to the north only: the solver's x slope
            # of v takes the cell's upper y edge for its eastern neighbour
            odd = self.face["N"] & ~self.face["S"] & ~self.face["E"] & ~self.face["W"]
            ks, js = torch.nonzero(odd, as_tuple=True)
            if ks.numel():
                v = w[nv + 1]
                b = (v[ks, js] - v[ks, js - 1]) / d
                a = (v[ks, js + 1] - v[ks, js]) / ((ks + 1) * d - (js + 0.5) * d)
                sl[nv + 1][ks, js] = torch.where(a * b > 0, torch.sign(a) * torch.minimum(a.abs(), b.abs()),
                                                 torch.zeros_like(a))
        sl = torch.where(use_hi | use_lo, torch.zeros_like(sl), sl)
        lo, hi = w - 0.5 * d * sl, w + 0.5 * d * sl
        # domain edges: zero gradient, no inflow through the edge; the
        # velocities of the edge cells take the edge state as a neighbour
        for e, side, cap in ((0, lo, torch.clamp_max), (-1, hi, torch.clamp_min)):
            edge = w[:nv, ..., e].clone()
            edge[mom] = cap(edge[mom], 0.0)
            uv = _quiet(edge[1:3], edge[0].expand(2, -1), (edge[0] > 0).expand(2, -1))
            c = w[nv:, ..., e]
            nb = w[nv:, ..., 1 if e == 0 else -2]
            inner, outer = (nb - c) / d, (c - uv) / (0.5 * d)
            if e == -1:
                inner, outer = (c - nb) / d, (uv - c) / (0.5 * d)
            if self.P["lim"] == 1:
                s = self.limited(inner, outer)
            else:
                m = torch.where(inner * outer > 0, torch.sign(inner) * torch.minimum(inner.abs(), outer.abs()),
                                torch.zeros_like(inner))
                cen = (nb - uv) / (1.5 * d) if e == 0 else (uv - nb) / (1.5 * d)
                s = torch.where(cen * m > 0, torch.sign(m) * torch.minimum(cen.abs(), m.abs()), torch.zeros_like(m))
            other = hi if e == 0 else lo
            other[nv:, ..., e] = c + (0.5 if e == 0 else -0.5) * d * s
            side[:nv, ..., e] = edge
            side[nv:, ..., e] = uv
        L = torch.cat([lo[..., :1], hi], -1)
        H = torch.cat([lo, hi[..., -1:]], -1)
        # wall mirror at the faces of the ring inlet
        pad = torch.zeros_like(hi_f[..., :1])
        mir_h = torch.cat([pad, use_hi], -1)
        mir_l = torch.cat([use_lo, pad], -1) & ~mir_h
        Lm, Hm = torch.where(mir_l, H, L), torch.where(mir_h, L, H)
        Lm[nv + n_axis] = torch.where(mir_l, -Lm[nv + n_axis], Lm[nv + n_axis])
        Hm[nv + n_axis] = torch.where(mir_h, -Hm[nv + n_axis], Hm[nv + n_axis])
        g = turn(self.gc)
        gf = torch.cat([g[..., :1], 0.5 * (g[..., 1:] + g[..., :-1]), g[..., -1:]], -1)
        return Lm, Hm, mir_l, mir_h, gf

    def side(self, qp, mirrored, gf, n_axis):
        P, nv, ns = self.P, self.nv, self.ns
        ok, al, rho_c, rho_m, rg = self.mixture(qp)
        xc = (1.0 - al.sum(0)) * rho_c / rho_m
        cm = sum(al[i] * P["rho_s"][i] / rho_m * P["cp_s"][i] for i in range(ns)) + xc * (CP_AIR if P["gas"] else CP_L)
        h, u, v = qp[0], qp[nv], qp[nv + 1]
        e = cm * qp[3] + (0.5 * (u * u + v * v) if P["energy"] else 0.0)
        qc = torch.stack([rho_m * h, rho_m * qp[1], rho_m * qp[2], h * rho_m * e] +
                         [al[i] * P["rho_s"][i] * h for i in range(ns)])
        zero = torch.zeros_like(qc)
        qc = torch.where(ok, qc, zero)
        rg = torch.where(ok, rg, zero[0])
        qc[1 + n_axis] = torch.where(mirrored, -qc[1 + n_axis], qc[1 + n_axis])
        vel = qp[nv + n_axis]
        c = torch.sqrt((rg * h * gf).clamp_min(0.0))
        p = 0.5 * rho_m * gf * rg * h * h
        f = vel * qc
        f[1 + n_axis] += p
        if P["energy"]:
            f[3] += vel * p
        s = f[4:].sum(0)
        over = (f[0] > 0) & (s > f[0])
        f[4:] = torch.where(over, f[4:] * _quiet(f[0], s, over), f[4:])
        f = torch.where(ok, f, zero)
        return qc, f, vel - c, vel + c

    def flux(self, qp, n_axis):
        nv = self.nv
        L, H, ml, mh, gf = self.faces(qp, n_axis)
        ql, fl, l1, l2 = self.side(L, ml, gf, n_axis)
        qh, fh, h1, h2 = self.side(H, mh, gf, n_axis)
        a1 = torch.minimum(l1, h1).clamp_max(0.0)
        a2 = torch.maximum(l2, h2).clamp_min(0.0)
        move = a1 != a2
        F = _quiet(a2 * fl - a1 * fh + a1 * a2 * (qh - ql), (a2 - a1).expand_as(fl), move.expand_as(fl))
        s = F[4:].sum(0)
        r = _quiet(s, F[0], F[0] != 0)
        over = r >= 1.0 if n_axis == 0 else r > 1.0
        F[4:] = torch.where(over, F[4:] / torch.where(over, r, torch.ones_like(r)), F[4:])
        still = (L[1] == 0) & (H[1] == 0) if n_axis == 0 else (ql[2] == 0) & (qh[2] == 0)
        keep = torch.ones(nv, 1, 1, dtype=torch.bool, device=DEV)
        keep[0] = keep[3:] = False
        F = torch.where(still & ~keep, torch.zeros_like(F), F)
        # a cell inside the ring takes part in no face
        amax = torch.maximum(a2, -a1)
        turn = (lambda a: a) if n_axis == 0 else (lambda a: a.transpose(-1, -2))
        ins = turn(self.inside)
        pad = torch.zeros_like(ins[..., :1])
        none = torch.cat([pad, ins], -1) & torch.cat([ins, pad], -1)
        amax = torch.where(none, torch.zeros_like(amax), amax)
        div = (F[..., 1:] - F[..., :-1]) / self.dx
        return turn(div), float(amax.max())

    def rate(self, q):
        """Divergence of the fluxes minus the explicit sources; the largest
        signal speeds along x and y."""
        qp, _ = self.to_phys(q)
        dx_, ax = self.flux(qp, 0)
        dy_, ay = self.flux(qp, 1)
        r = dx_ + dy_
        ok, _, _, rho_m, rg = self.mixture(qp)
        h = qp[0]
        zero = torch.zeros_like(h)
        e1 = torch.where(ok, -self.gc * rho_m * rg * h * self.Bx + 0.5 * rho_m * rg * h * h * self.gcx, zero)
        e2 = torch.where(ok, -self.gc * rho_m * rg * h * self.By + 0.5 * rho_m * rg * h * h * self.gcy, zero)
        r[1] -= e1
        r[2] -= e2
        if self.P["energy"]:
            r[3] -= e1 * qp[self.nv] + e2 * qp[self.nv + 1]
        if self.src is not None:
            r = r - self.src
        return torch.where(self.inside, torch.zeros_like(r), r), ax, ay

    # implicit stage ------------------------------------------------------------
    def friction(self, qf, dta):
        """Coulomb friction of the state qf, then the turbulent friction
        solved to convergence along the momentum; returns the stage state
        and (stage state - qf) / dta."""
        P, nv = self.P, self.nv
        if not P["rheo"]:
            return qf, torch.zeros_like(qf)
        wet = qf[0] > 0
        qp, _ = self.to_phys(qf)
        ok, _, _, rho_m, rg = self.mixture(qp)
        u, v = qp[nv], qp[nv + 1]
        w = u * self.Bx + v * self.By if P["slope"] else torch.zeros_like(u)
        mod = torch.sqrt(u * u + v * v + w * w)
        tt = torch.where(ok, (P["mu"] * rho_m * rg * qp[0] * torch.sqrt(self.gc)).clamp_min(0.0), torch.zeros_like(u))
        s1 = qf[1] - dta * _quiet(tt * u, mod, mod > 0)
        s2 = qf[2] - dta * _quiet(tt * v, mod, mod > 0)
        m0 = torch.sqrt(qf[1] ** 2 + qf[2] ** 2)
        rest = (m0 == 0) | (s1 * qf[1] < 0) | (s2 * qf[2] < 0)
        S = torch.where(rest, torch.zeros_like(m0), torch.sqrt(s1 * s1 + s2 * s2))
        e1, e2 = _quiet(qf[1], m0, m0 > 0), _quiet(qf[2], m0, m0 > 0)
        # s + dta K(s) s^2 = S by Newton, K = (rho_m(s) - rho_amb) g kappa phi^2 / xi
        q0 = torch.where(qf[0] > EPS, qf[0], torch.ones_like(qf[0]))
        inv = 1.0 / q0
        xs = qf[4:] * inv
        xc = 1.0 - xs.sum(0)
        cm = sum(xs[i] * P["cp_s"][i] for i in range(self.ns)) + xc * (CP_AIR if P["gas"] else CP_L)
        film = qf[0] <= self.eps_sing
        phi = torch.where(film, math.sqrt(2.0) * q0 / torch.sqrt(q0 ** 4 + self.eps_sing ** 4), inv)
        kap2 = 1.0 + (e1 * self.Bx + e2 * self.By) ** 2 if P["slope"] else torch.ones_like(phi)
        geo = GRAV * torch.sqrt(kap2) * phi * phi / P["xi"]
        base = sum(xs[i] / P["rho_s"][i] for i in range(self.ns))
        s = S.clone()
        for _ in range(30):
            T = qf[3] / (q0 * cm)
            dT = torch.zeros_like(T)
            if P["energy"]:
                T = T - 0.5 * s * s * inv / (q0 * cm)
                dT = -s * inv / (q0 * cm)
            low = (T <= 0) | film
            T = torch.where(low, torch.full_like(T, T_AMB), T)
            dT = torch.where(low, torch.zeros_like(dT), dT)
            cT = xc * R_AIR / PRES if P["gas"] else torch.zeros_like(T)
            rho = 1.0 / (base + (cT * T if P["gas"] else xc / RHO_L))
            K = geo * (rho - self.rho_amb)
            dK = -geo * rho * rho * cT * dT
            step = (s + dta * K * s * s - S) / (1.0 + dta * (dK * s * s + 2.0 * K * s))
            s = (s - step).clamp_min(0.0)
        go = wet & (qf[0] > EPS)
        out = qf.clone()
        out[1] = torch.where(wet, torch.where(go, s, S) * e1, qf[1])
        out[2] = torch.where(wet, torch.where(go, s, S) * e2, qf[2])
        return out, (out - qf) / dta

    def fixes(self, q):
        """Positivity after the assembly."""
        q = torch.where((q[0] < EPS) & (q[0] > -1.0e-7), torch.zeros_like(q), q)
        neg = (q[4:] < 0).any(0)
        q[4:] = torch.where(neg, torch.zeros_like(q[4:]), q[4:])
        s = q[4:].sum(0)
        over = s > q[0]
        q[4:] = torch.where(over, q[4:] * _quiet(q[0], s, over), q[4:])
        return q

    def settle(self, i, rho_c):
        """Terminal velocity of class i: fixed point on the drag law, left
        at a relative change below 1e-6."""
        P = self.P
        nu = NU_AIR if P["gas"] else NU_L
        const = torch.sqrt((4.0 / 3.0 * (P["rho_s"][i] / rho_c - 1.0) * P["diam"][i] * GRAV).clamp_min(0.0))
        sv = const.clone()
        Re = P["diam"][i] * sv / nu
        live = (Re <= 1000.0) & (const > 0)
        for _ in range(20):
            old = sv
            Rs = torch.where(live, Re, torch.ones_like(Re))
            new = const * torch.sqrt(Rs / (24.0 * (1.0 + 0.15 * Rs ** 0.687)))
            sv = torch.where(live, new, sv)
            Re = P["diam"][i] * sv / nu
            live = live & ((old - sv).abs() >= 1.0e-6 * old)
        return sv

    def mass_exchange(self, q, dt):
        """Deposition, erosion and entrainment of air; lift-off of what has
        become lighter than the air."""
        P, ns, nv = self.P, self.ns, self.nv
        qp, _ = self.to_phys(q)
        ok, al, rho_c, rho_m, rg = self.mixture(qp)
        h, u, v, T = qp[0], qp[nv], qp[nv + 1], qp[3]
        at = al.sum(0)
        w = u * self.Bx + v * self.By if P["slope"] else torch.zeros_like(u)
        v2 = u * u + v * v + w * w
        zero = torch.zeros_like(u)
        e = P["erosion"]
        por = e["porosity"] if e else 0.0
        ers = torch.zeros_like(al)
        if e:
            tot = e["coeff"] * torch.sqrt(v2) * h * (1.0 - at) * (1.0 - por)
            ers = torch.minimum(self.fract * tot, self.erodible / dt).clamp_min(0.0)
            ers = torch.where(ok, ers, torch.zeros_like(ers))
        live = ok & (at > 0.0)
        dep = torch.zeros_like(al)
        if P["settling"]:
            hind = (1.0 - (at / 0.6).clamp_max(1.0)) ** 4.65
            for i in range(ns):
                d = torch.minimum(al[i] * self.settle(i, rho_c) * hind, h * al[i] / dt)
                dep[i] = torch.where(live & (al[i] > 0), d, zero)
        cp = por / (1.0 - por)
        sd = dep.sum(0)
        cpl = torch.minimum(cp * sd, h * (0.64 - at).clamp_min(0.0) / dt)
        cpl = torch.minimum(cpl, (h * (1.0 - at) - cp * (h * at - dt * sd)) / dt)
        air = zero
        if P["entrain"]:
            Ri = torch.where(v2 > 0, _quiet(rg * h, u * u + v * v, u * u + v * v > 0).clamp_max(1.0e15), zero)
            up = ok & (h > 0) & (Ri > 0)
            air = torch.where(up, 0.075 / torch.sqrt(1.0 + 718.0 * Ri.clamp_min(0.0) ** 2.4) * torch.sqrt(v2), zero)
        rs = torch.tensor(P["rho_s"], dtype=torch.float64, device=DEV).view(-1, 1, 1)
        cs = torch.tensor(P["cp_s"], dtype=torch.float64, device=DEV).view(-1, 1, 1)
        rd, re, sdp, ser = (rs * dep).sum(0), (rs * ers).sum(0), (rs * cs * dep).sum(0), (rs * cs * ers).sum(0)
        cont = ers.sum(0) / (1.0 - por) * por
        Te = e["T"] if e else 300.0
        rho_sub = PRES / (R_AIR * Te) if P["gas"] else RHO_L
        cpc = CP_AIR if P["gas"] else CP_L
        out = rd + rho_c * cpl
        heat = -T * (sdp + rho_c * cpc * cpl) + Te * (ser + rho_sub * cpc * cont) + T_AMB * CP_AIR * self.rho_amb * air
        if P["energy"]:
            heat = heat - 0.5 * v2 * out
        eq = torch.stack([self.rho_amb * air + re - rd + rho_sub * cont - rho_c * cpl, -u * out, -v * out, heat] +
                         [P["rho_s"][i] * (ers[i] - dep[i]) for i in range(ns)])
        eq = torch.where(live, eq, torch.zeros_like(eq))
        q = q + dt * eq
        q[4:] = q[4:].clamp_min(0.0)
        q = torch.where(q[0] > 0, q, torch.zeros_like(q))
        s = q[4:].sum(0)
        over = (s > q[0]) & (q[0] < 1.0e-10)
        q[4:] = torch.where(over, q[4:] * _quiet(q[0], s, over), q[4:])
        qp, _ = self.to_phys(q)
        ok, _, _, _, rg = self.mixture(qp)
        q = torch.where(ok & (rg > 0), q, torch.zeros_like(q))
        self.deposit += dt * dep
        if e:
            self.erosion += dt * ers
            self.erodible -= dt * ers
            self.B = self.B + dt * torch.where(live, (dep.sum(0) - ers.sum(0)) / (1.0 - por), zero)
            self.topography()
        return q

    def post(self, qp, pdyn, wet):
        h, vel = qp[0], torch.sqrt(qp[self.nv] ** 2 + qp[self.nv + 1] ** 2)
        thick = wet & (h > 1.0e-3)
        for m, a, on in zip(range(3), (h, pdyn, vel), (wet, thick, thick)):
            self.maps[m] = torch.where(on, torch.maximum(self.maps[m], a), self.maps[m])

    def advance(self, steps):
        P = self.P
        for _ in range(steps):
            if not self.t < P["t_end"]:
                return
            q0 = self.q
            r0, ax, ay = self.rate(q0)
            dt = P["max_dt"]
            for a in (ax, ay):
                if a > 0.0:
                    dt = min(dt, P["cfl"] * self.dx / a)
            if self.t + dt > P["t_end"]:
                dt = P["t_end"] - self.t
            dt = min(dt, 1.1 * 0.5 * (self.dt1 + self.dt2))
            self.dt1, self.dt2, self.t = dt, self.dt1, self.t + dt
            if P["nrk"] == 2:
                q, _ = self.friction(q0 - dt * r0, dt)
            else:
                third = 1.0 / 3.0
                k1, i1 = self.friction(q0, 0.25 * dt)
                r1, _, _ = self.rate(k1)
                k2, i2 = self.friction(q0 - dt * 0.5 * r1, 0.25 * dt)
                r2, _, _ = self.rate(k2)
                k3, i3 = self.friction(q0 - dt * (0.5 * (r1 + r2) - third * (i1 + i2)), third * dt)
                r3, _, _ = self.rate(k3)
                q = q0 - dt * third * (r1 + r2 + r3 - i1 - i2 - i3)
            q = torch.where(self.inside, q0, self.fixes(q))
            if self.exchange:
                q = self.mass_exchange(q, dt)
            self.q = q
            qp, pdyn = self.to_phys(q)
            self.post(qp, pdyn, q[0] > 0)
