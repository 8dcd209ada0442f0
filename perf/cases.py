"""Workloads whose speed matters, each through the calls that a user's program makes.

Four kinds of call:
  noalloc   sv_timestep_noalloc: one FP64 timestep on device buffers that the caller owns
  timestep  SaintVenantSolver.do_timestep: one timestep of a host-controlled loop
  step      SaintVenantSolver.advance: a forecast cycle -- the analysis state goes in, one step
            with device-controlled dt is run, the new state comes out (pinned host arrays)
  batch     SaintVenantBatch.advance_steps: the same for many uneven catchments at once

The fields of an FP32 solver cross the interface as FP64 and are kept in FP32, as checkpoints
keep them. Sites (all seeded, made on the GPU):
  flood  a floodplain under 0.3-2 m of moving water with dry building blocks, land classes of
         roughness, rain on the streets, inflow and outflow depths on the x edges
  rain   a fractal hillside under a film of millimetres with ponds, rain, outflow on all edges;
         dt adapts, rejected timesteps included
  plane  the 256 x 256 tilted plane with Gaussian bumps at other sizes too, a film, rain, outflow
         on the lower x edge; dt adapts
  dam    a dam break over a flat bed at 350 m into shallow water, frictionless, walls
"""
import ctypes
import math
import random

import numpy as np
import torch

import mfcm_b200 as mf
from mfcm_b200.batch import SaintVenantBatch

G = 9.81
MM_PER_H = 1.0 / 3.6e6
CN = 0.5
LAND = (0.02, 0.035, 0.05, 0.1)
EDGES = {"flood": mf.EDGE_XMIN | mf.EDGE_XMAX, "rain": 15, "plane": mf.EDGE_XMAX, "dam": 0}
HEAD = {"flood": 1.0, "rain": 0.0, "plane": 0.0, "dam": 0.0}
# dt per metre of cell size: the fixed timestep (flood, dam: clamped below the CFL limit) or
# the first one (rain, plane: adapted from there)
DT = {"flood": 0.035, "rain": 0.1, "plane": 0.3, "dam": 0.045}
FIXED = ("flood", "dam")
TERM_FIELDS = ("ELOSS_FX", "ELOSS_FY", "INFIL_RATE", "INFIL_CAP")


def _case(name, kind, site, precision, nx, ny, dx, **kw):
    c = dict(name=name, kind=kind, site=site, precision=precision, nx=nx, ny=ny, dx=dx, rk="classic", steps=1,
             tuned=False, terms="")
    c.update(kw)
    return c


def _batch(name, precision, site, persistent, members, side_min, side_max, steps, calls, sizes):
    return dict(name=name, kind="batch", site=site, precision=precision, persistent=persistent, members=members,
                side_min=side_min, side_max=side_max, steps=steps, calls=calls, sizes=sizes)


def listed():
    return [
        # the smallest call: a coupled model's real-time loop on its own buffers
        _case("noalloc_f64_64x48", "noalloc", "flood", "f64", 64, 48, 2.0),
        # a host program that controls dt itself, odd sizes
        _case("timestep_f64_251x187", "timestep", "rain", "f64", 251, 187, 3.0),
        # the small catchment of the benchmark configurations, as it comes (no tuning call)
        _case("step_f64_plane_256", "step", "plane", "f64", 256, 256, 5.0, steps=16),
        # rain on a large catchment in plain FP64, tuned once as a long run is
        _case("step_f64_rain_2048", "step", "rain", "f64", 2048, 2048, 2.0, steps=16, tuned=True),
        # the headline: the 4096 x 4096 catchment in FP32 with FP64 bed datums, tuned once
        _case("step_f32d_flood_4096", "step", "flood", "f32_datum64", 4096, 4096, 2.0, steps=40, tuned=True),
        # an ordinary FP32 run on a ragged mesh, as it comes
        _case("step_f32_flood_1531x967", "step", "flood", "f32", 1531, 967, 3.0, steps=24),
        # the wet/dry-front study's mesh, frictionless, as it comes
        _case("step_f32d_dam_8192x1024", "step", "dam", "f32_datum64", 8192, 1024, 0.5, steps=24),
        # every further source term with a tableau that stores its stage derivatives
        _case("step_f64_terms_601x433", "step", "flood", "f64", 601, 433, 4.0, rk="ssprk3", steps=16, terms="all"),
        # eddy viscosity in FP32 on a mid-size mesh
        _case("step_f32_eddy_1200x900", "step", "flood", "f32", 1200, 900, 2.0, steps=24, terms="eddy"),
        # the ensemble: uneven catchments in one persistent launch
        _batch("batch_f32d_persistent_16", "f32_datum64", "flood", True, 16, 256, 1280, 16, 2, 11),
        # the server's default: FP32 catchments in one launch per stage
        _batch("batch_f32_stages_12", "f32", "flood", False, 12, 128, 1024, 12, 2, 12),
        # the plain-FP64 ensemble, its members at their own dt
        _batch("batch_f64_stages_8", "f64", "rain", False, 8, 128, 768, 8, 2, 13),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "timestep", "step", "step", "step", "step", "batch", "batch"])
    if kind == "noalloc":
        nx = _log(rng, 24, 256)
        c = _case("", kind, "flood", "f64", nx, _log(rng, 24, 256), rng.choice([1.0, 2.0, 3.0, 5.0]),
                  rk=rng.choice(["euler", "heun2", "ralston3", "classic"]))
    elif kind == "timestep":
        c = _case("", kind, "rain", "f64", _log(rng, 48, 700), _log(rng, 48, 700), rng.choice([1.0, 2.0, 3.0, 5.0]),
                  rk=rng.choice(["midpoint", "classic", "ssprk3", "3/8rule"]))
    elif kind == "step":
        precision = rng.choice(["f64", "f32", "f32_datum64"])
        site = rng.choice(["plane", "rain", "flood"]) if precision == "f64" else rng.choice(["flood", "flood", "dam"])
        hi = 1800 if precision == "f64" else 2600
        terms = rng.choice(["", "", "eddy", "all"]) if site == "flood" and precision != "f32_datum64" else ""
        c = _case("", kind, site, precision, _log(rng, 96, hi), _log(rng, 96, hi),
                  rng.choice([0.5, 1.0, 2.0, 3.0, 5.0]) if site != "plane" else 5.0,
                  steps=rng.randint(8, 24), tuned=rng.random() < 0.4, terms=terms,
                  rk=rng.choice(["classic", "classic", "heun3", "ssprk3"]))
    else:
        precision = rng.choice(["f64", "f32", "f32_datum64"])
        c = _batch("", precision, "rain" if precision == "f64" else "flood", rng.random() < 0.5, rng.randint(4, 16),
                   rng.choice([96, 128, 256]), rng.choice([640, 1024]), rng.randint(6, 14), 2, rng.randrange(10 ** 6))
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _smooth(nx, ny, length, gen):
    """Smooth noise of unit size: normal values on a grid `length` cells wide, interpolated."""
    w, h = max(4, int(nx / length) + 3), max(4, int(ny / length) + 3)
    a = torch.randn((1, 1, h, w), generator=gen, device="cuda", dtype=torch.float64)
    return torch.nn.functional.interpolate(a, size=(ny, nx), mode="bicubic", align_corners=True)[0, 0]


def _fractal(nx, ny, gen, hurst=0.8, coarse=256):
    """Sum of octaves of smooth noise, amplitude ~ length^hurst, unit size at the coarsest."""
    z, length = 0.0, min(coarse, max(nx, ny) / 3.0)
    top = length
    while length >= 2.0:
        z = z + (length / top) ** hurst * _smooth(nx, ny, length, gen)
        length /= 2.0
    return z


def _sizes(case):
    """Mesh sizes and cell size of a batch's members: sides log-uniform, any parity."""
    rng = random.Random(case["sizes"])
    lo, hi = case["side_min"], case["side_max"]
    return [(_log(rng, lo, hi), _log(rng, lo, hi), rng.choice([1.0, 2.0, 3.0, 5.0])) for _ in range(case["members"])]


def _site(site, nx, ny, dx, terms, seed):
    """Fields of a site as FP64 tensors on the GPU (bed, state, roughness, rain, further terms)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    y, x = torch.meshgrid(torch.arange(ny, device="cuda", dtype=torch.float64),
                          torch.arange(nx, device="cuda", dtype=torch.float64), indexing="ij")
    f = {}
    if site == "flood":
        bed = 0.6 * torch.tanh(_fractal(nx, ny, gen) / 1.5)
        f["Z"] = 35.0 + 0.0005 * dx * (nx - x) + bed
        f["H"] = 1.1 - bed + 0.05 * _smooth(nx, ny, 40, gen)
        f["U"] = 0.5 + 0.2 * _smooth(nx, ny, 48, gen)
        f["V"] = 0.2 * _smooth(nx, ny, 48, gen)
        # building blocks of 10 x 8 cells on a 26 x 22 lattice, two thirds of the lots built on
        lots = torch.rand((ny // 22 + 1, nx // 26 + 1), generator=gen, device="cuda") < 0.66
        built = lots[(y // 22).long(), (x // 26).long()] & (x % 26 >= 8) & (x % 26 < 18) & (y % 22 >= 7) & (y % 22 < 15)
        built &= (x >= 4) & (x < nx - 4) & (y >= 4) & (y < ny - 4)
        f["Z"] = torch.where(built, f["Z"] + 6.0, f["Z"])
        for k in "HUV":
            f[k] = torch.where(built, torch.zeros_like(x), f[k])
        f["RAIN_PATTERN"] = torch.where(built, torch.zeros_like(x),
                                        30.0 * MM_PER_H * torch.exp(0.3 * _smooth(nx, ny, 100, gen)))
    elif site == "rain":
        relief = _fractal(nx, ny, gen, coarse=512)
        f["Z"] = 100.0 + 0.005 * dx * (nx - x) + 0.02 * dx * min(512.0, max(nx, ny) / 3.0) * relief / 3.0
        pond = torch.clamp(-1.2 - relief, min=0.0)  # the lowest hollows hold up to half a metre
        f["H"] = 2e-3 * (1.0 + 0.4 * torch.rand((ny, nx), generator=gen, device="cuda", dtype=torch.float64))
        f["H"] = f["H"] + torch.clamp(pond, max=0.5)
        f["U"] = 0.02 * _smooth(nx, ny, 12, gen)
        f["V"] = 0.02 * _smooth(nx, ny, 12, gen)
        f["RAIN_PATTERN"] = 30.0 * MM_PER_H * torch.exp(0.5 * _smooth(nx, ny, 100, gen))
    elif site == "plane":
        f["Z"] = 0.01 * dx * (nx - x)
        for _ in range(8):
            a, s, cx, cy = (float(v) for v in torch.rand(4, generator=gen, device="cuda", dtype=torch.float64))
            s = 20.0 + 40.0 * s
            f["Z"] = f["Z"] + 2.0 * a * torch.exp(-((dx * (x - cx * nx)) ** 2 + (dx * (y - cy * ny)) ** 2) / (2 * s * s))
        f["H"] = 1e-3 * (1.0 + 0.2 * _smooth(nx, ny, 20, gen).clamp(-2, 2))
        f["U"] = 0.005 * _smooth(nx, ny, 20, gen)
        f["V"] = 0.005 * _smooth(nx, ny, 20, gen)
    else:
        f["Z"] = torch.full_like(x, 350.0)
        level = 1.0 + 0.05 * float(torch.rand(1, generator=gen, device="cuda"))
        f["H"] = torch.where(x < nx // 2, torch.full_like(x, level), torch.full_like(x, 0.1))
        f["U"] = torch.zeros_like(x)
        f["V"] = torch.zeros_like(x)
    if site in ("flood", "rain"):
        land = torch.tensor(LAND, device="cuda", dtype=torch.float64)
        cls = torch.bucketize(_smooth(nx, ny, 64, gen), torch.tensor([-0.5, 0.0, 0.5], device="cuda", dtype=torch.float64))
        f["N_SHALLOW"] = land[cls]
    if terms == "all":
        for k in ("ELOSS_FX", "ELOSS_FY"):
            f[k] = 0.1 * torch.rand((ny, nx), generator=gen, device="cuda", dtype=torch.float64)
        f["INFIL_RATE"] = torch.full_like(x, 2e-6)
        f["INFIL_CAP"] = 1e-5 * torch.rand((ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    return f


def _pinned(ny, nx, values=None):
    t = torch.empty((ny, nx), dtype=torch.float64, pin_memory=True)
    if values is not None:
        t.copy_(values)
    return t.numpy()


def _params(case):
    """Scheme parameters shared by every kind of call and by the 64-bit evaluation."""
    site, dx = case["site"], case["dx"]
    dt = DT[site] * dx
    steps = case.get("steps", 1)
    return dict(cn_target=CN, rain_mode="physical", manning=site != "dam", dt=dt,
                max_dt=dt if site in FIXED else 10.0, step_duration=(steps - 0.5) * dt if site in FIXED else steps * dt)


def _forcing(case, uniform=False):
    f = mf.Forcing()
    site = case["site"]
    if uniform or site == "plane":
        f.rain_kind, f.rain_q0, f.rain_q1 = mf.RAIN_UNIFORM, 50.0 * MM_PER_H, 40.0 * MM_PER_H
    elif site != "dam":
        f.rain_kind, f.rain_q0, f.rain_q1 = mf.RAIN_PATTERN, 1.0, 0.8
    if EDGES[site]:
        f.head_kind, f.head_edges, f.head_h0, f.head_h1 = mf.HEAD_EDGES, EDGES[site], HEAD[site], HEAD[site]
    return f


def _fill(b, case, fields):
    """Bed, roughness, rain and term fields of a solver or member, and its state in pinned arrays."""
    host = {k: _pinned(*v.shape, v) for k, v in fields.items() if k in ("H", "U", "V", "INFIL_CAP")}
    for k, v in fields.items():
        if k not in host:
            b.set_field(k, v.cpu().numpy())
    b.set_manning(0.03, 0.03, 0.1, 0.3)
    if "N_SHALLOW" in fields:
        n = fields["N_SHALLOW"].cpu().numpy()
        b.set_field("N_SHALLOW", n)
        b.set_field("N_DEEP", n)
    for k, v in host.items():
        b.set_field(k, v)
    if case.get("terms") in ("eddy", "all"):
        b.set_eddy_viscosity("smagorinsky")
    ny, nx = host["H"].shape
    return {"in": host, "out": {k: _pinned(ny, nx) for k in host}}


def _member_case(case, nx, ny, dx):
    return dict(kind="step", site=case["site"], precision=case["precision"], nx=nx, ny=ny, dx=dx, rk="classic",
                steps=case["steps"], tuned=False, terms="")


def prepare(case, seed):
    if case["kind"] == "batch":
        b = SaintVenantBatch(case["precision"])
        if case["persistent"]:
            b.set_persistent(True)
        members = []
        for i, (nx, ny, dx) in enumerate(_sizes(case)):
            mc = _member_case(case, nx, ny, dx)
            p = _params(mc)
            m = b.add(nx, ny, dx, cn_target=p["cn_target"], step_duration=p["step_duration"], initial_dt=p["dt"],
                      max_dt=p["max_dt"], rain_mode=p["rain_mode"], manning=p["manning"])
            buf = _fill(m, mc, _site(case["site"], nx, ny, dx, "", seed * 1000 + i))
            members.append((m, p["dt"], buf, [_forcing(mc)] * case["calls"]))
        return {"case": case, "batch": b, "members": members}
    nx, ny, dx = case["nx"], case["ny"], case["dx"]
    p = _params(case)
    fields = _site(case["site"], nx, ny, dx, case["terms"], seed * 1000)
    if case["kind"] == "noalloc":
        lib = mf.load_library()
        pd, pv = ctypes.POINTER(ctypes.c_double), ctypes.c_void_p
        lib.sv_timestep_noalloc.argtypes = [ctypes.POINTER(mf.MeshDesc), ctypes.POINTER(mf.Params), pd,
                                            ctypes.POINTER(mf.Forcing)] + [pv] * 7 + [ctypes.c_double] * 2 + [pv] * 2
        ins = [fields[k].contiguous() for k in ("Z", "H", "U", "V")]
        out = [torch.empty_like(ins[0]) for _ in range(3)] + [torch.zeros(3, dtype=torch.float64, device="cuda")]
        return {"case": case, "lib": lib, "in": ins, "out": out, "dt": p["dt"],
                "mesh": mf.MeshDesc(nx, ny, dx, dx, 0.0, 0.0),
                "params": mf.Params(mf.SV_F64, mf.RK_METHODS.index(case["rk"]), CN, 60.0, p["dt"], 0.0, 1, 1, 0, 0),
                "manning": (ctypes.c_double * 4)(0.03, 0.05, 0.1, 0.3), "forcing": _forcing(case, uniform=True)}
    s = mf.SaintVenantSolver(nx, ny, dx, precision=case["precision"], rk_method=case["rk"], cn_target=CN,
                             step_duration=p["step_duration"], initial_dt=p["dt"], max_dt=p["max_dt"],
                             rain_mode=p["rain_mode"], manning=p["manning"])
    buf = _fill(s, case, fields)
    s.set_forcing(_forcing(case))
    if case["tuned"]:
        s.autotune()
    return {"case": case, "solver": s, "dt": p["dt"], "buf": buf, "forcing": _forcing(case)}


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def _read(b, buf, precision, base=None):
    """The fields as the program keeps them: FP64 as read, FP32 solvers' values in FP32."""
    res = {}
    for i, (k, a) in enumerate(buf["out"].items()):
        b.get_field(k if base is None else base + i, out=a)
        t = torch.from_numpy(a)
        res[k] = t if precision == "f64" else t.to(torch.float32)
    return res


def run(state):
    case = state["case"]
    if case["kind"] == "noalloc":
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in state["in"] + state["out"]]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        r = state["lib"].sv_timestep_noalloc(ctypes.byref(state["mesh"]), ctypes.byref(state["params"]),
                                             state["manning"], ctypes.byref(state["forcing"]), *ptr[:7], 0.0,
                                             state["dt"], ptr[7], stream)
        if r != 0:
            raise mf.SvError(r, state["lib"].sv_last_error(None).decode())
        return state["out"]
    if case["kind"] == "timestep":
        s = state["solver"]
        cn, repeat, new_dt = s.do_timestep(0.0, state["dt"])
        return {**_read(s, state["buf"], "f64", 100 + 3 * s.nstages), "cn": cn, "repeat": repeat, "new_dt": new_dt}
    if case["kind"] == "step":
        s = state["solver"]
        for k, a in state["buf"]["in"].items():
            s.set_field(k, a)
        s.set_dt(state["dt"])
        s.set_forcing(state["forcing"])
        st = s.advance()
        return {**_read(s, state["buf"], case["precision"]), "accepted": st["accepted"], "repeated": st["repeated"],
                "volume": st["volume"]}
    for m, dt, buf, _ in state["members"]:
        for k, a in buf["in"].items():
            m.set_field(k, a)
        m.set_dt(dt)
    res = state["batch"].advance_steps({m: fs for m, _, _, fs in state["members"]})
    fields = [_read(m, buf, case["precision"]) for m, _, buf, _ in state["members"]]
    steps = [st for m, _, _, _ in state["members"] for st in res[m.slot]["steps"]]
    return {"fields": fields, "counts": np.array([[st["accepted"], st["repeated"]] for st in steps]),
            "volume": np.array([st["volume"] for st in steps], dtype=np.float32)}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
STAGES = dict(zip(mf.RK_METHODS, mf.RK_STAGES))


def work(case):
    """Bytes: per stage the state and its running sum in and out, the bed, roughness, rain and
    term fields once; per pass the state into and out of the device. Flops: about 350 per
    cell and stage (three limited slopes per axis, two faces, the cell's update)."""
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for nx, ny, dx in _sizes(case):
            w = work(_member_case(case, nx, ny, dx))
            total["bytes"] += case["calls"] * w["bytes"]
            total["flops"] += case["calls"] * w["flops"]
        return total
    n, stages = case["nx"] * case["ny"], STAGES[case["rk"]]
    size = 8 if case["precision"] == "f64" else 4
    # first stage: state, bed in; next state and sum out. later: also the sum in, on the last
    # stage only the state out
    values = 13 * stages - 6 if stages > 1 else 7
    fields = (1 if case["site"] in ("flood", "rain") and case["kind"] != "noalloc" else 0) * 2
    fields += 5 if case.get("terms") == "all" else 0
    per_step = n * size * (values + fields * stages)
    steps = case["steps"] if case["kind"] == "step" else 1
    io = 6 * 8 * n if case["kind"] == "step" else (3 * 8 * n if case["kind"] == "timestep" else 0)
    return {"bytes": float(per_step * steps + io), "flops": float(350 * n * stages * steps)}


# ---------------------------------------------------------------------------------------
# the same passes in 64 bits, whole arrays at a time
# ---------------------------------------------------------------------------------------
TABLEAU = {  # c and a of each stage, b
    "euler": ([0], [[]], [1]),
    "midpoint": ([0, 0.5], [[], [0.5]], [0, 1]),
    "heun2": ([0, 1], [[], [1]], [0.5, 0.5]),
    "heun3": ([0, 1 / 3, 2 / 3], [[], [1 / 3], [0, 2 / 3]], [0.25, 0, 0.75]),
    "ralston3": ([0, 0.5, 0.75], [[], [0.5], [0, 0.75]], [2 / 9, 1 / 3, 4 / 9]),
    "ssprk3": ([0, 1, 0.5], [[], [1], [0.25, 0.25]], [1 / 6, 1 / 6, 2 / 3]),
    "classic": ([0, 0.5, 0.5, 1], [[], [0.5], [0, 0.5], [0, 0, 1]], [1 / 6, 1 / 3, 1 / 3, 1 / 6]),
    "3/8rule": ([0, 1 / 3, 2 / 3, 1], [[], [1 / 3], [-1 / 3, 1], [1, -1, 1]], [1 / 8, 3 / 8, 3 / 8, 1 / 8]),
}


def _minmod(a, b):
    return 0.5 * (torch.sign(a) + torch.sign(b)) * torch.minimum(a.abs(), b.abs())


def _slope(a, d, axis):
    """Minmod3 slope (theta 2) along x (axis 1) or against y (axis 0); one-sided at the ends."""
    n = a.shape[axis]
    if n == 1:
        return torch.zeros_like(a)
    q = torch.diff(a, dim=axis) / d
    if axis == 0:
        q = -q
    lo, hi = q.narrow(axis, 0, n - 2), q.narrow(axis, 1, n - 2)
    mid = _minmod(_minmod(2 * lo, 2 * hi), (a.narrow(axis, 2, n - 2) - a.narrow(axis, 0, n - 2)) / (2 * d)
                  * (-1.0 if axis == 0 else 1.0))
    return torch.cat([q.narrow(axis, 0, 1), mid, q.narrow(axis, n - 2, 1)], dim=axis)


def _faces(z, h, un, ut, zn, hn, unn, utn, d, axis):
    """Fluxes (h, normal and tangential momentum, bed step) of every face along an axis,
    from cell values and their slopes along it; mesh edges are walls."""
    n = h.shape[axis]
    first, last = (lambda a: a.narrow(axis, 0, 1)), (lambda a: a.narrow(axis, n - 1, 1))

    def sides(a, s, lo, hi):
        m, p = a + 0.5 * d * s, a - 0.5 * d * s
        return torch.cat([lo(m, p), m], dim=axis), torch.cat([p, hi(m, p)], dim=axis)

    zero = torch.zeros_like(first(h))
    zm, zp = sides(z, zn, lambda m, p: first(z) + 2 * first(h), lambda m, p: last(z) + 2 * last(h))
    hm, hp = sides(h, hn, lambda m, p: zero, lambda m, p: zero)
    um, up = sides(un, unn, lambda m, p: zero, lambda m, p: zero)
    tm, tp = sides(ut, utn, lambda m, p: first(m), lambda m, p: last(p))
    zf = torch.maximum(zm, zp)
    above_m, above_p = zm + hm > zf, zp + hp > zf
    hm, hp = hm.clamp(min=0.0), hp.clamp(min=0.0)
    both, left, dry = above_m & above_p, above_m & ~above_p, ~above_m & ~above_p
    cm, cp = torch.sqrt(G * hm), torch.sqrt(G * hp)
    am = torch.where(um == 0, 0.0, um.abs() + cm)
    ap = torch.where(up == 0, 0.0, up.abs() + cp)
    a = torch.where(both, torch.maximum(am, ap), torch.where(left, am, ap))

    def flux(fm, fp, qm, qp):  # half the sum of the sides' fluxes less half a times the jump
        s = torch.where(both, fm + fp, torch.where(left, fm, fp))
        j = torch.where(both, qp - qm, torch.where(left, -qm, qp))
        return 0.5 * s - 0.5 * a * j

    fh = flux(hm * um, hp * up, hm, hp)
    fn = flux(0.5 * um * um + G * hm, torch.where(both, 0.5 * up * up - G * hp, 0.5 * up * up + G * hp), um, up)
    ft = flux(tm * um, tp * up, tm, tp)
    fz = torch.where(both, (zm - zp) * G, torch.where(left, hp, hm) / d)
    rise = zp > zm
    fn = torch.where(dry, torch.where(rise, 0.5 * G * hm, -0.5 * G * hp), fn)
    fz = torch.where(dry, torch.where(rise, -0.5 * G * hm, 0.5 * G * hp), fz)
    return torch.where(dry, 0.0, fh), fn, torch.where(dry, 0.0, ft), fz


def _capped(fu, u, dt):
    return torch.where(((fu * dt).abs() > u.abs()) & (torch.sign(fu) != torch.sign(u)), -u / dt, fu)


def _rates(case, prm, F, zs, h, u, v, t, dt, uniform):
    """dU/dt of a stage; consumes F["INFIL_CAP"]."""
    dx = case["dx"]
    hx, ux, vx = (_slope(a, dx, 1) for a in (h, u, v))
    hy, uy, vy = (_slope(a, dx, 0) for a in (h, u, v))
    xh, xu, xv, xz = _faces(F["Z"], h, u, v, zs[0], hx, ux, vx, dx, 1)
    yh, yv, yu, yz = _faces(F["Z"], h, v, u, zs[1], hy, vy, uy, dx, 0)
    div = lambda fx, fy: (fx[:, :-1] - fx[:, 1:]) / dx + (fy[:-1] - fy[1:]) / dx  # noqa: E731
    limit = lambda s: torch.where(s.abs() > h / dx, torch.sign(s) * h / dx, s)    # noqa: E731
    dh = div(xh, yh)
    du = div(xu, yu) - G * hx + (xz[:, :-1] - xz[:, 1:]) / dx - G * limit(zs[0])
    dv = div(xv, yv) - G * hy + (yz[:-1] - yz[1:]) / dx - G * limit(zs[1])
    wet, speed = h > 1e-6, torch.sqrt(u * u + v * v)
    if prm["manning"]:
        n = F["N"](h)
        sf = n * n * speed * (h / (h * h + 1e-3)).clamp(min=0.0) ** (4.0 / 3.0)
        du = du + torch.where(wet, _capped(-G * sf * u, u, dt), 0.0)
        dv = dv + torch.where(wet, _capped(-G * sf * v, v, dt), 0.0)
    if case.get("terms") == "all":
        du = du + torch.where(wet, _capped(-0.5 * u * F["ELOSS_FX"] * speed, u, dt), 0.0)
        dv = dv + torch.where(wet, _capped(-0.5 * v * F["ELOSS_FY"] * speed, v, dt), 0.0)
    if case.get("terms") in ("eddy", "all"):  # Smagorinsky, coefficients 0.05 and 0.5
        mu = 0.05 + 0.5 * dx * dx * torch.sqrt(ux * ux + vy * vy + 0.5 * (uy.abs() + vx.abs()) ** 2)
        du = du + torch.where(wet, _capped(-mu * (_slope(ux, dx, 1) + _slope(uy, dx, 0)), u, dt), 0.0)
        dv = dv + torch.where(wet, _capped(-mu * (_slope(vx, dx, 1) + _slope(vy, dx, 0)), v, dt), 0.0)
    if case.get("terms") == "all":
        take = torch.minimum(torch.minimum(F["INFIL_RATE"] * dt, h), F["INFIL_CAP"])
        dh = dh - take / dt
        F["INFIL_CAP"] = F["INFIL_CAP"] - take
    f = _forcing(case, uniform)
    if f.rain_kind != mf.RAIN_NONE:
        pattern = torch.ones_like(h) if f.rain_kind == mf.RAIN_UNIFORM else F["RAIN_PATTERN"]
        rate = (f.rain_q1 - f.rain_q0) / (60.0 if uniform else prm["step_duration"])
        q = pattern * (f.rain_q0 + t * rate + 0.5 * dt * rate)
        dh = dh + torch.where(pattern == 0, 0.0, torch.where(h + q * dt <= 0, -h / dt, q))
    e = torch.zeros_like(wet)
    e[:, 0] |= bool(f.head_edges & 1)
    e[:, -1] |= bool(f.head_edges & 2)
    e[0] |= bool(f.head_edges & 4)
    e[-1] |= bool(f.head_edges & 8)
    return torch.where(e, (f.head_h0 - h) / dt, dh), du, dv


def _timestep(case, prm, F, zs, U, t, dt, uniform=False):
    c, a, b = TABLEAU[case["rk"]]
    ks = []
    for s in range(len(b)):
        Y = [x + sum((dt * a[s][j] * ks[j][i] for j in range(s) if a[s][j]), torch.zeros_like(x)) for i, x in enumerate(U)]
        ks.append(_rates(case, prm, F, zs, *Y, t + c[s] * dt, dt, uniform))
    U = [x + sum(dt * b[j] * ks[j][i] for j in range(len(b)) if b[j]) for i, x in enumerate(U)]
    cel = torch.sqrt(G * U[0].clamp(min=0.0))
    cn = dt * float(((U[1].abs() + cel) / case["dx"] + (U[2].abs() + cel) / case["dx"]).max())
    if cn > CN:
        new, repeat = (dt / 5 if cn > 5 * CN else dt * CN / (cn * 1.1)), True
    else:
        new, repeat = (dt if cn > 0.9 * CN else dt * CN / cn), False
    return U, cn, repeat, min(new, prm["max_dt"]) if prm["max_dt"] > 0 else new


def _solve(case, seed, calls=1):
    prm = _params(case)
    F = _site(case["site"], case["nx"], case["ny"], case["dx"], case["terms"], seed)
    n = F.get("N_SHALLOW")
    if case["kind"] == "noalloc":
        prm["max_dt"] = 0.0

        def mixed(h):  # shallow to deep over 0.1-0.3 m
            w = ((h - 0.1) / 0.2).clamp(0.0, 1.0)
            return 0.03 + 0.02 * w * w * (3.0 - 2.0 * w)
        F["N"] = mixed
    else:
        F["N"] = lambda h: 0.03 if n is None else n
    zs = _slope(F["Z"], case["dx"], 1), _slope(F["Z"], case["dx"], 0)
    U, dt, vol = [F[k] for k in "HUV"], prm["dt"], []
    if case["kind"] != "step":
        return _timestep(case, prm, F, zs, U, 0.0, dt, case["kind"] == "noalloc")
    L = prm["step_duration"]
    for _ in range(calls):
        t = 0.0
        while t < L:
            new_U, cn, repeat, new = _timestep(case, prm, F, zs, U, t, dt)
            if not repeat:
                U, t = new_U, t + dt
            if t < L:
                new = L - t if t + new > L else ((L - t) * 0.4 if t + 2 * new > L else new)
            dt = new
        vol.append(float(U[0].sum()) * case["dx"] ** 2)
    res = dict(zip("HUV", U))
    if case["terms"] == "all":
        res["INFIL_CAP"] = F["INFIL_CAP"]
    return res, vol


def exact(case, seed):
    if case["kind"] == "batch":
        got = [_solve(_member_case(case, nx, ny, dx), seed * 1000 + i, case["calls"])
               for i, (nx, ny, dx) in enumerate(_sizes(case))]
        return {"fields": [g[0] for g in got], "counts": None,
                "volume": torch.tensor([v for g in got for v in g[1]], dtype=torch.float64)}
    if case["kind"] == "step":
        res, vol = _solve(case, seed * 1000)
        return {**res, "accepted": None, "repeated": None, "volume": torch.tensor(vol[0], dtype=torch.float64)}
    U, cn, repeat, new = _solve(case, seed * 1000)
    if case["kind"] == "noalloc":
        return [*U, torch.tensor([cn, new, float(repeat)], dtype=torch.float64, device="cuda")]
    return {**dict(zip("HUV", U)), "cn": torch.tensor(cn, dtype=torch.float64), "repeat": None,
            "new_dt": torch.tensor(new, dtype=torch.float64)}
