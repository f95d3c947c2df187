"""The work a user of this framework has it do, as timed cases: time steps of the
elastic wave equation on Cartesian grids and on grids with topography (FP64 and
FP32-mixed levels), whole shots with receivers, misfit gradients by the discrete
adjoint, and the kernel-level operators.

Every case is one call sequence through the public entry points on device data made
from a seed.  The levels are a developed wave field (plane waves of 8 to 20 points per
wavelength under a smooth envelope, the previous level one time step earlier), the
material a smooth medium or a layer over a half-space, the time step from the CFL
number 1.3 that the benchmark and the reference's decks use.
"""
import math

import torch

import sw4lite_gb300 as sg

H = 50.0  # grid spacing of every case (m)
CFL = 1.3
FREE_TOP = "free"  # free surface at k = 1, absorbing (supergrid) on the other sides


def listed():
    return [
        # one step on a very small grid: launches and latency count (coupling loops,
        # unit-test sized runs)
        {"name": "step_small", "kind": "step", "nx": 48, "ny": 40, "nz": 36, "gp": 15, "top": FREE_TOP,
         "precision": 0, "order": 4, "steps": 1},
        # a whole short shot at the size of the Gaussian point-force deck: levels from
        # rest, receivers recorded each step, records read back to the host
        {"name": "shot_101", "kind": "shot", "nx": 101, "ny": 101, "nz": 101, "gp": 20, "top": "absorbing",
         "precision": 0, "order": 4, "steps": 12},
        # FP64 steps on an odd, ragged grid, absorbing sides all round
        {"name": "step_ragged", "kind": "step", "nx": 203, "ny": 117, "nz": 95, "gp": 20, "top": "absorbing",
         "precision": 0, "order": 4, "steps": 2},
        # the headline set-up: layer over half-space, free surface, 512^3, FP64
        {"name": "step_512", "kind": "step", "nx": 512, "ny": 512, "nz": 512, "gp": 30, "top": FREE_TOP,
         "precision": 0, "order": 4, "steps": 1},
        # the same set-up in the FP32-mixed form
        {"name": "step_mixed_320", "kind": "step", "nx": 320, "ny": 320, "nz": 320, "gp": 30, "top": FREE_TOP,
         "precision": 1, "order": 4, "steps": 2},
        # FP32-mixed on extents that are no multiple of the copy alignment
        {"name": "step_mixed_ragged", "kind": "step", "nx": 157, "ny": 90, "nz": 75, "gp": 20,
         "top": "absorbing", "precision": 1, "order": 4, "steps": 2},
        # sixth-order damping, FP64, free surface
        {"name": "step_order6", "kind": "step", "nx": 160, "ny": 144, "nz": 128, "gp": 25, "top": FREE_TOP,
         "precision": 0, "order": 6, "steps": 2},
        # topography: the curvilinear grid over a Gaussian hill on a Cartesian grid
        {"name": "topo_192", "kind": "topo", "nx": 192, "ny": 192, "nz": 60, "gp": 20, "precision": 0,
         "steps": 2},
        # the FP32-mixed form of the same, ragged
        {"name": "topo_mixed", "kind": "topo", "nx": 150, "ny": 131, "nz": 50, "gp": 20, "precision": 1,
         "steps": 2},
        # one iteration of a waveform inversion: misfit and gradient of one shot
        {"name": "gradient_64", "kind": "gradient", "nx": 64, "ny": 64, "nz": 64, "gp": 15, "precision": 0,
         "steps": 20, "every": 10},
        # the kernel-level operator as a caller with its own time loop uses it
        {"name": "operator", "kind": "operator", "nx": 256, "ny": 200, "nz": 150, "soa": 1},
        # the curvilinear kernel-level operator, point-major layout
        {"name": "operator_curv", "kind": "operator_curv", "nx": 130, "ny": 121, "nz": 64, "soa": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "shot", "topo", "gradient", "operator", "operator_curv"])
    c = {"kind": kind}
    if kind in ("step", "shot"):
        top = 400 if kind == "step" else 160
        c.update(nx=_log(rng, 40, top), ny=_log(rng, 40, top), nz=_log(rng, 36, top))
        c.update(gp=rng.randint(15, 30) if min(c["nx"], c["ny"], c["nz"]) > 64 else 15,
                 top=rng.choice([FREE_TOP, "absorbing"]), precision=rng.choice([0, 0, 1]),
                 order=rng.choice([4, 4, 6]) if kind == "step" else 4,
                 steps=rng.randint(1, 3) if kind == "step" else rng.randint(6, 30))
        if c["order"] == 6:
            c["gp"] = max(c["gp"], 20)
    elif kind == "topo":
        c.update(nx=_log(rng, 60, 240), ny=_log(rng, 60, 240), nz=rng.randint(40, 90),
                 gp=rng.randint(18, 25), precision=rng.choice([0, 1]), steps=rng.randint(1, 3))
    elif kind == "gradient":
        c.update(nx=_log(rng, 40, 90), ny=_log(rng, 40, 90), nz=_log(rng, 40, 90), gp=15,
                 precision=rng.choice([0, 1]), steps=rng.randint(8, 30), every=rng.randint(4, 12))
    else:
        big = 300 if kind == "operator" else 150
        c.update(nx=_log(rng, 20, big), ny=_log(rng, 20, big), nz=_log(rng, 20, 150),
                 soa=rng.choice([0, 1]))
    return c


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _axes(c):
    """Point coordinates, ghosts included, broadcast over (nz+4, ny+4, nx+4)."""
    def line(n):
        return (torch.arange(n + 4, dtype=torch.float64, device="cuda") - 2) * H
    return line(c["nx"])[None, None, :], line(c["ny"])[None, :, None], line(c["nz"])[:, None, None]


def _rng(seed):
    return torch.Generator().manual_seed(int(seed))


def _uniform(g, n, lo, hi):
    return (lo + (hi - lo) * torch.rand(n, generator=g, dtype=torch.float64)).tolist()


def _material(c, seed):
    """(rho, mu, lambda): a 1 km layer over a half-space (vp 4000 / 6000 m/s) with smooth
    variations of a few percent."""
    x, y, z = _axes(c)
    g = _rng(seed)
    layer = z <= 1000.0
    vp, vs, rho = (torch.where(layer, a, b) for a, b in ((4000.0, 6000.0), (2000.0, 3464.0), (2600.0, 2700.0)))
    out = []
    for base, amp in ((vp, 0.02), (vs, 0.02), (rho, 0.02)):
        k = _uniform(g, 3, 2e-4, 8e-4)
        p = _uniform(g, 3, 0.0, 6.28)
        f = torch.sin(k[0] * x + p[0]) * torch.sin(k[1] * y + p[1])
        out.append((base * (1 + amp * f * torch.cos(k[2] * z + p[2]))).to(torch.float64).contiguous())
    vp, vs, rho = out
    mu = rho * vs * vs
    la = rho * vp * vp - 2 * mu
    return [a.reshape(-1) for a in (rho, mu, la)]


def _time_step(mat):
    rho, mu, la = mat
    return CFL * H / math.sqrt(float(((4 * mu + la) / rho).max()))


def _levels(c, seed, dt):
    """The current and previous level of a developed wave field (3 x npts each)."""
    x, y, z = _axes(c)
    g = _rng(seed + 1)
    size = [(c[n] - 1) * H for n in ("nx", "ny", "nz")]
    mid = [s * u for s, u in zip(size, _uniform(g, 3, 0.4, 0.6))]
    if c.get("top") == FREE_TOP:
        mid[2] = 0.25 * size[2]
    env = torch.exp(-((x - mid[0]) / (0.28 * size[0])) ** 2) * torch.exp(-((y - mid[1]) / (0.28 * size[1])) ** 2)
    env = env * torch.exp(-((z - mid[2]) / (0.28 * size[2])) ** 2)
    now, before = (torch.zeros((3,) + tuple(env.shape), dtype=torch.float64, device="cuda") for _ in range(2))
    for comp in range(3):
        for _ in range(2):
            d = torch.randn(3, generator=g, dtype=torch.float64)
            d = (d / d.norm()).tolist()
            wave, phase, amp = _uniform(g, 1, 8 * H, 20 * H)[0], _uniform(g, 1, 0.0, 6.28)[0], _uniform(g, 1, 0.3, 1.0)[0]
            k = 2 * math.pi / wave
            arg = k * (d[0] * x + d[1] * y + d[2] * z) + phase
            now[comp] += amp * torch.cos(arg)
            before[comp] += amp * torch.cos(arg + k * 3464.0 * dt)
    now *= env
    before *= env
    if c.get("top") is not None:  # ghost planes as a time loop leaves them on absorbing sides
        for u in (now, before):
            lo = 2 if c["top"] == FREE_TOP else 0
            u[:, :, :, :2] = 0
            u[:, :, :, -2:] = 0
            u[:, :, :2] = 0
            u[:, :, -2:] = 0
            u[:, -2:] = 0
            if lo == 0:
                u[:, :2] = 0
    return now.reshape(-1), before.reshape(-1)


def _grid(c):
    top = sg.FREE if c.get("top") == FREE_TOP else sg.SUPERGRID
    return sg.grid_desc(c["nx"], c["ny"], c["nz"], H, bc=(sg.SUPERGRID,) * 4 + (top, sg.SUPERGRID),
                        sg_gp=c["gp"], sg_order=c.get("order", 4), precision=c["precision"])


def _points(c, g, n):
    """n grid points inside the absorbing layers."""
    m = min(c["gp"] + 1, (min(c["nx"], c["ny"], c["nz"]) - 4) // 2)
    return [[int(u) for u in (_uniform(g, 1, m + 1, c[a] - m)[0] for a in ("nx", "ny", "nz"))] for _ in range(n)]


def _sources(c, seed):
    """Grid-point forces (Gaussian in time) as a discretised source leaves them."""
    g = _rng(seed + 2)
    ijk = _points(c, g, 6)
    amp = [_uniform(g, 3, -1e14, 1e14) for _ in ijk]
    return ijk, amp, [20.0] * 6, [0.02] * 6, [sg.GAUSSIAN] * 6


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _object(c, seed):
    mat = _material(c, seed)
    ew = sg.EW(_grid(c))
    ew.set_material(*mat)
    dt = _time_step(mat)
    ew.set_time_step(dt, 0.0)
    return ew, mat, dt


def _prepare_step(c, seed):
    ew, mat, dt = _object(c, seed)
    del mat
    ew.add_grid_point_sources(*_sources(c, seed))
    u, um = _levels(c, seed, dt)
    return {"case": c, "ew": ew, "dt": dt, "u": u, "um": um, "new": torch.empty_like(u),
            "old": torch.empty_like(u)}


def _prepare_shot(c, seed):
    ew, mat, dt = _object(c, seed)
    ew.add_grid_point_sources(*_sources(c, seed))
    zero = torch.zeros(3 * ew.npts, dtype=torch.float64, device="cuda")
    rec = _points(c, _rng(seed + 3), 16)
    return {"case": c, "ew": ew, "dt": dt, "zero": zero, "rec": rec, "new": torch.empty_like(zero)}


def _prepare_gradient(c, seed):
    c = dict(c, top="absorbing")
    ew, mat, dt = _object(c, seed)
    ew.add_grid_point_sources(*_sources(c, seed))
    rec = _points(c, _rng(seed + 3), 12)
    ew.set_receivers(rec, [sg.REC_DISPLACEMENT] * len(rec), c["steps"] + 1)
    u, um = _levels(c, seed, dt)
    obs = torch.randn((c["steps"] + 1, 3 * len(rec)), generator=_rng(seed + 4), dtype=torch.float64)
    g = [torch.empty(ew.npts, dtype=torch.float64, device="cuda") for _ in range(3)]
    return {"case": c, "ew": ew, "dt": dt, "u": u, "um": um, "obs": (0.1 * obs).cuda(), "grad": g}


def _hill(c):
    xc, yc = 0.5 * (c["nx"] - 1) * H, 0.5 * (c["ny"] - 1) * H
    return 400.0, xc, yc, 0.15 * (c["nx"] - 1) * H, 0.15 * (c["ny"] - 1) * H


def _prepare_topo(c, seed):
    amp, xc, yc, lx, ly = _hill(c)
    bottom = 1500.0  # the interface between the two grids
    g = sg.grid_desc(c["nx"], c["ny"], c["nz"], H, bc=(sg.SUPERGRID,) * 4 + (sg.INTERFACE, sg.SUPERGRID),
                     zmin=bottom, sg_gp=c["gp"], precision=c["precision"])
    ew = sg.EW(g, topo=sg.topo_desc(amp, xc, yc, lx, ly))
    x, y, _ = _axes(c)
    surface = -amp * torch.exp(-((x - xc) / lx) ** 2 - ((y - yc) / ly) ** 2)

    def material(z):
        vs = 2000.0 + 0.5 * torch.clamp(z - surface, min=0.0)
        rho = torch.full_like(vs, 2500.0)
        mu = rho * vs * vs
        return [a.reshape(-1).contiguous() for a in (rho, mu, mu.clone())]

    zc = bottom + (torch.arange(c["nz"] + 4, dtype=torch.float64, device="cuda") - 2)[:, None, None] * H
    ew.set_material(*material(zc.expand(c["nz"] + 4, c["ny"] + 4, c["nx"] + 4)))
    _, _, nc, n1 = ew.grid_dims(1)
    z1 = torch.empty(n1, dtype=torch.float64, device="cuda")
    ew.curvilinear_arrays(z=z1)
    ew.set_material_grid(1, *material(z1.reshape(nc + 4, c["ny"] + 4, c["nx"] + 4)))
    dt, _ = ew.compute_time_step(CFL, 1.0)
    ew.set_time_step(dt, 0.0)
    ew.add_source(sg.source_desc(xc, yc, bottom + 6 * H, force=(1e13, -2e13, 5e13), freq=20.0, t0=0.02,
                                 kind=sg.GAUSSIAN))
    # one wave field over both grids, continuous across the interface: the Cartesian
    # grid's planes follow the curvilinear grid's
    both = _levels(dict(c, nz=c["nz"] + nc - 1), seed, dt)
    both = [u.reshape(3, c["nz"] + nc + 3, c["ny"] + 4, c["nx"] + 4) for u in both]
    cart = [u[:, nc - 1:].contiguous().reshape(-1) for u in both]
    curv = [u[:, :nc + 4].contiguous().reshape(-1) for u in both]
    return {"case": c, "ew": ew, "dt": dt, "cart": cart, "curv": curv, "new": torch.empty_like(cart[0]),
            "new_curv": torch.empty_like(curv[0])}


def _layout(a, npts, comps, soa):
    """A component-major array in the layout `soa` asks for."""
    return a if soa else a.reshape(comps, npts).t().contiguous().reshape(-1)


def _bounds(c):
    return [-1, c["nx"] + 2, -1, c["ny"] + 2, -1, c["nz"] + 2]


def _prepare_operator(c, seed):
    _, mu, la = _material(c, seed)
    u, _ = _levels(c, seed, 0.005)
    g = _rng(seed + 5)
    stretch = [(0.5 + 0.5 * torch.rand(c[n] + 4, generator=g, dtype=torch.float64)).cuda() for n in ("nx", "ny", "nz")]
    u = _layout(u, mu.numel(), 3, c["soa"])
    return {"case": c, "u": u, "mu": mu, "la": la, "stretch": stretch, "lu": torch.zeros_like(u),
            "sides": (sg.C.c_int * 6)()}


def _prepare_operator_curv(c, seed):
    _, mu, la = _material(c, seed)
    u, _ = _levels(c, seed, 0.005)
    x, y, z = _axes(c)
    amp, xc, yc, lx, ly = _hill(c)
    depth = (c["nz"] - 1) * H
    hill = -0.6 * amp * torch.exp(-((x - xc) / lx) ** 2 - ((y - yc) / ly) ** 2)
    z3 = (z + hill * (1 - z / depth)).contiguous().reshape(-1)
    met, jac = torch.zeros(4 * z3.numel(), dtype=torch.float64, device="cuda"), torch.zeros_like(z3)
    sg.check(sg.lib().sw4g_metric(c["soa"], *_bounds(c), H, *[a.data_ptr() for a in (z3, met, jac)], _stream()))
    one = [torch.ones(c[n] + 4, dtype=torch.float64, device="cuda") for n in ("nx", "ny")]
    u = _layout(u, mu.numel(), 3, c["soa"])
    return {"case": c, "u": u, "mu": mu, "la": la, "met": met, "jac": jac, "stretch": one,
            "lu": torch.zeros_like(u), "sides": (sg.C.c_int * 6)()}


def _stream():
    return torch.cuda.current_stream().cuda_stream or None


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_step(s):
    ew = s["ew"]
    ew.set_time_step(s["dt"], 0.0)
    ew.set_fields(s["u"], s["um"])
    ew.step(s["case"]["steps"])
    ew.get_fields(s["new"], s["old"])
    return s["new"], s["old"]


def _run_shot(s):
    ew, c = s["ew"], s["case"]
    ew.set_time_step(s["dt"], 0.0)
    ew.set_fields(s["zero"], s["zero"])
    ew.set_receivers(s["rec"], [sg.REC_VELOCITY] * len(s["rec"]), c["steps"] + 1)
    ew.step(c["steps"])
    records = ew.records()
    ew.get_fields(s["new"], None)
    return s["new"], records


def _run_topo(s):
    ew = s["ew"]
    ew.set_time_step(s["dt"], 0.0)
    ew.set_fields(*s["cart"])
    ew.set_fields_grid(1, *s["curv"])
    ew.step(s["case"]["steps"])
    ew.get_fields(s["new"], None)
    ew.get_fields_grid(1, s["new_curv"])
    return s["new"], s["new_curv"]


def _run_gradient(s):
    ew, c = s["ew"], s["case"]
    ew.set_time_step(s["dt"], 0.0)
    ew.set_fields(s["u"], s["um"])
    misfit = ew.gradient(c["steps"], c["every"], s["obs"], *s["grad"])
    return [misfit] + s["grad"]


def _run_operator(s):
    c = s["case"]
    sx, sy, sz = s["stretch"]
    sg.check(sg.lib().sw4g_rhs4sg(c["soa"], *_bounds(c), c["nz"], s["sides"], *[a.data_ptr() for a in
             (s["lu"], s["u"], s["mu"], s["la"])], H, *[a.data_ptr() for a in (sx, sy, sz)], _stream()))
    return s["lu"]


def _run_operator_curv(s):
    c = s["case"]
    sg.check(sg.lib().sw4g_rhs4sgcurv(c["soa"], *_bounds(c), s["sides"], *[a.data_ptr() for a in
             (s["lu"], s["u"], s["mu"], s["la"], s["met"], s["jac"], *s["stretch"])], _stream()))
    return s["lu"]


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    """Bytes: each input read once and each output written once.  Operations: per point
    of one operator 3 x 3 second differences (9 each), 3 x 6 mixed terms (about 10 each
    with shared inner differences) and the update."""
    n = (case["nx"] + 4) * (case["ny"] + 4) * (case["nz"] + 4)
    word = 8
    per_op = 9 * 9 + 18 * 10
    if case["kind"] == "operator":
        return {"bytes": n * word * (3 + 3 + 2), "flops": n * per_op}
    if case["kind"] == "operator_curv":
        return {"bytes": n * word * (3 + 3 + 2 + 5), "flops": n * 2 * per_op}
    if case["kind"] == "topo":
        n += (case["nx"] + 4) * (case["ny"] + 4) * 40
    steps = case["steps"] * (3 if case["kind"] == "gradient" else 1)
    # two levels and the material in, per step two new levels out
    return {"bytes": n * word * (6 + 3 + 6 * steps), "flops": steps * n * 2 * (per_op + 12)}


# --------------------------------------------------------------------------
# The same in plain torch, 64 bits, for grids with absorbing sides
# --------------------------------------------------------------------------
def _roll(a, m, ax):
    """a at the point m further along axis ax (0 x, 1 y, 2 z)."""
    return torch.roll(a, -m, dims=-1 - ax)


def _d1(a, ax):
    return (_roll(a, -2, ax) - _roll(a, 2, ax)) + 8 * (_roll(a, 1, ax) - _roll(a, -1, ax))


def _d2(coef, f, ax):
    """(coef f')' on five points, times 6 (Sjogreen & Petersson, J. Sci. Comput. 52, 2012)."""
    a = {m: _roll(coef, m, ax) for m in range(-2, 3)}
    w = {-2: a[-1] - 0.75 * (a[0] + a[-2]), -1: a[-2] + a[1] + 3 * (a[0] + a[-1]),
         1: a[-1] + a[2] + 3 * (a[1] + a[0]), 2: a[1] - 0.75 * (a[0] + a[2])}
    return sum(w[m] * (_roll(f, m, ax) - f) for m in w)


def _interior(a, edge=2):
    out = torch.zeros_like(a)
    cut = (Ellipsis,) + (slice(edge, -edge),) * 3
    out[cut] = a[cut]
    return out


def _operator(u, mu, la, s):
    """Divergence of stress with stretching s = (sx, sy, sz), zero on the two outer layers."""
    out = []
    for c in range(3):
        r = 0
        for ax in range(3):
            coef = (2 * mu + la if ax == c else mu) * s[ax]
            r = r + s[ax] * _d2(coef, u[c], ax) / 6
        for ax in range(3):
            if ax != c:
                r = r + s[c] * s[ax] * (_d1(la * _d1(u[ax], ax), c) + _d1(mu * _d1(u[ax], c), ax)) / 144
        out.append(r / (H * H))
    return _interior(torch.stack(out))


def _profiles(n, gp, left):
    """Supergrid damping, stretching and corner taper along an axis of n points."""
    x = (torch.arange(n + 4, dtype=torch.float64, device="cuda") - 2) * H
    width, end = gp * H, (n - 1) * H
    into = torch.where(x > end - width, x - (end - width), torch.zeros_like(x))
    if left:
        into = torch.where(x < width, width - x, into)

    def smooth(xi):
        xi = xi.clamp(0.0, 1.0)
        p = xi ** 6 * (462 - 1980 * xi + 3465 * xi ** 2 - 3080 * xi ** 3 + 1386 * xi ** 4 - 252 * xi ** 5)
        return torch.where(xi >= 1, torch.ones_like(p), p)

    stretch = 1 - (1 - 1e-4) * smooth(into / width)
    return smooth(into / (0.5 * width)) / stretch, stretch, 1 - (1 - 0.33) * into / width


def _damping(d, rho, prof):
    """Fourth-order supergrid damping of d = u - um."""
    (dx, sx, cx), (dy, sy, cy), (dz, sz, cz) = prof
    out = 0
    for ax, (dc, w) in enumerate(((dx, sx * cy * cz), (dy, sy * cx * cz), (dz, sz * cx * cy))):
        e = rho * dc
        q = e * (_roll(d, 1, ax) - 2 * d + _roll(d, -1, ax))
        out = out + w * (_roll(q, 1, ax) - 2 * q + _roll(q, -1, ax))
    return _interior(out)


def _force(src, shape, t, second):
    ijk, amp, freq, t0, _ = src
    f = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for (i, j, k), a, w, s in zip(ijk, amp, freq, t0):
        x = ((t - s) * w) ** 2 / 2
        g = w / math.sqrt(2 * math.pi) * math.exp(-x) * (w * w * (2 * x - 1) if second else 1.0)
        f[:, k + 1, j + 1, i + 1] += g * torch.tensor(a, dtype=torch.float64, device="cuda")
    return f


def _steps(c, mat, src, u, um, dt, each=None):
    shape = (c["nz"] + 4, c["ny"] + 4, c["nx"] + 4)
    rho, mu, la = [a.reshape(shape) for a in mat]
    prof = []
    for ax, n in enumerate(("nx", "ny", "nz")):
        prof.append([p.reshape([-1 if d == 2 - ax else 1 for d in range(3)]) for p in _profiles(c[n], c["gp"], True)])
    s = [p[1] for p in prof]
    u, um = u.reshape((3,) + shape), um.reshape((3,) + shape)
    if each:
        each(0, u, um)
    for n in range(c["steps"]):
        t = n * dt
        up = _interior(2 * u - um + dt * dt / rho * (_operator(u, mu, la, s) + _force(src, u.shape, t, False)))
        acc = (up - 2 * u + um) / (dt * dt)
        new = up + dt ** 4 / (12 * rho) * (_operator(acc, mu, la, s) + _force(src, u.shape, t, True))
        new = _interior(new - 0.02 / rho * _damping(u - um, rho, prof))
        if each:
            each(n + 1, new, um)
        u, um = new, u
    return u.reshape(-1), um.reshape(-1)


def exact(case, seed):
    c = case
    if c["kind"] == "operator":
        _, mu, la = _material(c, seed)
        s = prepare(c, seed)
        shape = (c["nz"] + 4, c["ny"] + 4, c["nx"] + 4)
        u = _levels(c, seed, 0.005)[0].reshape((3,) + shape)
        st = [p.reshape([-1 if d == 2 - ax else 1 for d in range(3)]) for ax, p in enumerate(s["stretch"])]
        return _layout(_operator(u, mu.reshape(shape), la.reshape(shape), st).reshape(-1), mu.numel(), 3, c["soa"])
    absorbing = c.get("top") == "absorbing" or c["kind"] == "gradient"
    if c["kind"] not in ("step", "shot", "gradient") or not absorbing or c.get("order", 4) != 4:
        return None
    mat = _material(c, seed)
    dt = _time_step(mat)
    src = _sources(c, seed)
    if c["kind"] == "step":
        return _steps(c, mat, src, *_levels(c, seed, dt), dt)
    rec = _points(c, _rng(seed + 3), 16 if c["kind"] == "shot" else 12)
    at = [torch.tensor([r[a] + 1 for r in rec], device="cuda") for a in (2, 1, 0)]
    rows = []
    if c["kind"] == "shot":
        zero = torch.zeros(3 * mat[0].numel(), dtype=torch.float64, device="cuda")

        def velocity(n, new, um):
            rows.append(((new - um) / (2 * dt) if n else 0 * new)[:, at[0], at[1], at[2]].t().reshape(-1))
        u, _ = _steps(c, mat, src, zero, zero.clone(), dt, velocity)
        return u, torch.stack(rows).cpu().numpy()
    c = dict(c, top="absorbing")
    mat = [a.requires_grad_() for a in mat]
    obs = (0.1 * torch.randn((c["steps"] + 1, 36), generator=_rng(seed + 4), dtype=torch.float64)).cuda()
    _steps(c, mat, src, *_levels(c, seed, dt), dt,
           lambda n, new, um: rows.append(new[:, at[0], at[1], at[2]].t().reshape(-1)))
    misfit = 0.5 * (torch.stack(rows) - obs).square().sum()
    return [float(misfit)] + [g.detach() for g in torch.autograd.grad(misfit, mat)]
