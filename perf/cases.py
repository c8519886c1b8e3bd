"""Measured work of the LES core: the calls a user of the library makes, through its public entry points.

Two kinds of user are covered.  A Fortran program that keeps its own time loop calls single routines of the drop-in
boundary on its device arrays (horizontal derivatives, the filtering of a field, the 3/2-rule products, the pressure
solve).  A program or a server that leaves the time loop to the library advances resident members by whole steps, one
member or an ensemble, in the FP64 form, the FP64 form with float-float transforms and the FP32-mixed form.

Step cases advance one dynamic-model cycle (cs_count = 5 steps) a pass, so each pass holds the same mix of ordinary and
Lagrangian steps.  Grids are those of the repository's configurations, tests and benchmarks, and other 2^a 3^b sizes.
"""
import math

import numpy as np
import torch

import les_gb300 as lg

CYCLE = 5          # steps a pass of the step cases: one update of the dynamic model
TADV1 = 1.5        # Adams-Bashforth weight of the new right-hand side, in the pressure equation


def listed():
    return [
        # one surface plane's horizontal derivatives (a boundary-condition routine): the smallest call, all latency
        {"name": "ddxy_plane_32", "kind": "ddxy", "nx": 32, "ny": 32, "nz": 1},
        # Nyquist filter and derivatives of one field of a small rectangular domain, sizes with factors of 3
        {"name": "filt_da_96x64x37", "kind": "filt_da", "nx": 96, "ny": 64, "nz": 37},
        # the same for a slab of the largest grid
        {"name": "filt_da_256x256x64", "kind": "filt_da", "nx": 256, "ny": 256, "nz": 64},
        # a field to the 3/2 grid and back: the dealiased product of a caller's own advection routine
        {"name": "dealias_192x192x32", "kind": "dealias", "nx": 192, "ny": 192, "nz": 32},
        # the pressure solve of a large member, called from a Fortran time loop
        {"name": "press_256x256x128", "kind": "press", "nx": 256, "ny": 256, "nz": 128},
        # the smallest member, neutral, from captured graphs: launches and short kernels
        {"name": "step_fp64_32", "kind": "step", "nx": 32, "ny": 32, "nz": 32, "precision": 0, "model": 5,
         "theta": False, "humid": False, "jt0": 0, "graph": True},
        # the reference's usual resolution with temperature over a striped surface
        {"name": "step_fp64_128", "kind": "step", "nx": 128, "ny": 128, "nz": 128, "precision": 0, "model": 5,
         "theta": True, "humid": False, "jt0": 500, "graph": False},
        # the benchmark grid in full FP64: the largest
        {"name": "step_fp64_256", "kind": "step", "nx": 256, "ny": 256, "nz": 256, "precision": 0, "model": 5,
         "theta": True, "humid": False, "jt0": 0, "graph": False},
        # FP64 state with float-float transforms at the usual resolution
        {"name": "step_ff_128", "kind": "step", "nx": 128, "ny": 128, "nz": 128, "precision": 2, "model": 5,
         "theta": True, "humid": False, "jt0": 500, "graph": False},
        # the benchmark's headline form and grid
        {"name": "step_mixed_256", "kind": "step", "nx": 256, "ny": 256, "nz": 256, "precision": 1, "model": 5,
         "theta": True, "humid": False, "jt0": 0, "graph": False},
        # a moist mixed member on a rectangular grid, as a server steps it
        {"name": "step_mixed_humid_96x64x40", "kind": "step", "nx": 96, "ny": 64, "nz": 40, "precision": 1, "model": 5,
         "theta": True, "humid": True, "jt0": 500, "graph": True},
        # a batch of mixed members of the ensemble benchmark's sizes, one graph launch a step
        {"name": "ensemble_mixed_8", "kind": "ensemble", "precision": 1, "jt0": 500,
         "sizes": "32x32x32 32x32x32 32x32x32 64x64x48 64x64x48 96x96x64 96x96x64 128x128x128"},
    ]


SIZES = [16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256]     # 2^a 3^b, divisible by 4
STEP_SIZES = [32, 48, 64, 72, 96, 128, 144, 192, 256]
MODELS = [5, 5, 5, 4, 2, 7]


def _levels(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ddxy", "filt_da", "dealias", "press", "step", "step", "step", "ensemble"])
    if kind in ("ddxy", "filt_da", "dealias", "press"):
        nx, ny = rng.choice(SIZES), rng.choice(SIZES)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": _levels(rng, 4 if kind == "press" else 1, 129)}
    if kind == "ensemble":
        sizes = []
        for _ in range(rng.randint(2, 6)):
            n = rng.choice([32, 48, 64, 96])
            sizes.append("%dx%dx%d" % (n, rng.choice([n, n // 2 * 3 if n < 64 else n]), _levels(rng, 16, 64)))
        return {"kind": kind, "precision": rng.choice([0, 1, 1, 2]), "jt0": 500, "sizes": " ".join(sizes)}
    precision = rng.choice([0, 0, 1, 1, 2])
    while True:
        nx, ny, nz = rng.choice(STEP_SIZES), rng.choice(STEP_SIZES), _levels(rng, 16, 160)
        if nx * ny * nz <= 3_000_000:
            break
    theta = rng.random() < 0.75
    model = 5 if precision == 1 else rng.choice(MODELS if theta else MODELS[:5])
    return {"kind": "step", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "model": model, "theta": theta,
            "humid": theta and rng.random() < 0.35, "jt0": rng.choice([0, 500]) if nz <= 128 else 0,
            "graph": rng.random() < 0.5}


# ---- inputs -----------------------------------------------------------------------------------------------------------
class _Field:
    """A module array of a context, for torch: keeps the context that owns the memory."""

    def __init__(self, ctx, name, shape):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "version": 3,
                                         "data": (ctx.device_ptr(name), False), "strides": None}


def _view(ctx, name):
    return torch.as_tensor(_Field(ctx, name, lg.config.field_shape(ctx.cfg, name)), device="cuda")


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _noise(gen, *shape):
    return 2.0 * torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64) - 1.0


def _wind(gen, cfg, nlev, pad=2):
    """One velocity-like field (nlev, ny, ld): the log-law mean of its levels and the initial noise; zero padding columns."""
    z = (torch.arange(nlev, device="cuda", dtype=torch.float64) + 0.5) / max(cfg.nz - 1, 1)
    f = torch.zeros(nlev, cfg.ny, cfg.nx + pad, device="cuda", dtype=torch.float64)
    f[:, :, :cfg.nx] = torch.log(z / 1e-4)[:, None, None] / cfg.vonk + 0.1 * _noise(gen, nlev, cfg.ny, cfg.nx)
    return f


def _dt(nx, nz):
    # the benchmark's step; on the largest grids the one that stays inside the explicit diffusion limit
    return 2e-4 if max(nx, nz) <= 160 else 4e-5


def _member(nx, ny, nz, precision, model, theta, humid, jt0, seed, surface=None):
    """A resident member with its seeded start state, as the repository's workloads set it, made on the GPU."""
    cfg = lg.make_config(nx, ny, nz, s_flag=int(theta), q_flag=int(humid), model=model, precision=precision,
                         jt_total0=jt0, dt=_dt(nx, nz), rmsdiv_every=0)
    surf = surface(cfg) if surface else (lg.striped_surface(cfg) if theta else lg.uniform_surface(cfg, 1e-4, 0.0))
    ctx = lg.Context(cfg, surf)
    gen = _gen(seed)
    top = cfg.nz - 1
    state = {"u": _view(ctx, "u"), "v": _view(ctx, "v"), "w": _view(ctx, "w")}
    state["u"].copy_(_wind(gen, cfg, cfg.nz))
    for name in ("v", "w"):
        state[name][:, :, :nx] = 0.1 * _noise(gen, cfg.nz, ny, nx)
    state["w"][0] = 0.0
    state["w"][top] = 0.0
    if theta:
        t = state["theta"] = _view(ctx, "theta")
        # temperature noise through the whole depth: the dynamic scalar model has no value for a uniform level
        t[:, :, :nx] = (300.0 + 0.1 * _noise(gen, cfg.nz, ny, nx)) / cfg.t_scale
    if humid:
        q = state["q"] = _view(ctx, "q")
        q[:, :, :nx] = (10.0 + 0.2 * _noise(gen, cfg.nz, ny, nx)) / cfg.q_scale
        ctx.set("wq_s", lg.config.moisture_flux(cfg))
    for name in state:
        if name != "w":
            state[name][top] = state[name][top - 1]
    return ctx, state


def _patches(seed):
    def surface(cfg):
        s = lg.patch_surface(cfg, seed)
        s.wt_s[:] = 0.05
        return s
    return surface


def _sizes(case):
    return [tuple(int(n) for n in s.split("x")) for s in case["sizes"].split()]


def _routine_inputs(case, seed):
    nx, ny, nlev = case["nx"], case["ny"], case["nz"]
    cfg = lg.make_config(nx, ny, max(nlev, 4), dt=_dt(nx, nlev), rmsdiv_every=0)
    gen = _gen(seed)
    if case["kind"] == "press":
        u = _wind(gen, cfg, cfg.nz)
        v, w, divtz = (torch.zeros_like(u) for _ in range(3))
        for f, a in ((v, 0.1), (w, 0.1), (divtz, 1.0)):
            f[:, :, :nx] = a * _noise(gen, cfg.nz, ny, nx)
        w[0] = 0.0
        w[-1] = 0.0
        return cfg, {"u": u, "v": v, "w": w, "divtz": divtz}
    return cfg, {"f": _wind(gen, cfg, nlev)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        ctx, fields = _member(case["nx"], case["ny"], case["nz"], case["precision"], case["model"], case["theta"],
                              case["humid"], case["jt0"], seed)
        torch.cuda.synchronize()
        return {"kind": kind, "ctx": ctx, "graph": case["graph"], "out": fields}
    if kind == "ensemble":
        made = [_member(nx, ny, nz, case["precision"], 5, True, False, case["jt0"], seed * 64 + k, _patches(seed * 64 + k))
                for k, (nx, ny, nz) in enumerate(_sizes(case))]
        torch.cuda.synchronize()
        return {"kind": kind, "ensemble": lg.Ensemble([m for m, _ in made]), "out": [f for _, f in made]}
    cfg, inp = _routine_inputs(case, seed)
    ctx = lg.Context(cfg, lg.uniform_surface(cfg))
    ctx.set_pointer_mode(True)
    state = {"kind": kind, "ctx": ctx, "nlev": case["nz"], "cfg": cfg}
    if kind == "press":
        for name, value in inp.items():
            _view(ctx, name).copy_(value)
        state["p"] = torch.zeros(cfg.nz + 1, cfg.ny, cfg.nx + 2, device="cuda", dtype=torch.float64)
        state["dpdx"], state["dpdy"] = torch.zeros_like(inp["u"]), torch.zeros_like(inp["u"])
    else:
        f = state["f"] = inp["f"]
        if kind == "dealias":
            state["big"] = torch.zeros(case["nz"], 3 * cfg.ny // 2, 3 * cfg.nx // 2 + 2, device="cuda", dtype=torch.float64)
            state["back"] = torch.zeros_like(f)
        else:
            state["dfdx"], state["dfdy"] = torch.zeros_like(f), torch.zeros_like(f)
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "step":
        (state["ctx"].step_graph if state["graph"] else state["ctx"].step)(CYCLE)
        return state["out"]
    if kind == "ensemble":
        state["ensemble"].step(CYCLE)
        return state["out"]
    ctx, nlev = state["ctx"], state["nlev"]
    if kind == "ddxy":
        ctx.call("ddxy", state["dfdx"], state["dfdy"], state["f"], ints=(nlev,))
        return {"dfdx": state["dfdx"], "dfdy": state["dfdy"]}
    if kind == "filt_da":   # in place; the filter leaves a filtered field as it is
        ctx.call("filt_da", state["f"], state["dfdx"], state["dfdy"], ints=(nlev,))
        return {"f": state["f"], "dfdx": state["dfdx"], "dfdy": state["dfdy"]}
    if kind == "dealias":
        ctx.call("dealias1", state["f"], state["big"], ints=(nlev,))
        ctx.call("dealias2", state["back"], state["big"], ints=(nlev,))
        return {"big": state["big"], "back": state["back"]}
    ctx.call("press_stag_array", state["p"], state["dpdx"], state["dpdy"])
    n = state["cfg"].nz   # the top level of each array is a filler that no caller reads
    return {"p": state["p"][:n], "dpdx": state["dpdx"][:n - 1], "dpdy": state["dpdy"][:n - 1]}


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _fft(nx, ny):
    """Operations of one real plane transform."""
    return 2.5 * nx * ny * math.log2(nx * ny)


def _step_work(nx, ny, nz, scalars, cycle=CYCLE):
    pts, nf = nx * ny * nz, 3 + scalars
    # prognostic fields and their last right-hand sides read and written each step; the Lagrangian averages, the
    # coefficient and the path sums read and written once a cycle
    nbytes = 8 * pts * (cycle * 4 * nf + 2 * 8)
    # plane transforms a level: velocities and scalars with their gradients, stress and flux divergences, vorticity and
    # products on the 3/2 grid, the pressure; the dynamic model's filters once a cycle
    small = 9 + 3 + 6 + 3 + 5 + scalars * 7
    big = 9 + 4 * scalars
    lag = 21 + 42
    return {"bytes": nbytes, "flops": nz * (cycle * (small * _fft(nx, ny) + big * _fft(1.5 * nx, 1.5 * ny)) + lag * _fft(nx, ny))}


def work(case):
    kind = case["kind"]
    if kind == "step":
        return _step_work(case["nx"], case["ny"], case["nz"], int(case["theta"]) + int(case["humid"]))
    if kind == "ensemble":
        w = [_step_work(*s, 1) for s in _sizes(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    plane, one = 8 * nx * ny, _fft(nx, ny)
    if kind == "ddxy":
        return {"bytes": 3 * plane * nz, "flops": 3 * one * nz}
    if kind == "filt_da":
        return {"bytes": 4 * plane * nz, "flops": 4 * one * nz}
    if kind == "dealias":
        big = _fft(1.5 * nx, 1.5 * ny)
        return {"bytes": (1 + 2.25 * 2 + 1) * plane * nz, "flops": 2 * (one + big) * nz}
    return {"bytes": 6 * plane * nz, "flops": 6 * one * nz}


# ---- the routines in plain torch, 64 bits --------------------------------------------------------------------------------
def _waves(cfg):
    kx = torch.arange(cfg.nx // 2 + 1, device="cuda", dtype=torch.float64) * (2 * math.pi / cfg.l_x)
    ky = torch.fft.fftfreq(cfg.ny, 1.0 / cfg.ny, device="cuda", dtype=torch.float64) * (2 * math.pi / cfg.l_y)
    kx, ky = kx[None, :].repeat(cfg.ny, 1), ky[:, None].repeat(1, cfg.nx // 2 + 1)
    keep = torch.ones_like(kx)
    keep[:, -1] = 0.0
    keep[cfg.ny // 2] = 0.0
    return kx * keep, ky * keep, keep


def _padded(a):
    return torch.nn.functional.pad(a, (0, 2))


def _back(h, cfg):
    """Inverse transform of normalised coefficients, with the zero padding columns."""
    return _padded(torch.fft.irfft2(h, s=(cfg.ny, cfg.nx), norm="forward"))


def _exact_press(cfg, inp):
    nx, ny, nz = cfg.nx, cfg.ny, cfg.nz
    dz = cfg.lz_over_zi / (nz - 1)
    kx, ky, keep = _waves(cfg)
    hat = {k: torch.fft.rfft2(inp[k][:, :, :nx], norm="forward") * keep for k in inp}
    hx, hy, hz = (hat[k] / (TADV1 * cfg.dt) for k in ("u", "v", "w"))
    hz[nz - 1] = 0.0
    bot, top = hat["divtz"][0], hat["divtz"][nz - 1]
    # rows 0..nz of each mode: -p0 + p1 = -dz bot;  second difference - k^2 p = divergence;  -p(nz-1) + p(nz) = -dz top
    r = torch.empty(nz + 1, ny, nx // 2 + 1, device="cuda", dtype=torch.complex128)
    r[0], r[nz] = -dz * bot, -dz * top
    r[1:nz] = 1j * (kx * hx[:-1] + ky * hy[:-1]) + (hz[1:] - hz[:-1]) / dz
    k2 = kx * kx + ky * ky
    k2[(k2 == 0)] = 1.0   # the mean and the removed modes: set below
    off, diag = 1.0 / (dz * dz), -(k2 + 2.0 / (dz * dz))
    gam, p = [None] * (nz + 1), torch.empty_like(r)
    bet = -torch.ones_like(k2)
    p[0] = r[0] / bet
    for j in range(1, nz + 1):
        a, b, c_prev = (off, diag, off if j > 1 else 1.0) if j < nz else (-1.0, 1.0, off)
        gam[j] = c_prev / bet
        bet = b - a * gam[j]
        p[j] = (r[j] - a * p[j - 1]) / bet
    for j in range(nz - 1, -1, -1):
        p[j] -= gam[j + 1] * p[j + 1]
    p *= keep
    p[0, 0, 0] = 0.0
    p[1, 0, 0] = -dz * bot[0, 0]
    for j in range(2, nz + 1):
        p[j, 0, 0] = p[j - 1, 0, 0] + hz[j - 1, 0, 0] * dz
    return {"p": _back(p[:nz], cfg), "dpdx": _back(1j * kx * p[1:nz], cfg), "dpdy": _back(1j * ky * p[1:nz], cfg)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "ensemble"):   # a whole time step of the model has no short restatement
        return None
    cfg, inp = _routine_inputs(case, seed)
    if kind == "press":
        return _exact_press(cfg, inp)
    nx, ny = cfg.nx, cfg.ny
    h = torch.fft.rfft2(inp["f"][:, :, :nx], norm="forward")
    if kind == "dealias":
        nx2, ny2, half = 3 * nx // 2, 3 * ny // 2, ny // 2
        hb = torch.zeros(h.shape[0], ny2, nx2 // 2 + 1, device="cuda", dtype=torch.complex128)
        hb[:, :half, :nx // 2] = h[:, :half, :nx // 2]
        hb[:, ny2 - half + 1:, :nx // 2] = h[:, half + 1:, :nx // 2]
        _, _, keep = _waves(cfg)
        return {"big": _padded(torch.fft.irfft2(hb, s=(ny2, nx2), norm="forward")), "back": _back(h * keep, cfg)}
    kx, ky, keep = _waves(cfg)
    out = {"dfdx": _back(1j * kx * h, cfg), "dfdy": _back(1j * ky * h, cfg)}
    if kind == "filt_da":
        out["f"] = _back(h * keep, cfg)
    return out
