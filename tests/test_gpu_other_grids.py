"""The dynamic models away from 32 x 32: other even lengths, factors of 3, rectangles, against the CPU oracle.

Whole steps, ten of them from jt_total0 = 500 (two updates of Cs^2), are held to 1e-12 or a multiple of the oracle's own
rounding sensitivity on that grid (`python -m oracle.rounding_spread model<M>-<nx>x<ny>`: built with FMA contraction
against without): three times for the fields, ten times for Cs^2, which passes single-precision roundings.
"""
import numpy as np
import pytest

import les_gb300 as lg

pytestmark = pytest.mark.gpu

TOL = 1e-12
FIELDS = ("u", "v", "w", "theta")
# (model, nx, ny): spread of u, v, w, theta, Cs_opt2, rmsdiv
SPREAD = {
    (2, 48, 48): (9.2e-16, 2.9e-14, 7.3e-14, 5.7e-16, 1.6e-12, 6.6e-3),
    (2, 64, 96): (8.9e-16, 4.1e-14, 7.6e-14, 6.1e-16, 1.9e-12, 6.2e-3),
    (2, 96, 64): (8.2e-16, 3.6e-14, 8.5e-14, 5.5e-16, 8.9e-12, 1.1e-2),
    (3, 48, 48): (1.36e-9, 1.28e-7, 7.9e-8, 5.5e-16, 2.5e-2, 1.5e-2),
    (3, 64, 96): (7.8e-10, 7.8e-8, 4.5e-8, 6.3e-16, 1.2e-3, 2.1e-3),
    (4, 48, 48): (8.8e-16, 3.0e-14, 7.4e-14, 5.6e-16, 3.7e-11, 1.1e-2),
    (4, 64, 96): (9.4e-16, 4.2e-14, 7.8e-14, 5.9e-16, 2.8e-11, 1.1e-2),
    (5, 48, 48): (4.9e-15, 5.7e-13, 4.4e-13, 5.2e-16, 9.7e-11, 3.7e-3),
    (5, 64, 96): (6.3e-15, 8.7e-13, 7.2e-13, 2.0e-15, 3.8e-10, 1.2e-4),
    (5, 96, 64): (6.6e-15, 9.1e-13, 8.8e-13, 5.5e-16, 9.3e-10, 3.7e-3),
    (7, 48, 48): (3.3e-15, 2.5e-12, 1.1e-12, 1.6e-14, 3.4e-10, 3.6e-3),
    (7, 96, 64): (3.6e-15, 1.5e-12, 1.0e-12, 1.4e-14, 3.6e-10, 4.6e-3),
}


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def pair(cfg, surf, seed=11, levels=10):
    from oracle.oracle import Oracle
    Oracle.set_threads(max(1, Oracle.max_threads()))
    g, o = lg.Context(cfg, surf), Oracle(cfg, surf)
    for k, v in lg.initial_state(cfg, surf, seed=seed, theta_levels=levels).items():
        g.set(k, v)
        o.set(k, v)
    return g, o


@pytest.mark.parametrize("model,nx,ny", sorted(SPREAD))
def test_steps(gpu_lib, oracle_lib, model, nx, ny):
    cfg = lg.make_config(nx, ny, 32, s_flag=1, jt_total0=500, model=model, rmsdiv_every=1)
    g, o = pair(cfg, lg.striped_surface(cfg), levels=cfg.nz if model == 7 else 10)
    g.step(10)
    assert o.step(10) == 0
    lev = slice(0, cfg.nz - 1)
    for nm, spread in zip(FIELDS + ("Cs_opt2",), SPREAD[model, nx, ny]):
        e = rel(g.get(nm)[lev, :, :nx], o.get(nm)[lev, :, :nx])
        assert e < max(TOL, (10 if nm == "Cs_opt2" else 3) * spread), (nm, e)
    rg, ro = g.rmsdiv(), o.rmsdiv()
    if model == 3:  # runs with transforms that round as the oracle's: the divergence left is the oracle's too
        assert abs(rg - ro) < 10 * SPREAD[model, nx, ny][5] * ro, (rg, ro)
    else:
        assert rg < 1.1 * ro, (rg, ro)
    g.close()


@pytest.mark.parametrize("nx,ny", [(48, 48), (64, 96), (96, 64)])
def test_std_dynamic_routine(gpu_lib, oracle_lib, nx, ny):
    """Cs^2(z) of one call on smooth strain-like fields, whose plane sums cancel: the tolerance of the 32 x 32 case."""
    cfg = lg.make_config(nx, ny, 20, model=2, s_flag=0)
    g, o = pair(cfg, lg.uniform_surface(cfg), seed=5)
    rng = np.random.default_rng(6)
    shp = lg.field_shape(cfg, "u")
    X, Y = np.meshgrid(np.arange(nx) * 2 * np.pi / nx, np.arange(ny) * 2 * np.pi / ny)
    S = [np.zeros(shp) for _ in range(6)]
    for a in S:
        for k in range(shp[0]):
            a[k, :, :nx] = sum(rng.standard_normal() * np.cos(i * X + j * Y + rng.uniform(0, 6.3))
                               for i in range(4) for j in range(-3, 4)) / 10.0
    cg, co = np.zeros(cfg.nz), np.zeros(cfg.nz)
    g.call("std_dynamic", cg, *S)
    o.call("std_dynamic", co, *S)
    assert np.all(co >= 0) and np.any(co > 0)
    assert rel(cg, co) < TOL
    g.close()


def exact_press(cfg, u, v, w, divtz):
    """press_stag_array.f90 in extended precision: p on levels 0..nz-1, dp/dx and dp/dy on 1..nz-1."""
    L = np.longdouble
    nx, ny, nz = cfg.nx, cfg.ny, cfg.nz
    dz = L(cfg.lz_over_zi) / (nz - 1)
    kx = np.arange(nx // 2 + 1).astype(L)[None, :].repeat(ny, 0) * (2 * L(np.pi) / L(cfg.l_x))
    ky = (((np.arange(ny) + ny // 2) % ny) - ny // 2).astype(L)[:, None].repeat(nx // 2 + 1, 1) * (2 * L(np.pi) / L(cfg.l_y))
    keep = np.ones((ny, nx // 2 + 1))
    keep[ny // 2] = 0
    keep[:, -1] = 0
    kx, ky = kx * keep, ky * keep
    hx, hy, hz, d = (np.fft.rfft2(a[:, :, :nx].astype(L)) / (nx * ny) * keep for a in (u, v, w, divtz))
    hx, hy, hz = (h / (L(1.5) * L(cfg.dt)) for h in (hx, hy, hz))
    hz[nz - 1] = 0
    r = np.empty((nz + 1, ny, nx // 2 + 1), dtype=np.clongdouble)
    r[0], r[nz] = -dz * d[0], -dz * d[nz - 1]
    r[1:nz] = 1j * (kx * hx[:-1] + ky * hy[:-1]) + (hz[1:] - hz[:-1]) / dz
    k2 = kx * kx + ky * ky
    k2[k2 == 0] = 1
    off, diag = 1 / (dz * dz), -(k2 + 2 / (dz * dz))
    gam, p = [None] * (nz + 1), np.empty_like(r)
    bet = -np.ones_like(k2)
    p[0] = r[0] / bet
    for j in range(1, nz + 1):
        a, b, above = (off, diag, off if j > 1 else L(1)) if j < nz else (L(-1), L(1), off)
        gam[j] = above / bet
        bet = b - a * gam[j]
        p[j] = (r[j] - a * p[j - 1]) / bet
    for j in range(nz - 1, -1, -1):
        p[j] -= gam[j + 1] * p[j + 1]
    p *= keep
    p[0, 0, 0] = 0
    p[1, 0, 0] = -dz * d[0, 0, 0]
    for j in range(2, nz + 1):
        p[j, 0, 0] = p[j - 1, 0, 0] + hz[j - 1, 0, 0] * dz
    back = lambda h: np.fft.irfft2(h, s=(ny, nx)) * (nx * ny)
    return back(p[:nz]), back(1j * kx * p[1:nz]), back(1j * ky * p[1:nz])


@pytest.mark.parametrize("nx,ny", [(32, 32), (48, 48), (64, 96), (72, 64), (96, 64), (128, 128), (144, 64), (216, 32), (288, 64)])
def test_press_routine(gpu_lib, oracle_lib, nx, ny):
    """The pressure of a projected state, where it cancels most: no further from the exact result than the oracle's
    (whose own error is 1e-14 to 4e-11), on the small planes that keep its roundings up to 1e-12 of the result."""
    cfg = lg.make_config(nx, ny, 24, s_flag=1, rmsdiv_every=0)
    g, o = pair(cfg, lg.striped_surface(cfg), seed=17)
    assert o.step(6) == 0
    args = [o.get(nm) for nm in ("u", "v", "w", "divtz")]
    for nm, a in zip(("u", "v", "w", "divtz"), args):
        g.set(nm, a)
    want = exact_press(cfg, *args)
    shp = lg.field_shape(cfg, "u")
    err = []
    for c in (g, o):
        p, x, y = np.zeros(lg.field_shape(cfg, "p")), np.zeros(shp), np.zeros(shp)
        c.call("press_stag_array", p, x, y)
        got = (p[:cfg.nz, :, :nx], x[:cfg.nz - 1, :, :nx], y[:cfg.nz - 1, :, :nx])
        err.append([float(rel(a.astype(np.longdouble), b)) for a, b in zip(got, want)])
    for eg, eo in zip(*err):
        assert eg < (eo if max(nx, ny) > 32 else eo + TOL), err
    g.close()
