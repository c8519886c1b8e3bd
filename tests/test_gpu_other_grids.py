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
    (3, 48, 48): (1.36e-9, 1.28e-7, 7.9e-8, 5.5e-16, 2.5e-2, 1.5e-2),
    (3, 64, 96): (7.8e-10, 7.8e-8, 4.5e-8, 6.3e-16, 1.2e-3, 2.1e-3),
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
