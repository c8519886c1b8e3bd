"""The float-float transforms of precision 2 (fft_fixed.cu, fft_kernels.cuh), which its step takes where the FP64
integer-pipe transforms do not cover the grid.

Each grid has one direction that they do not cover and one whose float-float kernels have a fixed length: 36 is outside
their x and their y lengths.  Tolerances are those of the form, 1e-12 relative L2 after ten steps against the oracle
(stated for its transforms of about 48 bits with the plane means taken out).
"""
import numpy as np
import pytest

import les_gb300 as lg
from les_gb300.config import moisture_flux

pytestmark = pytest.mark.gpu

TOL = 1e-12
RMSDIV_ABS = 1e-12


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nx,ny,q,jt0", [(36, 64, 0, 0), (64, 36, 0, 500), (36, 32, 1, 0), (96, 36, 0, 0),
                                         (36, 128, 0, 0), (128, 36, 0, 0)])
def test_step_against_oracle(gpu_lib, oracle_lib, nx, ny, q, jt0):
    from oracle.oracle import Oracle
    Oracle.set_threads(max(1, Oracle.max_threads()))
    cfg = lg.make_config(nx, ny, 24, s_flag=1, q_flag=q, jt_total0=jt0, rmsdiv_every=1, precision=2)
    surf = lg.striped_surface(cfg)
    g, o = lg.Context(cfg, surf), Oracle(cfg, surf)
    if q:
        wq = moisture_flux(cfg)
        g.set("wq_s", wq)
        o.set("wq_s", wq)
    for k, v in lg.initial_state(cfg, surf, seed=11).items():
        g.set(k, v)
        o.set(k, v)
    g.step(10)
    assert o.step(10) == 0
    for nm in ("u", "v", "w", "theta") + (("q",) if q else ()):
        e = rel(g.get(nm)[:-1, :, :nx], o.get(nm)[:-1, :, :nx])
        assert e < TOL, (nm, e)
    assert g.rmsdiv() < RMSDIV_ABS
    # not the FP64 form's step, which agrees with the oracle to a few roundings
    ref = lg.Context(lg.make_config(nx, ny, 24, s_flag=1, q_flag=q, jt_total0=jt0, rmsdiv_every=1, precision=0), surf)
    if q:
        ref.set("wq_s", wq)
    for k, v in lg.initial_state(cfg, surf, seed=11).items():
        ref.set(k, v)
    ref.step(10)
    assert not np.array_equal(g.get("w"), ref.get("w"))
    g.close()
    ref.close()
