"""The measurement hook counts every launch of a family in a step, whichever of the context's streams it is on.

A mixed step's transforms with 8-byte reals, x passes (y passes): the filtered surface u, v, 2 (1); the wall planes of
du/dz, dv/dz and of the stress divergence, 1 (1) each; the mean wind's linear terms, 2 (1); the pressure, 3 (3).  With
theta its wall planes, 1 (1).
"""
import ctypes

import pytest

import les_gb300 as lg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [0, 1])
@pytest.mark.parametrize("family,per_step", [(3, 9), (1, 7)])
def test_counts_every_stream(gpu_lib, theta, family, per_step):
    cfg = lg.make_config(32, s_flag=theta, precision=1, rmsdiv_every=0)
    surf = lg.striped_surface(cfg) if theta else lg.uniform_surface(cfg)
    g = lg.Context(cfg, surf)
    for k, v in lg.initial_state(cfg, surf, seed=3).items():
        g.set(k, v)
    g.step(1)
    n, ms, by = ctypes.c_int(), ctypes.c_double(), ctypes.c_double()
    lg.check(g.L.les_profile_begin(g.h, family, 64))
    g.step(2)
    lg.check(g.L.les_profile_end(g.h, ctypes.byref(n), ctypes.byref(ms), ctypes.byref(by)))
    assert n.value == 2 * (per_step + theta)
    assert ms.value > 0.0 and by.value > 0.0
    g.close()
