"""Level-walking FP64 pointwise kernels (Nu_t and tau_ij, the convective
products) and the fused step around them on grids where a thread walks one
level and where it walks eight with a remainder, against the CPU oracle.

Tolerance: the FP64 parity tolerance of the step, 1e-12 relative L2 after
three steps.  The 256 x 256 grid has the blocks for eight levels a thread (27
levels: three full walks and a remainder); the small one walks single levels.
"""
import numpy as np
import pytest

import les_gb300 as lg

pytestmark = pytest.mark.gpu
TOL = 1e-12


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nx,ny,levels", [(64, 32, 5), (256, 256, 27)])
def test_step_walks(gpu_lib, oracle_lib, nx, ny, levels):
    from oracle.oracle import Oracle
    cfg = lg.make_config(nx, ny, levels, s_flag=1, rmsdiv_every=0)
    surf = lg.striped_surface(cfg)
    g, o = lg.Context(cfg, surf), Oracle(cfg, surf)
    for k, v in lg.initial_state(cfg, surf, seed=21).items():
        g.set(k, v)
        o.set(k, v)
    g.step(3)
    assert o.step(3) == 0
    for nm in ("u", "v", "w", "theta", "Nu_t", "txx", "txy", "tyy", "tzz", "txz", "tyz"):
        lev = slice(0, cfg.nz - 1)
        assert rel(g.get(nm)[lev, :, :nx], o.get(nm)[lev, :, :nx]) < TOL, nm
    g.close()
