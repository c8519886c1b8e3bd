"""The autotuner times what its knobs change and nothing else: on grids whose transforms all run on the integer pipe the
FP64 and float-float forms have nothing to tune, and the defaults come back without a probe."""
import pytest

import les_gb300 as lg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,precision,probes", [(64, 0, False), (64, 2, False), (36, 0, True), (36, 2, True), (64, 1, True)])
def test_probes(gpu_lib, nx, precision, probes):
    cfg = lg.make_config(nx, 48, 5, s_flag=1, precision=precision, rmsdiv_every=0)   # a size no other test tunes
    g = lg.Context(cfg, lg.striped_surface(cfg))
    n0 = g.L.les_kernel_launch_count()
    tuned = g.autotune()
    assert (g.L.les_kernel_launch_count() > n0) == probes
    if not probes:
        assert tuned["tx64"] == 4 and tuned["rpc_scale"] == 0
    g.close()
