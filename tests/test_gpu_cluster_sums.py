"""Sums of the cluster's integrators that have to keep the digits of the other
paths.

A load that is the same everywhere has one value of the raw right-hand side, C,
in every cell (on a grid of powers of two each transform only adds equal numbers
or takes them from one another, which is exact), so with each stage's corner
mean taken off before the stages are summed the step is exactly zero.  Summed
first, C + 2 C + 2 C + C rounds at six times the size of C.
"""
import numpy as np
import pytest

from fastisostasy_gb300 import workloads as W
from fastisostasy_gb300.isostasy import Domain
from harness import gpu_bsl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stepper,nx,ny", [("cluster", 64, 64), ("cluster", 128, 32), ("cluster", 16, 256),
                                           ("engine", 256, 256), ("engine", 32, 512), ("kernels", 32, 1024)])
def test_uniform_load_moves_nothing(stepper, nx, ny):
    p = dict(W.P.DEFAULTS)
    p.update(E=66.0, nu=0.28, dt_method=1, dt_init=1.0, dt_max=1.0, stage_mode=1, rho_uppermantle=3300.0,
             nx_target=nx, ny_target=ny)
    dom = Domain(p, nx, ny, 30e3, precision=1)
    assert dom.metrics()["stepper"] == stepper
    one = np.ones((ny, nx))
    dom.set_fields(D_lith=4e24 * one, eta_eff=1.3e21 * one, R=one, maskactive=one.astype(np.uint8))
    b = gpu_bsl()
    dom.init_state(1e6 * one, 0 * one, 0.0, b)
    for k, H in enumerate((1000.0, 777.7, 1234.5, 3141.6, 271.8)):
        dom.update(H * one, 10.0 * (k + 1), b)
        assert dom.scalars()["n_accept"] == 10 * (k + 1)
        assert not dom.field("x").any() and not dom.field("w").any()
    dom.close()
