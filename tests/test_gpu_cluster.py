"""Small mixed domains advanced in one thread-block cluster, against the
oracle: sizes at the edges of the row and column splits (odd multiples, two
rows a block, blocks without rows, lengths with and without a register line),
rectangles, a mask and both Hartley forms.

The bound is the mixed form's, 1e-5 of the largest displacement.
"""
import numpy as np
import pytest

from fastisostasy_gb300 import workloads as W
from harness import Pair, rel

pytestmark = pytest.mark.gpu


def workload(nx, ny, seed, even, **par):
    rng = np.random.default_rng(seed)
    p = dict(W.P.DEFAULTS)
    p.update(E=66.0, nu=0.28, dt_method=1, dt_init=1.0, dt_max=1.0, stage_mode=1, lithosphere=3, mantle=3,
             rho_uppermantle=3300.0, nx_target=nx, ny_target=ny)
    p.update(par)
    D = 4e24 * (1 + 0.5 * rng.random((ny, nx)))
    fields = {"D_lith": D, "eta_eff": 1e21 * (1 + 0.5 * rng.random((ny, nx))),
              "R": np.ones((ny, nx)) if even else 1 + 0.2 * rng.random((ny, nx)),
              "maskactive": (rng.random((ny, nx)) > 0.1).astype(np.uint8)}
    yy, xx = np.mgrid[0:ny, 0:nx]
    H = 1500.0 * np.exp(-((xx - 0.4 * nx) ** 2 + (yy - 0.55 * ny) ** 2) / (0.05 * nx * ny)) + 50 * rng.random((ny, nx))
    return W.Workload(name="cluster", params=p, nx_ice=nx, ny_ice=ny, dx=30e3, z_bed=np.full((ny, nx), 1e6), H_final=H,
                      fields=fields)


@pytest.mark.parametrize("nx,ny", [(16, 16), (18, 18), (34, 34), (50, 50), (64, 64), (48, 80), (96, 96), (64, 20),
                                   (256, 32), (32, 256), (128, 192), (192, 128), (384, 48), (256, 256)])
@pytest.mark.parametrize("even", [True, False])
def test_rk4_in_a_cluster(nx, ny, even):
    pair = Pair(workload(nx, ny, nx + 3 * ny, even), precision=1)
    assert pair.dom.metrics()["step_engine"]
    pair.init()
    pair.step(3)
    for f in ("w", "z_bed"):
        assert rel(pair.dom.field(f), pair.orc.field(f)) <= 1e-5
    assert rel(pair.dom.field("dwdt"), pair.orc.field("dwdt")) <= 1e-4
    assert pair.dom.scalars()["t"] == pair.t and pair.dom.scalars()["n_accept"] == 30
    pair.close()


def test_cluster_against_the_kernel_sequence(monkeypatch):
    """The same steps through the one-kernel-per-pass path, including an update
    cut short by its target time."""
    res = []
    for env in ("1", "0"):
        monkeypatch.setenv("FI_NO_ENGINE", env)
        pair = Pair(workload(64, 64, 5, True), precision=1)
        pair.wl.dtt = 2.5
        pair.init()
        pair.step(4)
        res.append(pair.dom.field("x"))
        assert pair.dom.scalars()["n_accept"] == 12
        pair.close()
    assert rel(res[1], res[0]) <= 1e-5


@pytest.mark.parametrize("nx,ny", [(16, 16), (34, 34), (64, 64), (96, 96), (64, 20), (32, 256), (128, 192), (192, 192),
                                   (256, 256)])
@pytest.mark.parametrize("stage_mode", [0, 1])
def test_tsit54_in_a_cluster(nx, ny, stage_mode):
    """Same attempts as the oracle, rejections among them, within the bound."""
    wl = workload(nx, ny, nx + 5 * ny, nx != 64, dt_method=2, stage_mode=stage_mode, dt_init=8.0, dt_max=8.0)
    pair = Pair(wl, precision=1)
    assert pair.dom.metrics()["step_engine"]
    pair.init()
    pair.step(3)
    a, b = pair.dom.scalars(), pair.orc.scalars()
    assert a["t"] == pair.t and a["n_accept"] == b["n_accept"] and a["n_reject"] == b["n_reject"]
    for f in ("w", "z_bed"):
        assert rel(pair.dom.field(f), pair.orc.field(f)) <= 1e-5
    pair.close()


def test_rejection_limit_in_a_cluster():
    """The step floor ends the update in every block alike: FI_E_STEP, and the domain answers on."""
    from fastisostasy_gb300 import _lib
    wl = workload(64, 64, 9, True, dt_method=2, stage_mode=0, dt_init=8.0, dt_max=8.0, dt_min=4.0, atol=1e-9, rtol=0.0)
    pair = Pair(wl, precision=1)
    pair.init()
    with pytest.raises(_lib.FiError) as e:
        pair.dom.update(wl.H_at(10.0), 10.0, pair.bg)
    assert e.value.code == _lib.FI_E_STEP
    assert pair.dom.scalars()["n_reject"] >= 1
    pair.close()
