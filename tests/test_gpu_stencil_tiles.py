"""The mixed tile stencil (one kernel per pass, no step engine) against the
oracle at the edges of its 64 x 16 tiles: exactly one tile, last tiles of two
columns or two rows, grids smaller than a tile, and several tiles; first and
later RK4 stages, and Tsit5 with and without the mantle term at the stages.

The bound is the mixed form's, 1e-5 of the largest displacement.
"""
import pytest

from harness import Pair, rel
from test_gpu_cluster import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(4, 4), (16, 14), (64, 16), (62, 18), (66, 16), (66, 18), (130, 34), (128, 48)])
@pytest.mark.parametrize("par", [dict(dt_method=1), dict(dt_method=2, stage_mode=0, dt_init=8.0, dt_max=8.0),
                                 dict(dt_method=2, stage_mode=1, dt_init=8.0, dt_max=8.0)],
                         ids=["rk4", "tsit54", "tsit54-true"])
def test_tile_edges(monkeypatch, nx, ny, par):
    monkeypatch.setenv("FI_NO_ENGINE", "1")
    pair = Pair(workload(nx, ny, nx + 7 * ny, nx != 64, **par), precision=1)
    assert not pair.dom.metrics()["step_engine"]
    pair.init()
    pair.step(2)
    a, b = pair.dom.scalars(), pair.orc.scalars()
    assert a["t"] == pair.t and a["n_accept"] == b["n_accept"] and a["n_reject"] == b["n_reject"]
    for f in ("w", "z_bed"):
        assert rel(pair.dom.field(f), pair.orc.field(f)) <= 1e-5
    pair.close()


@pytest.mark.parametrize("nx,ny", [(6, 4), (32, 6), (34, 66), (66, 160), (224, 226), (322, 162), (512, 130)])
@pytest.mark.parametrize("par", [dict(dt_method=1), dict(dt_method=2, stage_mode=1, dt_init=8.0, dt_max=8.0)],
                         ids=["rk4", "tsit54-true"])
def test_fp64_tile_rows(nx, ny, par):
    """FP64 tiles of 4, 8 and 16 rows, with last tiles of two rows or columns;
    the FP64 form's bound."""
    pair = Pair(workload(nx, ny, nx + 9 * ny, nx != 34, **par), precision=0)
    pair.init()
    pair.step(2)
    a, b = pair.dom.scalars(), pair.orc.scalars()
    assert a["t"] == pair.t and a["n_accept"] == b["n_accept"] and a["n_reject"] == b["n_reject"]
    for f in ("w", "z_bed"):
        assert rel(pair.dom.field(f), pair.orc.field(f)) <= 1e-10
    pair.close()
