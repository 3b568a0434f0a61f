"""Which of the three steppers a mixed domain takes (one thread-block cluster,
the grid-wide step engine, one kernel a pass), and the step engine against the
oracle on each of its forms: register lines in its phases, and shared-memory
stages for lengths without one.

The bound is the mixed form's, 1e-5 of the largest displacement.
"""
import ctypes as C

import pytest

from fastisostasy_gb300.isostasy import Domain
from harness import Pair, rel
from test_gpu_cluster import workload

pytestmark = pytest.mark.gpu
RK4, TSIT, TSIT_TRUE = dict(dt_method=1), dict(dt_method=2, stage_mode=0), dict(dt_method=2, stage_mode=1)
SMALL = [(16, 16), (18, 18), (34, 34), (50, 50), (64, 64), (48, 80), (96, 96), (64, 20), (256, 32), (32, 256), (128, 192),
         (192, 128), (384, 48), (192, 192), (128, 128)]


@pytest.mark.parametrize("stepper,par,sizes", [
    ("cluster", RK4, SMALL), ("cluster", TSIT, SMALL + [(256, 256)]), ("cluster", TSIT_TRUE, SMALL + [(256, 256)]),
    ("engine", RK4, [(256, 256), (80, 60), (100, 100), (200, 200), (384, 384), (512, 512), (32, 512), (512, 128)]),
    ("kernels", RK4, [(64, 1024), (1024, 512), (640, 640)]),
    ("kernels", TSIT_TRUE, [(100, 100), (200, 200), (384, 384), (512, 128)]),
], ids=["cluster-rk4", "cluster-tsit54", "cluster-tsit54-true", "engine-rk4", "kernels-rk4", "kernels-tsit54-true"])
def test_stepper_of_a_size(stepper, par, sizes):
    for nx, ny in sizes:
        wl = workload(nx, ny, 1, True, **par)
        dom = Domain(wl.params, nx, ny, wl.dx, precision=1)
        assert dom.metrics()["stepper"] == stepper, (nx, ny)
        dom.close()


def check_engine(nx, ny, even):
    pair = Pair(workload(nx, ny, 5 * nx + ny, even), precision=1)
    m = pair.dom.metrics()
    assert m["stepper"] == "engine" and m["step_engine"]
    pair.init()
    pair.step(2)
    assert pair.dom.scalars()["t"] == pair.t and pair.dom.scalars()["n_accept"] == 20
    for f in ("w", "z_bed"):
        assert rel(pair.dom.field(f), pair.orc.field(f)) <= 1e-5
    assert rel(pair.dom.field("dwdt"), pair.orc.field("dwdt")) <= 1e-4
    pair.close()


@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("nx,ny", [(256, 256), (384, 256), (256, 384), (384, 384), (512, 384), (384, 512)])
def test_engine_on_lines(nx, ny, even):
    check_engine(nx, ny, even)


@pytest.mark.parametrize("nx,ny", [(50, 50), (66, 46), (100, 100), (122, 98), (76, 140), (200, 200), (464, 466),
                                   (72, 54), (144, 288), (216, 486)])
def test_engine_without_lines(monkeypatch, nx, ny):
    """Shared-memory stages, with radices 5, 7 and larger primes and of 2 and 3 only, two and four rows a block."""
    monkeypatch.setenv("FI_NO_CLUSTER", "1")
    check_engine(nx, ny, nx != 100)


@pytest.mark.parametrize("even", [True, False])
@pytest.mark.parametrize("nx,ny", [(4, 4), (8, 6), (12, 8), (16, 12), (24, 16), (32, 24), (48, 32), (64, 48), (96, 64),
                                   (128, 96), (192, 128), (384, 192), (512, 24), (768, 96), (1024, 48), (1024, 256),
                                   (4, 512), (16, 512), (32, 384), (512, 128), (768, 512), (24, 500)])
def test_engine_on_every_line(monkeypatch, nx, ny, even):
    """Every length of the line phases in both directions: several lines or
    columns in a warp, a line of two warps, grids wider than a block (and a last
    one with a column length that has no line)."""
    monkeypatch.setenv("FI_NO_CLUSTER", "1")
    check_engine(nx, ny, even)


@pytest.mark.parametrize("n", [32, 64, 192, 256])
def test_engine_trace(monkeypatch, n):
    """Traced updates stamp the engine's phases also where the domain otherwise
    steps in a cluster, and give its result within the mixed form's bound."""
    monkeypatch.setenv("FI_NO_GRAPHS", "1")
    pair = Pair(workload(n, n, n, True), precision=1)
    L = pair.dom.L
    pair.init()
    pair.step(1)
    assert pair.dom.metrics()["stepper"] == ("engine" if n == 256 else "cluster")
    buf = (C.c_ulonglong * 256)()
    assert L.fi_engine_trace(pair.dom.h, buf, 256) == 0
    pair.step(2)
    assert pair.dom.metrics()["stepper"] == "engine"
    assert L.fi_engine_trace(pair.dom.h, buf, 256) == 0
    stamps = [v for v in buf if v]
    # step begin and end, and for each of the four stages six phase boundaries
    assert len(stamps) >= 4 * 6 + 2 and stamps == sorted(stamps)
    assert stamps[-1] - stamps[0] < 1e9
    for f in ("w", "z_bed"):
        assert rel(pair.dom.field(f), pair.orc.field(f)) <= 1e-5
    assert pair.dom.scalars()["n_accept"] == 30
    pair.close()
