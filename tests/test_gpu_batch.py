"""Batches of domains that run in the batched attempt loop beside domains that
make their whole update in a thread-block cluster of their own: each member's
result equals that of the member driven alone, with the default shapes and with
autotuned ones.

The mixed bound is the mixed form's, 1e-5 of the largest displacement (the
batched kernels are compiled apart from the single-domain ones, so the compiler
may fuse multiply-adds differently); FP64 members agree bit for bit.
"""
import numpy as np
import pytest

from fastisostasy_gb300.isostasy import Domain
from fastisostasy_gb300.serve import Ensemble
from harness import gpu_bsl
from test_gpu_cluster import workload

pytestmark = pytest.mark.gpu
TIMES = (10.0, 20.0, 30.0)


def member(nx, ny, stage_mode):
    """A member on nx x ny cells, with attempts that the first step sizes reject."""
    wl = workload(nx, ny, 3 * nx + ny, nx != 200, dt_method=2, stage_mode=stage_mode, dt_init=8.0, dt_max=8.0)
    wl.name = "member_%d_%d" % (nx, ny)
    return wl


def ensemble_w(wls, precision, autotune):
    ens = Ensemble(wls, precision=precision, mode="graph", autotune=autotune)
    ens.first_update(TIMES[0])
    for t in TIMES[1:]:
        ens.update(t)
    ens.synchronize()
    w = [d.field("w") for d in ens.doms]
    steppers = [d.metrics()["stepper"] for d in ens.doms]
    counts = [(d.scalars()["n_accept"], d.scalars()["n_reject"]) for d in ens.doms]
    ens.close()
    return w, counts, steppers


def alone_w(wl, precision):
    dom = Domain(wl.params, wl.nx_ice, wl.ny_ice, wl.dx, precision=precision)
    dom.set_fields(**wl.padded_fields(dom.nx, dom.ny))
    b = gpu_bsl()
    dom.init_state(wl.z_bed, np.zeros_like(wl.H_final), 0.0, b)
    for t in TIMES:
        dom.update(wl.H_final, t, b)
    w, sc = dom.field("w"), dom.scalars()
    dom.close()
    return w, (sc["n_accept"], sc["n_reject"])


def check(sizes, precision, stage_mode, autotune, clustered=False):
    wls = [member(nx, ny, stage_mode) for nx, ny in sizes]
    got, counts, steppers = ensemble_w(wls, precision, autotune)
    assert "kernels" in steppers and (precision == 0 or not clustered or "cluster" in steppers)
    for wl, g, c in zip(wls, got, counts):
        w, ca = alone_w(wl, precision)
        assert c == ca and np.abs(w).max() > 0, wl.name
        if precision == 1:
            assert np.abs(w - g).max() <= 1e-5 * np.abs(w).max(), wl.name
        else:
            assert np.array_equal(w, g), wl.name


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("stage_mode", [0, 1])
def test_cluster_members_beside_loop_members(stage_mode, autotune):
    """64^2 and 128^2 fit a cluster, 384^2 (register lines) and 200^2 (none) do not."""
    check([(64, 64), (384, 384), (128, 128), (200, 200)], 1, stage_mode, autotune, clustered=True)


@pytest.mark.parametrize("autotune", [False, True])
def test_fp64_members_on_lines_of_three_times_a_power(autotune):
    """Row lines of 8, 16 and 32 threads in one block (96, 192 and 384 points,
    each on a grid large enough for FP64 lines of that kind)."""
    check([(192, 1368), (384, 684), (768, 342)], 0, 0, autotune)


@pytest.mark.parametrize("rows,cols", [(3, 5), (5, 3), (1, 1), (16, 16), (7, 6)])
@pytest.mark.parametrize("precision,sizes", [(0, [(64, 2048), (128, 64), (40, 48)]),
                                             (1, [(64, 2048), (512, 256), (384, 384), (200, 200)])])
def test_any_rows_and_columns_a_block(monkeypatch, precision, sizes, rows, cols):
    """Block shapes asked for by the environment that are no powers of two, over
    lines of different lengths."""
    monkeypatch.setenv("FI_BATCH_RB", str(rows))
    monkeypatch.setenv("FI_BATCH_CB", str(cols))
    check(sizes, precision, 0, False)


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("stage_mode", [0, 1])
def test_small_members_in_the_loop(monkeypatch, stage_mode, autotune):
    """Members that would fit a cluster, batched (and driven alone) without it."""
    monkeypatch.setenv("FI_NO_CLUSTER", "1")
    check([(40, 40), (56, 34), (192, 192), (128, 96)], 1, stage_mode, autotune)
