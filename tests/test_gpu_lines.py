"""Transforms on register lines: every length they take, both
Hartley forms, against the oracle and a direct linear convolution.

Tolerances are the ones the right-hand side and the convolutions are held to
elsewhere: 1e-10 in FP64, 1e-5 in the mixed form, of the largest value.
"""
import json
import os

import numpy as np
import pytest

from fastisostasy_gb300.isostasy import Domain
from harness import rel
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")
TOL = {0: 1e-10, 1: 1e-5}


def _domain(name, nx, ny, precision):
    with open(os.path.join(GOLDEN, "params_%s.json" % name)) as fh:
        p = json.load(fh)
    p.update(min_pad=0.0, nx_target=nx if nx != ny else 0, ny_target=ny if nx != ny else 0)
    dom = Domain(p, nx, ny, 50e3, precision=precision)
    assert (dom.nx, dom.ny) == (nx, ny)
    return dom, p


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny,even", [(32, 2048, False), (32, 2048, True), (64, 1024, False), (128, 512, True),
                                        (512, 32, False), (1024, 16, True), (2048, 64, False), (256, 48, False),
                                        (2048, 34, True), (48, 1536, False), (1536, 96, True), (384, 192, False),
                                        (768, 24, True), (96, 768, False)])
def test_rate_on_lines(nx, ny, even, precision):
    _check_rate(nx, ny, even, precision)


@pytest.mark.parametrize("nx,ny,even", [(384, 768, False), (768, 384, True), (192, 1536, True), (1536, 192, False),
                                        (512, 768, True), (340, 768, False)])
def test_rate_on_double_lines_of_three_times_a_power(nx, ny, even):
    """FP64 lines of 3 2^k points, taken from 131,072 points of the half
    spectrum on (the last size has a few less)."""
    _check_rate(nx, ny, even, 0)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny,even", [(70, 44, True), (50, 98, False), (154, 26, False), (34, 250, True),
                                        (122, 142, False)])
def test_rate_with_odd_radices(nx, ny, even, precision):
    """Radices 5 and 7 in registers, larger primes by the symmetry of their roots."""
    _check_rate(nx, ny, even, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny,even", [(66, 46, True), (46, 58, False), (76, 26, False), (136, 74, True)])
def test_rate_with_primes_around_the_one_pass_limit(nx, ny, even, precision):
    """11, 13, 17, 19 and 23 take one pass in the mixed form, 29 and 37 two."""
    _check_rate(nx, ny, even, precision)


def _check_rate(nx, ny, even, precision):
    dom, p = _domain("test1d", nx, ny, precision)
    rng = np.random.default_rng(nx + ny)
    w, cf = rng.standard_normal((ny, nx)) * 100, rng.standard_normal((ny, nx)) * 1e5
    D, eta = 1e24 * (1 + rng.random((ny, nx))), 1e21 * (1 + rng.random((ny, nx)))
    R = np.ones((ny, nx)) if even else 1 + 0.2 * rng.random((ny, nx))
    mask = (rng.random((ny, nx)) > 0.15).astype(np.uint8)
    dom.set_fields(D_lith=D, eta_eff=eta, R=R, maskactive=mask)
    dxm = np.full((ny, nx), 50e3)
    ref = O.lvelva(w, cf, mask, p["g"], p["nu"], D, eta, R, dom.field("kappa"), dxm, dxm,
                   dom.scalars()["sec_per_year"])
    assert rel(dom.lvelva(w, cf), ref) <= TOL[precision]
    dom.close()


def linear_convolution(G, x):
    """The linear convolution, the mean of its four extreme lags subtracted, cropped around the centre."""
    ny, nx = x.shape
    s = (2 * ny, 2 * nx)
    full = np.fft.irfft2(np.fft.rfft2(G, s) * np.fft.rfft2(x, s), s)[:2 * ny - 1, :2 * nx - 1]
    full = full - 0.25 * (full[0, 0] + full[-1, -1] + full[-1, 0] + full[0, -1])
    return full[ny // 2 - 1:ny // 2 - 1 + ny, nx // 2 - 1:nx // 2 - 1 + nx]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny", [(2048, 32), (32, 2048), (16, 16), (512, 64), (64, 1024), (1536, 48), (48, 1536), (192, 96)])
def test_convolution_on_lines(nx, ny, precision):
    dom, _ = _domain("test2c", nx, ny, precision)
    x = np.random.default_rng(nx).standard_normal((ny, nx)) * 1e7
    for k, G in ((0, dom.field("GE")), (1, dom.field("GN"))):
        assert rel(dom.convolve(k, x), linear_convolution(G, x)) <= TOL[precision]
    dom.close()


def test_convolution_of_a_domain_that_does_not_convolve():
    """Green's functions and spectra made on demand equal those of a domain whose updates use them."""
    got = []
    for name in ("test2c", "test1d"):
        dom, p = _domain(name, 48, 48, 0)
        assert bool(p["include_elastic"] or p["heterogeneous_ssh"]) == (name == "test2c")
        x = np.random.default_rng(1).standard_normal((48, 48)) * 1e7
        got.append([dom.convolve(0, x), dom.convolve(1, x), dom.field("GE"), dom.field("GN")])
        dom.close()
    for a, b in zip(*got):
        assert rel(a, b) <= 1e-13
