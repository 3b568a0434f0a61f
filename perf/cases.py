"""Timed cases of the LV-ELVA library: what a coupled ice-sheet program, an
ensemble run and a solve server have it do.

A case is a dict of plain values.  ``kind`` says which public entry points it
goes through:

``couple``    one domain of the reference's call surface: ``isos_update`` (all
              of ``isos%out`` in ordinary numpy arrays) or ``Domain.update``
              into page-locked arrays, once per coupling interval, the ice load
              in host memory and changing from interval to interval
``async``     one domain driven without waiting: ``update_async`` with the ice
              thickness on the device and an ``output_async`` snapshot
``ensemble``  members of several sizes advanced in lockstep by ``Ensemble``
``serve``     a burst of independent solves through ``Server``
``rate``      one right-hand side, ``fi_lvelva_static``, on device arrays

Fields of the FP64 form are returned as they come (float64).  The mixed form
evaluates its right-hand sides in FP32 and its fields are good to single
precision; the programs that use it hold bed and sea level in single precision
and take them over as such, so a mixed case returns float32.

The inputs are synthetic: a fractal bed, an ice dome whose place and size
depend on the seed, a lithosphere and mantle that vary laterally.  Spacing and
step keep every explicit step inside its stability region, as a user has to.
"""
import ctypes
import math

import numpy as np
import torch

from fastisostasy_gb300 import _lib
from fastisostasy_gb300 import isostasy as fi
from fastisostasy_gb300 import params as fi_params
from fastisostasy_gb300.serve import Ensemble, Server
from fastisostasy_gb300.workloads import Workload

YEAR = float(np.float32(3600.0 * 24.0) * np.float32(365.25))   # s, as the reference rounds it
RESULT = ("w", "we", "z_bed", "z_ss")                          # what an ice model takes from a coupling step
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, kind, n, **over):
    c = dict(name=name, kind=kind, nx=n, ny=n, precision=1, dt_method=1, stage_mode=1, dx=25e3, dt=1.0, dtt=10.0,
             elastic=False, sealevel=False, distorted=False, rheology="random", nx_pad=0, ny_pad=0, pinned=False,
             members=0)
    c.update(over)
    return c


def listed():
    return [
        # a regional model or a served request: the smallest domain, every call waited for
        _case("couple_64", "couple", 64),
        # the reference's own disc experiment: 121^2 at 50 km, FP64, its adaptive integrator; 122 = 2 * 61 cells
        _case("disc_121_fp64", "couple", 121, precision=0, dt_method=2, stage_mode=0, dx=50e3, rheology="uniform"),
        # the adaptive pair with true stages, at an ensemble member's size
        _case("adaptive_true_192", "couple", 192, dt_method=2, dt=0.5),
        # laterally variable lithosphere, elastic and geoid on: regional and continental size
        _case("couple_256", "couple", 256, dx=11.71875e3, elastic=True, rheology="thinned"),
        _case("couple_512", "couple", 512, dx=11.71875e3, elastic=True, rheology="thinned", pinned=True),
        _case("couple_512_fp64", "couple", 512, precision=0, dx=11.71875e3, elastic=True, rheology="thinned",
              pinned=True),
        # a Greenland-like domain: 336 x 560 ice grid in 512 x 1024, interactive sea level, layered mantle
        _case("greenland_512x1024", "couple", 336, ny=560, dx=16e3, dt=0.5, dtt=5.0, elastic=True, sealevel=True,
              rheology="layered", nx_pad=512, ny_pad=1024, pinned=True),
        # a large FP64 domain that never waits for its output
        _case("async_1024_fp64", "async", 1024, precision=0, dx=11.71875e3, elastic=True, rheology="thinned"),
        # the largest domain
        _case("couple_2048", "couple", 2048, dx=11.71875e3, elastic=True, rheology="thinned", pinned=True),
        # an ensemble over rheology, load and grid size, batched
        _case("ensemble_24", "ensemble", 128, dt_method=2, stage_mode=0, dt=0.5, members=24),
        # a burst of independent solves of 2 to 8 coupling steps: set-up, steps and result of each
        _case("serve_12", "serve", 64, members=12),
        # one right-hand side of a caller that may not allocate, on a distorted grid
        _case("rate_256", "rate", 256, precision=0, distorted=True),
    ]


def _smooth(n):
    """The next even size without a prime factor above 7, as large grids are laid out."""
    n = int(n) + int(n) % 2
    while True:
        m = n
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        if m == 1:
            return n
        n += 2


def _size(rng, lo, hi):
    """A side length, spread over its logarithm; any size where grids are small."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if n <= 200 else min(hi, _smooth(n))


def draw(rng):
    kind = rng.choice(["couple"] * 6 + ["async", "ensemble", "serve", "rate"])
    if kind == "rate":
        c = _case("", kind, 2 * rng.randint(16, 128), precision=0, distorted=rng.random() < 0.5)
        c["ny"] = 2 * rng.randint(16, 128)
        c["nx_pad"], c["ny_pad"] = c["nx"], c["ny"]
    elif kind == "ensemble":
        c = _case("", kind, 64 * rng.randint(1, 2), dt_method=2, stage_mode=0, dt=0.5, members=rng.randint(4, 24))
    elif kind == "serve":
        c = _case("", kind, rng.choice([48, 64, 80]), members=rng.randint(2, 12))
    else:
        prec = rng.choice([0, 1, 1]) if kind == "couple" else 0
        method, stage = rng.choice([(1, 1), (1, 1), (1, 1), (2, 0), (2, 1), (0, 1)])
        if kind == "async":
            method, stage = 1, 1
        top = (1024 if prec == 0 else 2048) if method != 2 else 512
        n = _size(rng, 48, top)
        c = _case("", kind, n, precision=prec, dt_method=method, stage_mode=stage,
                  dx=round(rng.uniform(24e3, 40e3), 1), elastic=rng.random() < 0.5,
                  rheology=rng.choice(["random", "thinned", "layered"]), pinned=rng.random() < 0.5,
                  dt=0.5 if method != 1 else 1.0)
        if c["rheology"] == "layered":
            c["dt"], c["dtt"] = c["dt"] / 2, c["dtt"] / 2
        if rng.random() < 0.35:                      # a rectangle, padded as asked
            c["ny"] = max(32, int(n * rng.uniform(0.4, 1.0)))
            c["nx_pad"] = _smooth(n + 8) if n > 200 else n + n % 2 + 2 * rng.randint(0, 6)
            c["ny_pad"] = _smooth(c["ny"] + 8) if c["ny"] > 200 else c["ny"] + c["ny"] % 2 + 2 * rng.randint(0, 6)
            c["nx_pad"], c["ny_pad"] = min(2048, c["nx_pad"]), min(2048, c["ny_pad"])
        c["sealevel"] = c["nx_pad"] > 0 and rng.random() < 0.5
        c["distorted"] = prec == 0 and rng.random() < 0.3
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _noise(ny, nx, filt, gen):
    z = torch.randn((ny, nx), generator=gen, dtype=torch.float64, device=DEV)
    kx = 2 * math.pi * torch.fft.fftfreq(nx, dtype=torch.float64, device=DEV)
    ky = 2 * math.pi * torch.fft.fftfreq(ny, dtype=torch.float64, device=DEV)
    k = torch.sqrt(kx[None, :] ** 2 + ky[:, None] ** 2)
    f = torch.fft.ifft2(torch.fft.fft2(z) * filt(k)).real
    return (f - f.mean()) / f.std()


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _params(c):
    p = dict(fi_params.DEFAULTS)
    p.update(nu=0.28, rho_litho=3200.0, rho_uppermantle=3300.0, dt_method=c["dt_method"], stage_mode=c["stage_mode"],
             include_elastic=int(c["elastic"]), heterogeneous_ssh=int(c["elastic"]),
             interactive_sealevel=int(c["sealevel"]), min_pad=400e3 if c["sealevel"] else 0.0,
             nx_target=c["nx_pad"], ny_target=c["ny_pad"], dt_diagnostics=c["dtt"], precision=c["precision"])
    if c["dt_method"] != 2:
        p.update(dt_init=c["dt"], dt_max=c["dt"])
    elif c["rheology"] != "uniform":
        p.update(dt_init=c["dt"] / 4, dt_max=c["dt"], atol=0.1)   # the controller's step stays a stable one
    if c["rheology"] == "uniform":
        p.update(zl=[88e3], viscosities=[1e21])
    elif c["rheology"] == "layered":
        p.update(nl=2, zl=[100e3, 400e3], viscosities=[1e20, 1e21], lumping=5)
    else:
        p.update(lithosphere=3, mantle=3, zl=[150e3])
    return p


def _padded(c, p):
    """(nx, ny, first ice column, first ice row) of the padded domain."""
    out = []
    for n, target, other in ((c["nx"], c["nx_pad"], c["ny"]), (c["ny"], c["ny_pad"], c["nx"])):
        m = n + n % 2
        if c["nx_pad"] and c["ny_pad"]:
            pad = (target - m) // 2
        else:
            pad = int(math.floor(p["min_pad"] / c["dx"] + 0.5)) + max(0, (other + other % 2 - m) // 2)
        out.append((m + 2 * pad, pad + n % 2))
    return out[0][0], out[1][0], out[0][1], out[1][1]


def _rheology(c, nx, ny, gen):
    """Padded rigidity and viscosity of the laterally variable mantles, {} where the library makes them."""
    E, nu, dx = 66e9, 0.28, c["dx"]
    if c["rheology"] in ("uniform", "layered"):
        return {}
    if c["rheology"] == "thinned":
        x = (torch.arange(1, nx + 1, dtype=torch.float64, device=DEV) - nx // 2 - 1) * dx
        y = (torch.arange(1, ny + 1, dtype=torch.float64, device=DEV) - ny // 2 - 1) * dx
        he = 150e3 - 100e3 * torch.exp(-(x[None, :] ** 2 + y[:, None] ** 2) / (2 * 500e3 ** 2))
        eta = torch.full((ny, nx), 1e21, dtype=torch.float64, device=DEV)
    else:
        corr = 500e3 / dx
        smooth = lambda k: torch.exp(-(k * corr) ** 2 / 4)   # noqa: E731
        he = torch.clamp(85e3 + 15e3 * _noise(ny, nx, smooth, gen), 50e3, 120e3)
        eta = 10.0 ** torch.clamp(21 + 0.25 * _noise(ny, nx, smooth, gen), 20.3, 21.7)
    return {"D_lith": E * he ** 3 / (12 * (1 - nu ** 2)), "eta_eff": eta}


def _inputs(c, seed):
    """Bed, four ice loads of one advance and retreat, rheology and distortion of one domain."""
    gen, rng = _gen(seed), np.random.default_rng(int(seed))
    p = _params(c)
    nx, ny, i0, j0 = _padded(c, p)
    bed = _noise(c["ny"], c["nx"], lambda k: torch.where(k > 0, 1 / torch.clamp(k, min=1e-9), 0.0), gen) * 500 + 200
    x = torch.linspace(-1, 1, c["nx"], dtype=torch.float64, device=DEV)[None, :] - rng.uniform(-0.15, 0.15)
    y = torch.linspace(-1, 1, c["ny"], dtype=torch.float64, device=DEV)[:, None] - rng.uniform(-0.15, 0.15)
    r = rng.uniform(0.35, 0.6)
    dome = rng.uniform(1500.0, 3000.0) * torch.sqrt(torch.clamp(1 - (x ** 2 + y ** 2) / r ** 2, min=0.0))
    ice = [f * torch.where(bed > -50.0, dome, 0.0) for f in (0.7, 1.0, 0.85, 0.55)]
    K = None
    if c["distorted"]:                               # a polar stereographic projection's scale factor
        xx = (torch.arange(nx, dtype=torch.float64, device=DEV) - (nx - 1) / 2) * c["dx"]
        yy = (torch.arange(ny, dtype=torch.float64, device=DEV) - (ny - 1) / 2) * c["dx"]
        K = 0.97 * (1 + (xx[None, :] ** 2 + yy[:, None] ** 2) / (4 * 6378e3 ** 2))
    return dict(p=p, nx=nx, ny=ny, i0=i0, j0=j0, bed=bed, ice=ice, K=K, fields=_rheology(c, nx, ny, gen))


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.pin_memory().numpy() if torch.cuda.is_available() else t.numpy()


def _member_case(c, i, seed):
    """Member i of an ensemble: its own grid size, spacing and rheology."""
    n = (1, 2, 1, 3, 1, 2)[i % 6] * c["nx"]
    return dict(c, nx=n, ny=n, dx=float(np.random.default_rng([int(seed), i]).uniform(24e3, 30e3)))


def _member(c, i, seed):
    m = _member_case(c, i, seed)
    q = _inputs(m, 1000 * int(seed) + i)
    fields = {k: _host(v) for k, v in q["fields"].items()}
    return Workload(name="member_%d" % i, params=q["p"], nx_ice=m["nx"], ny_ice=m["ny"], dx=m["dx"],
                    z_bed=_host(q["bed"]), H_final=_host(q["ice"][1]), dtt=c["dtt"], t_end=c["dtt"],
                    fields_fn=lambda nx, ny, dx, f=fields: f)


class State:
    """What the program keeps from one coupling step to the next."""


def prepare(case, seed):
    s = State()
    s.case, s.t, s.step = case, 0.0, 0
    if case["kind"] == "ensemble":
        s.ens = Ensemble([_member(case, i, seed) for i in range(case["members"])], precision=case["precision"],
                         groups=2 if case["members"] > 8 else 1)
        s.ens.first_update(case["dtt"])
        s.t = case["dtt"]
        s.bufs = [torch.empty(d.output_bytes() // 8, dtype=torch.float64).pin_memory() for d in s.ens.doms]
        return s
    if case["kind"] == "serve":
        s.srv = Server(max_inflight=16, reserve_gb=1.0)
        s.reqs = [s.srv.prepare(_member(case, i, seed), t_end=case["dtt"] * (2 + i % 7), precision=case["precision"])
                  for i in range(case["members"])]
        return s
    if case["kind"] == "rate":
        q = _inputs(case, seed)
        gen, nx, ny = _gen(seed + 7), q["nx"], q["ny"]
        s.lib = _lib.load()
        s.dims, s.mask = (nx, ny), torch.ones((ny, nx), dtype=torch.uint8, device=DEV)
        s.D, s.eta = q["fields"]["D_lith"].contiguous(), q["fields"]["eta_eff"].contiguous()
        s.kappa = _kappa(nx, ny, case["dx"])
        s.R = 1 + 0.2 * torch.rand((ny, nx), generator=gen, dtype=torch.float64, device=DEV)
        s.w = 100 * _noise(ny, nx, lambda k: torch.exp(-(k * 8) ** 2), gen)
        s.load = 1e5 * _noise(ny, nx, lambda k: torch.exp(-(k * 4) ** 2), gen)
        s.dxm = None if q["K"] is None else (case["dx"] * q["K"]).contiguous()
        s.out = torch.empty((ny, nx), dtype=torch.float64, device=DEV)
        return s
    q = _inputs(case, seed)
    s.isos, s.bsl = fi.IsosClass(), fi.BslClass()
    fi.bsl_init(s.bsl, method="const")
    fi.isos_init(s.isos, None, "isostasy", case["nx"], case["ny"], case["dx"], case["dx"], params=q["p"],
                 K=None if q["K"] is None else _host(q["K"]), precision=case["precision"])
    if q["fields"]:
        s.isos.dom.set_fields(**{k: _host(v) for k, v in q["fields"].items()})
    zero = np.zeros((case["ny"], case["nx"]))
    fi.isos_init_state(s.isos, _host(q["bed"]), zero, 0.0, s.bsl)
    if case["kind"] == "async":
        s.ice = [h.contiguous() for h in q["ice"]]
        s.buf = torch.empty((11, case["ny"], case["nx"]), dtype=torch.float64).pin_memory()
    elif case["pinned"]:
        s.ice = [_pinned(_host(h)) for h in q["ice"]]
        s.out = {k: _pinned(zero) for k in RESULT}
    else:
        s.ice = [_host(h) for h in q["ice"]]
    return s


def _taken(out, case):
    """The fields an ice model takes over: FP64 as they are, mixed in single precision; FP64 runs take the masks too."""
    r = {k: torch.from_numpy(out[k]) for k in RESULT}
    if case["precision"]:
        return {k: v.to(torch.float32) for k, v in r.items()}
    r.update({k: torch.from_numpy(out[k]) for k in ("dwdt", "maskocean", "maskgrounded") if k in out})
    return r


def run(s):
    c = s.case
    if c["kind"] == "rate":
        ptr = lambda a: None if a is None else ctypes.c_void_p(a.data_ptr())   # noqa: E731
        rc = s.lib.fi_lvelva_static(ptr(s.w), ptr(s.load), ptr(s.mask), ptr(s.D), ptr(s.eta), ptr(s.kappa), ptr(s.R),
                                    ptr(s.dxm), ptr(s.dxm), s.dims[0], s.dims[1], c["dx"], c["dx"], 9.81, 0.28, YEAR,
                                    ptr(s.out), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("fi_lvelva_static: %d" % rc)
        return s.out
    if c["kind"] == "serve":
        ids = [s.srv.submit_prepared(q) for q in s.reqs]
        for i in ids:
            s.srv.wait(i)
        return [[torch.from_numpy(a).to(torch.float32) for a in s.srv.result(i)] for i in ids]
    s.t += c["dtt"]
    s.step += 1
    if c["kind"] == "ensemble":
        s.ens.update(s.t)
        s.ens.synchronize()
        for d, b in zip(s.ens.doms, s.bufs):
            d.output_async(b.data_ptr())
        for d in s.ens.doms:
            d.output_wait()
        got = []
        for d, b in zip(s.ens.doms, s.bufs):
            a = b.view(11, d.ny_ice, d.nx_ice)
            got.append(torch.stack([a[0], a[3]]).to(torch.float32))   # z_bed, w
        return got
    H = s.ice[s.step % len(s.ice)]
    if c["kind"] == "async":
        s.isos.dom.update_async(H.data_ptr(), s.t, s.bsl.c)
        s.isos.dom.output_async(s.buf.data_ptr())
        return dict(zip(s.isos.dom.OUTPUT_FIELDS, s.buf))
    if c["pinned"]:
        s.isos.dom.update(H, s.t, s.bsl.c, out=s.out)
        return _taken(s.out, c)
    fi.isos_update(s.isos, H, s.t, s.bsl)
    return _taken(s.isos.out, c)


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _domain_work(c, fields_out):
    """Compulsory traffic and arithmetic of one coupling step of one domain."""
    p = _params(c)
    nx, ny = _padded(c, p)[:2]
    n, ni = nx * ny, c["nx"] * c["ny"]
    f = 4 if c["precision"] else 8
    steps = max(1, int(round(c["dtt"] / (c["dt"] if c["rheology"] != "uniform" else 10.0))))
    rhs = steps * {0: 1, 1: 4 if c["stage_mode"] else 1, 2: 6 if c["stage_mode"] else 1}[c["dt_method"]]
    fft = 5.0 * n * math.log2(n)                      # a real transform forth and back
    flops = rhs * (fft + 70.0 * n)
    # state in and out, bed, reference, sea level and geoid; D, 1/(2 eta), 1/(kappa R), mask; the load and the outputs
    byts = n * (8 * 8 + 3 * f + 1) + 8.0 * ni * (1 + fields_out)
    if c["elastic"]:
        flops += 2 * (5.0 * 4 * n * math.log2(4.0 * n))
        byts += 2 * (2 * nx * ny * 2 * f + n * 8)     # the two kernel spectra, we and dz_ss
    return {"bytes": byts, "flops": flops}


def work(case):
    if case["kind"] == "rate":
        n = case["nx"] * case["ny"]
        return {"bytes": n * (8.0 * (8 if case["distorted"] else 7) + 1), "flops": 5.0 * n * math.log2(n) + 70.0 * n}
    if case["kind"] in ("ensemble", "serve"):
        got = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["members"]):
            w = _domain_work(dict(_member_case(case, i, 1)), 2 if case["kind"] == "serve" else 11)
            for k in got:
                got[k] += w[k] * ((2 + i % 7) if case["kind"] == "serve" and k == "flops" else 1)
        return got
    return _domain_work(case, 11 if case["kind"] == "async" or not case["pinned"] else len(RESULT))


# ---------------------------------------------------------------------------
# The same steps in plain torch, 64 bits
# ---------------------------------------------------------------------------
_RN = (0.0, 0.011, 0.111, 1.112, 2.224, 3.336, 4.448, 6.672, 8.896, 11.12, 17.79, 22.24, 27.80, 33.36, 44.48, 55.60,
       66.72, 88.96, 111.2, 133.4, 177.9, 222.4, 278.0, 333.6, 444.8, 556.0, 667.2, 778.4, 889.6, 1001.0, 1112.0,
       1334.0, 1779.0, 2224.0, 2780.0, 3336.0, 4448.0, 5560.0, 6672.0, 7784.0, 8896.0, 10008.0)
_GE = (-33.6488, -33.64, -33.56, -32.75, -31.86, -30.98, -30.12, -28.44, -26.87, -25.41, -21.80, -20.02, -18.36,
       -17.18, -15.71, -14.91, -14.41, -13.69, -13.01, -12.31, -10.95, -9.757, -8.519, -7.533, -6.131, -5.237, -4.660,
       -4.272, -3.999, -3.798, -3.640, -3.392, -2.999, -2.619, -2.103, -1.530, -0.292, 0.848, 1.676, 2.083, 2.057,
       1.643)


def _f32(x):
    return float(np.float32(x))


def _kappa(nx, ny, dx):
    pi = _f32(3.14159265359)

    def axis(n):
        i = torch.arange(1, n + 1, dtype=torch.float64, device=DEV)
        mu = 2 * pi / ((n - 1) * dx)
        return torch.where(i <= (n - 1) // 2 + 1, mu * (i - 1), mu * (n - i + 1))
    k = torch.sqrt(axis(nx)[None, :] ** 2 + axis(ny)[:, None] ** 2)
    k[0, 0] = (k[1, 0] + k[0, 1]) / 2
    return k.contiguous()


def _corner(a, ny, nx):
    return 0.25 * (a[0, 0] + a[ny - 1, nx - 1] + a[ny - 1, 0] + a[0, nx - 1])


def _d1(u, h):
    d = torch.empty_like(u)
    d[:, 1:-1] = (u[:, 2:] - u[:, :-2]) / (2 * h[:, 1:-1])
    d[:, 0] = (u[:, 1] - u[:, 0]) / h[:, 0]
    d[:, -1] = (u[:, -1] - u[:, -2]) / h[:, -1]
    return d


def _d2(u, h, last):
    d = torch.empty_like(u)
    d[:, 1:-1] = (u[:, 2:] - 2 * u[:, 1:-1] + u[:, :-2]) / h[:, 1:-1] ** 2
    d[:, 0] = (u[:, 2] - 2 * u[:, 1] + u[:, 0]) / h[:, 0] ** 2
    d[:, -1] = (u[:, -1] - 2 * u[:, -2] + u[:, -3]) / h[:, last] ** 2
    return d


def _rate(w, load, D, eta, m, h, nu, g):
    """calc_lvelva with m = 1/(kappa R); the load is zero where the mask is off."""
    t = lambda a: a.transpose(0, 1)   # noqa: E731
    dy = lambda u: t(_d1(t(u), t(h)))   # noqa: E731
    dyy = lambda u: t(_d2(t(u), t(h), -1))   # noqa: E731
    wxx, wyy, wxy = _d2(w, h, 0), dyy(w), dy(_d1(w, h))
    f = -g * load + _d2(-D * (wxx + nu * wyy), h, 0) + dyy(-D * (wyy + nu * wxx))
    f = (f + 2 * dy(_d1(-D * (1 - nu) * wxy, h))) / (2 * eta)

    def dht(a):
        F = torch.fft.fft2(a)
        return torch.roll(torch.flip(F.real, (0,)), 1, 0) - F.imag
    f = dht(dht(f) * m) / f.numel()
    return (f - _corner(f, *f.shape)) * YEAR


class _Exact:
    def __init__(self, c, q):
        p, nx, ny, dx = q["p"], q["nx"], q["ny"], c["dx"]
        self.c, self.p, self.nx, self.ny = c, p, nx, ny
        z = lambda v=0.0: torch.full((ny, nx), v, dtype=torch.float64, device=DEV)   # noqa: E731
        self.win = (slice(q["j0"], q["j0"] + c["ny"]), slice(q["i0"], q["i0"] + c["nx"]))
        K = q["K"] if q["K"] is not None else z(1.0)
        self.h, self.A, self.K2 = dx * K, (dx * K) ** 2, K ** 2
        kap, self.g = _kappa(nx, ny, dx), p["g"]
        he = p["zl"][0]
        self.D = q["fields"].get("D_lith", z(p["E"] * 1e9 * he ** 3 / (12 * (1 - p["nu"] ** 2))))
        R = z(1.0)
        if "eta_eff" in q["fields"]:
            self.eta = q["fields"]["eta_eff"]
        else:
            e = p["viscosities"][-1] * p["viscosity_scaling"]
            self.eta = z(math.exp(math.log10(p["eta_ref"] / e)) * e)
            if p["nl"] == 2:
                er, d = p["viscosities"][0] / p["viscosities"][1], p["zl"][1] - p["zl"][0]
                k, s, ch = d * kap, torch.sinh(d * kap), torch.cosh(d * kap)
                R = (2 * er * ch * s + (1 - er * er) * k * k + (er * s) ** 2 + ch * ch) / (
                    (er + 1 / er) * ch * s + (er - 1 / er) * k + s * s + ch * ch)
        self.m = 1 / (kap * R)
        self.active = z(1.0) > 0
        if p["interactive_sealevel"]:
            self.active = z() > 0
            if p["min_pad"] > 100e3:
                self.active[self.win] = True
        self.bed_ref = z(1e6)
        self.bed_ref[self.win] = q["bed"]
        self.bed, self.w, self.x, self.we, self.dz, self.dwdt = self.bed_ref.clone(), z(), z(), z(), z(), z()
        self.t, self.dt, self.t_diag, self.mantle = 0.0, p["dt_init"], 0.0, z()
        self.green = None
        if p["include_elastic"]:
            P = 2 * max(nx, ny)
            ax = lambda n: (torch.arange(n, dtype=torch.float64, device=DEV) - nx // 2) * dx   # noqa: E731
            r = torch.sqrt(ax(nx)[None, :] ** 2 + ax(ny)[:, None] ** 2)
            rn = torch.tensor([float(np.float32(v) * np.float32(1e3)) for v in _RN], dtype=torch.float64, device=DEV)
            ge = torch.tensor([_f32(v) for v in _GE], dtype=torch.float64, device=DEV)
            k = torch.clamp(torch.searchsorted(rn, r, right=True) - 1, 0, 40)
            v = ge[k] + (r - rn[k]) / (rn[k + 1] - rn[k]) * (ge[k + 1] - ge[k])
            v = torch.where(r > rn[41], 0.0, v) * _f32(1e-12) * (dx * dx) / (_f32(9.81) * torch.clamp(r, min=dx))
            gn = p["r_earth"] / (2 * p["m_earth"] * torch.sin(torch.clamp(r, min=dx / 2) / (2 * p["r_earth"])))
            self.green = [torch.fft.rfft2(a, s=(P, P)) for a in (v, gn)]
            self.P = P

    def conv(self, i, a):
        full = torch.fft.irfft2(self.green[i] * torch.fft.rfft2(a, s=(self.P, self.P)), s=(self.P, self.P))
        j, k, e = self.ny // 2 - 1, self.nx // 2 - 1, 2 * max(self.nx, self.ny) - 1
        return full[j:j + self.ny, k:k + self.nx] - _corner(full, e, e)

    def rhs(self, y, mantle):
        load = torch.where(self.active, self.base + mantle, 0.0)
        return _rate(y, load, self.D, self.eta, self.m, self.h, self.p["nu"], self.g)

    def update(self, ice, tf):
        p, c = self.p, self.c
        H = torch.zeros_like(self.w)
        H[self.win] = ice
        frac = p["rho_seawater"] / p["rho_ice"]
        zss = self.dz.clone()
        haf = torch.clamp(H - torch.clamp((zss - self.bed) * frac, min=0.0), min=0.0)
        ref = torch.clamp(-torch.clamp(-self.bed_ref * frac, min=0.0), min=0.0)
        grounded = (H > 0) & (haf > 0)
        ocean = lambda s: ~((self.bed > s) | grounded)   # noqa: E731

        def columns(s):
            a = p["rho_ice"] * (haf - ref)
            if p["interactive_sealevel"]:
                a = a + torch.where(ocean(s), p["rho_water"] * s, 0.0)
            return torch.where(self.active, a, 0.0)
        a = columns(zss)
        diag = tf - self.t_diag >= _f32(1e-3)
        if diag:
            self.t_diag += p["dt_diagnostics"]
            if p["include_elastic"]:
                self.we = self.conv(0, a * p["g"] * self.K2)
        litho = p["rho_litho"] * self.we
        if diag and p["heterogeneous_ssh"]:
            self.dz = self.conv(1, self.A * torch.where(self.active, a + litho + self.mantle, 0.0))
        zss = self.dz.clone()
        self.base = columns(zss) + litho
        if p["stage_mode"] == 1:
            f = lambda y: self.rhs(y, p["rho_uppermantle"] * y)   # noqa: E731
        else:
            f = lambda y: self.rhs(y, self.mantle)   # noqa: E731
        k0, tries = None, 0
        while self.t < tf:
            tries += 1
            if p["dt_method"] == 0:
                self.dt = min(self.dt, tf - self.t)
                self.dwdt = f(self.x if p["stage_mode"] else self.w)
                self.x = self.x + self.dt * self.dwdt
                self.w, self.t = self.x, self.t + self.dt
            elif p["dt_method"] == 1:
                h = min(self.dt, tf - self.t)
                k1 = f(self.x)
                k2 = f(self.x + 0.5 * h * k1)
                k3 = f(self.x + 0.5 * h * k2)
                self.dwdt = f(self.x + h * k3)
                self.x = self.x + h / 6 * (k1 + 2 * k2 + 2 * k3 + self.dwdt)
                self.w, self.t = self.x, self.t + h
            else:
                self.dt = h = min(self.dt, tf - self.t)
                if p["stage_mode"] == 0:
                    if k0 is None:
                        k0 = self.dwdt = f(self.w)
                    x2, x1 = self.x + h * k0, self.x + h * (1 - 0.2) * k0
                else:
                    A = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
                         (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
                         (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
                         (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
                    b = (5179 / 57600, 0.0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40)
                    k = [k0 if k0 is not None else f(self.x)]
                    for row in A:
                        x2 = self.x + h * sum(r * v for r, v in zip(row, k))
                        k.append(f(x2))
                    self.dwdt = k[6]
                    x1 = self.x + h * sum(r * v for r, v in zip(b, k))
                tol = p["atol"] + p["rtol"] * max(float(x1.abs().max()), float(x2.abs().max()))
                err = float(torch.sqrt((((x2 - x1) / tol) ** 2).sum() / x1.numel()))
                if err < 1:
                    self.x = self.w = x2
                    self.t, self.dt = self.t + h, min(h / max(err, 1e-300), p["dt_max"])
                    k0 = k[6] if p["stage_mode"] else None
                else:
                    self.dt *= 0.5
                    k0 = k[0] if p["stage_mode"] else k0
            if tries > 4000:
                return None
        self.w = self.w - _corner(self.w, self.ny, self.nx)
        self.mantle = p["rho_uppermantle"] * self.w
        self.bed = self.bed_ref + self.w + self.we
        return {k: v[self.win].cpu() for k, v in dict(w=self.w, we=self.we, z_bed=self.bed, z_ss=zss, dz_ss=self.dz,
                                                      dwdt=self.dwdt).items()}


def exact(case, seed):
    if case["kind"] == "rate":
        s = prepare(case, seed)
        h = s.dxm if s.dxm is not None else torch.full_like(s.w, case["dx"])
        return _rate(s.w, s.load, s.D, s.eta, 1 / (s.kappa * s.R), h, 0.28, 9.81)
    if case["kind"] in ("ensemble", "serve"):
        got = []
        for i in range(case["members"]):
            c = _member_case(case, i, seed)
            q = _inputs(c, 1000 * int(seed) + i)
            model, steps = _Exact(c, q), 2 if case["kind"] == "ensemble" else 2 + i % 7
            for k in range(steps):
                r = model.update(q["ice"][1], (k + 1) * case["dtt"])
            got.append(torch.stack([r["z_bed"], r["w"]]) if case["kind"] == "ensemble" else [r["w"], r["z_bed"]])
        return got
    q = _inputs(case, seed)
    r = _Exact(case, q).update(q["ice"][1], case["dtt"])
    if r is None:
        return None
    if case["kind"] == "async":
        return {k: r.get(k) for k in fi.Domain.OUTPUT_FIELDS}
    got = {k: r[k] for k in RESULT}
    if not case["precision"] and not case["pinned"]:
        got.update(dwdt=r["dwdt"], maskocean=None, maskgrounded=None)
    return got
