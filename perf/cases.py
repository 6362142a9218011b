"""The framework's work as a user has it done, as cases that can be timed and compared.

Kinds of case, each one pass through a public entry point on device-resident inputs:

* ``step``      LW then SW radiation of one domain (``rrtmg_lwrad_wrf_columns`` and ``rrtmg_swrad_wrf_columns``);
* ``lw``, ``sw`` one of the two calls alone;
* ``infer``     the learned surrogate with its gate and (``fallback``) the plain-kernel fallback;
* ``train``     one Adam step of the surrogate's training, in the middle of a run;
* ``prologue``  cloud fraction, CAM ozone, cos zenith and the condensate flag in one call;
* ``tendency``  LW + SW heating coupled with the column mass and added to the theta tendency.

Column states follow the recipe of the package's seeded generator (``synthetic.make_columns``), drawn on the GPU.
A checkout need not hold the RRTMG data files, so the context is made from a seeded stand-in table set: the entries and
shapes of the real one, absorption coefficients spread over five decades across a band's g-points, standard-atmosphere
reference profiles, Planck integrals, Pade tables and single-scattering tables of ordinary magnitudes.  The kernels
gather from it exactly as from the real tables.
"""

from __future__ import annotations

import importlib.util
import math
import os
import sys
import tempfile
from pathlib import Path

import numpy as np
import torch

REPO = Path(__file__).resolve().parents[1]


def _package():
    """The package by path (its folder's name is not an identifier); compiled first where a checkout is not."""
    if "wrf_jax_b200" not in sys.modules:
        root = REPO / "wrf-jax_b200"
        spec = importlib.util.spec_from_file_location("wrf_jax_b200", root / "__init__.py",
                                                      submodule_search_locations=[str(root)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["wrf_jax_b200"] = mod
        spec.loader.exec_module(mod)
        from wrf_jax_b200 import build
        if not build.LIB.exists():
            build.build_library()
    return sys.modules["wrf_jax_b200"]


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _columns(kind, nx, ny, nk, **more):
    return dict(dict(kind=kind, nx=nx, ny=ny, nk=nk, p_top=5000.0, night=0.3, radii=False, fractional=False,
                     noahmp=False), **more)


def listed():
    return [
        # a single-column or unit-test sized model step: launches and latency only
        dict(_columns("step", 4, 4, 44), name="step_4x4x44"),
        # the small domain of the package's CPU workload, and one tile of a decomposed run
        dict(_columns("step", 64, 64, 44), name="step_64x64x44"),
        # odd extents and level count, a 20 hPa top, prescribed effective radii, fractional clouds, Noah-MP albedos
        dict(_columns("step", 97, 61, 57, p_top=2000.0, radii=True, fractional=True, noahmp=True),
             name="step_97x61x57_radii"),
        # the regional domain that the plain kernels are quoted on, each call by itself
        dict(_columns("lw", 425, 425, 50), name="lw_425x425x50"),
        dict(_columns("sw", 425, 425, 50), name="sw_425x425x50"),
        # surrogate radiation of one tile: the fallback's latency beside a short network pass
        dict(kind="infer", nx=64, ny=64, fallback=True, name="infer_64x64"),
        # a ragged domain, the network and gate alone
        dict(kind="infer", nx=423, ny=311, fallback=False, name="network_423x311"),
        # the surrogate's headline workload
        dict(kind="infer", nx=1000, ny=1000, fallback=True, name="infer_1000x1000"),
        # training: a small batch (fine tuning) and the batch of the shipped training run
        dict(kind="train", batch=1024, name="train_1024"),
        dict(kind="train", batch=16384, name="train_16384"),
        # the radiation stage's inputs before the calls, and its result's way into the dynamics
        dict(kind="prologue", nx=1000, nk=50, ny=1000, name="prologue_1000x50x1000"),
        dict(kind="tendency", nx=1000, nk=50, ny=1000, halo=0, name="tendency_1000x50x1000"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, ncol):
    """Two extents with a product of at most ncol, neither much longer than the other."""
    nx = max(1, int(math.sqrt(ncol) * math.exp(rng.uniform(-0.7, 0.7))))
    return nx, max(1, ncol // nx)


def draw(rng):
    kind = rng.choice(("step", "step", "lw", "sw", "infer", "infer", "train", "prologue", "tendency"))
    if kind in ("step", "lw", "sw"):
        nk = rng.randint(17, 60)
        most = 425 * 425 * 50 // (80 if kind == "step" else 40)
        nx, ny = _grid(rng, _logint(rng, 16, min(most, most * 35 // nk)))
        radii = rng.random() < 0.3
        return _columns(kind, nx, ny, nk, p_top=rng.choice((5000.0, 5000.0, 2000.0, 1000.0)),
                        night=rng.choice((0.3, 0.3, 0.5)), radii=radii, fractional=rng.random() < 0.3,
                        noahmp=kind != "lw" and rng.random() < 0.3)
    if kind == "infer":
        nx, ny = _grid(rng, _logint(rng, 1000, 1000000))
        return dict(kind=kind, nx=nx, ny=ny, fallback=rng.random() < 0.7)
    if kind == "train":
        return dict(kind=kind, batch=128 * _logint(rng, 4, 128))
    nx, ny = _grid(rng, _logint(rng, 1000, 1000000))
    nk = rng.randint(30, 60)
    nx = max(1, min(nx, 50 * 1000 * 1000 // (nk * ny)))
    case = dict(kind=kind, nx=nx, nk=nk, ny=ny)
    return dict(case, halo=rng.choice((0, 3))) if kind == "tendency" else case


# ---------------------------------------------------------------------------
# stand-in tables
# ---------------------------------------------------------------------------
_LW_NGC = (10, 12, 16, 14, 16, 8, 12, 8, 12, 6, 8, 8, 4, 2, 2, 2)
_SW_NGC = (6, 12, 8, 8, 10, 10, 2, 10, 8, 6, 6, 8, 6, 12)
_LW_BAND_EDGES = (10, 350, 500, 630, 700, 820, 980, 1080, 1180, 1390, 1480, 1800, 2080, 2250, 2380, 2600, 3250)


def _standard_temperature(p_hpa):
    return np.where(p_hpa > 200.0, 288.0 * (p_hpa / 1013.25) ** 0.19, np.where(p_hpa > 1.0, 217.0 + 50.0 * np.clip(
        np.log(20.0 / np.minimum(p_hpa, 20.0)) / 3.0, 0.0, 1.0), 260.0))


def _planck_table():
    """Planck radiance of each LW band over its width, W cm^-2 sr^-1 / cm^-1, at 160 .. 340 K."""
    t = np.arange(160.0, 341.0)[:, None]
    out = np.empty((181, 16))
    for b in range(16):
        lo, hi = _LW_BAND_EDGES[b:b + 2]
        v = (np.linspace(lo, hi, 65)[:-1] + (hi - lo) / 128.0)[None, :]
        out[:, b] = (1.191042972e-12 * v ** 3 / np.expm1(1.438777 * v / t)).mean(1)
    return out


def _gas_table(rng, shape, scale):
    """Absorption coefficients (..., ngc), rising over five decades across the g-points."""
    g = (np.arange(shape[-1]) + 0.5) / shape[-1]
    return scale * 10.0 ** (-3.5 + 5.0 * g) * rng.uniform(0.5, 1.5, shape)


def _band_tables(rng, prefix, records, ngc, t):
    share = np.linspace(2.0, 0.2, ngc)
    share /= share.sum()
    for name, kind, shape in records:
        if shape is None:
            value = dict(rayl=2.0e-9, strrat=5.0, strrat1=250.0, givfac=1.029, scalekur=50.15 / 48.37,
                         layreffr=18 if prefix != "sw27" else 32)[name]
            t[f"{prefix}.{name}"] = np.asarray([value], np.int32 if kind == "i" else np.float32)
            continue
        base = name[:2] + name[3:] if name.startswith(("kao_", "kbo_")) else name
        base = base[:-1] if base.endswith("o") and not name.startswith(("kao_", "kbo_")) else base
        if name in ("fracrefao", "fracrefbo", "sfluxrefo"):
            total = 1.0 if prefix.startswith("lw") else 100.0
            rest = shape[1:] or (1,)
            a = total * share[:, None] * rng.uniform(0.95, 1.05, (ngc,) + rest)
            a = a.reshape((ngc,) + tuple(shape[1:]))
        elif name in ("kao", "kbo"):
            rows = int(np.prod(shape[:-1]))
            # the shortwave bands are far more transparent than the longwave ones
            a = _gas_table(rng, (rows, ngc), (1.0e-2 if name == "kao" else 1.0) * (1.0 if prefix[0] == "l" else 2.0e-3))
        elif name in ("raylo", "raylao", "raylbo"):
            base = "rayl" if name == "raylo" else base
            a = 2.0e-9 * rng.uniform(0.5, 2.0, (ngc,) + tuple(shape[1:]))
        elif len(shape) == 1:
            a = _gas_table(rng, (ngc,), 1.0e-2)
        else:
            a = _gas_table(rng, tuple(shape[:-1]) + (ngc,), 1.0e-4 if "ref" in name else 1.0e-3)
        t[f"{prefix}.{base}"] = np.ascontiguousarray(a, np.float32)


def _tables(seed=7):
    from wrf_jax_b200 import tables
    rng = np.random.default_rng(seed)
    t = {}
    preflog = 6.96 - 0.2 * np.arange(59)
    pref = np.exp(preflog)
    tref = _standard_temperature(pref)
    t["lw.pref"], t["lw.preflog"], t["lw.tref"] = pref, preflog, tref
    t["sw.preflog"], t["sw.tref"] = preflog, tref
    h2o = np.maximum(1.9e-2 * np.exp(-2.6 * np.log(1013.0 / np.minimum(pref, 1013.0))), 4.0e-6)
    o3 = 3.0e-8 + 8.0e-6 * np.exp(-0.5 * (np.log(pref / 10.0) / 1.1) ** 2)
    one = np.ones(59)
    t["lw.chi_mls"] = np.stack([h2o, 3.55e-4 * one, o3, 3.2e-7 * one, 1.5e-7 * one, 1.7e-6 * one, 0.209 * one])
    t["lw.totplnk"] = _planck_table()
    # ice and liquid cloud optics per effective-size row and band
    size = np.arange(46)[:, None]
    t["lw.absice3"] = (0.2 / (1.0 + 0.15 * size)) * rng.uniform(0.8, 1.2, (1, 16)) + 0.0 * size
    t["lw.absliq1"] = (0.3 / (1.0 + 0.1 * np.arange(58)[:, None])) * rng.uniform(0.8, 1.2, (1, 16))
    t["sw.extliq1"] = (1.0 / (1.0 + 0.35 * np.arange(58)[:, None])) * rng.uniform(0.9, 1.1, (1, 14))
    t["sw.ssaliq1"] = rng.uniform(0.8, 0.9999, (1, 14)) - 0.001 * np.arange(58)[:, None]
    t["sw.asyliq1"] = 0.80 + 0.001 * np.arange(58)[:, None] + rng.uniform(0.0, 0.02, (1, 14))
    t["sw.extice3"] = (0.6 / (1.0 + 0.2 * size)) * rng.uniform(0.9, 1.1, (1, 14))
    t["sw.ssaice3"] = rng.uniform(0.7, 0.9999, (1, 14)) - 0.002 * size
    t["sw.asyice3"] = 0.72 + 0.003 * size + rng.uniform(0.0, 0.02, (1, 14))
    t["sw.fdlice3"] = 0.05 + 0.001 * size + rng.uniform(0.0, 0.02, (1, 14))
    # Pade interpolation tables: position i of 10000 stands for tau = bpade x / (1 - x), x = i / 10000
    bpade = 1.0 / 0.278
    x = np.arange(10001) / 10000.0
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        tau = bpade * x / (1.0 - x)
        tau[-1] = 1.0e10
        ex = np.maximum(np.exp(-tau), 1.0e-20)
        tfn = np.where(tau < 0.06, tau / 6.0, 1.0 - 2.0 * (1.0 / np.where(tau > 0, tau, 1.0) - ex / (1.0 - np.where(
            tau > 0, ex, 0.0))))
    t["lw.pade_bpade"], t["lw.pade_tau_tbl"], t["lw.pade_exp_tbl"], t["lw.pade_tfn_tbl"] = [bpade], tau, ex, tfn
    t["sw.pade_bpade"], t["sw.pade_tau_tbl"], t["sw.pade_exp_tbl"] = [bpade], tau, ex
    # profiles: ice radius by temperature, ozone climatologies, the LW buffer's standard atmosphere
    t["retab"] = 5.0 + 120.0 * (np.arange(95) / 94.0) ** 2
    level = np.geomspace(1000.0, 0.3, 31)
    for season, amp in (("sum", 1.0), ("win", 0.9)):
        t["o3" + season] = amp * (5.0e-8 + 1.2e-5 * np.exp(-0.5 * (np.log(level / 8.0) / 1.2) ** 2))
        t["pp" + season] = level * (1.0 if season == "sum" else 0.985)
    pprof = np.geomspace(1000.0, 0.1, 60)
    t["lw_buffer_pprof"], t["lw_buffer_tprof"] = pprof, _standard_temperature(pprof)
    t = {k: np.ascontiguousarray(np.asarray(v), np.float32) for k, v in t.items()}
    for side, records, counts, first in (("lw", tables._LW_RECORDS, _LW_NGC, 1), ("sw", tables._SW_RECORDS, _SW_NGC, 16)):
        for b, ngc in enumerate(counts):
            _band_tables(rng, f"{side}{first + b}", records[first + b], ngc, t)
        t[f"{side}.ngc"] = np.asarray(counts, np.int32)
        t[f"{side}.ngn"] = np.ones(sum(counts), np.int32)
    # binary64 logarithm and exponential: reciprocal and log of each interval's centre with a cubic, 2^(i/32) with a cubic
    first = np.uint32(0x3F330000)
    lo = (first + (np.arange(16, dtype=np.uint32) << np.uint32(19))).view(np.float32).astype(np.float64)
    hi = (first + (np.arange(1, 17, dtype=np.uint32) << np.uint32(19))).view(np.float32).astype(np.float64)
    centre = 0.5 * (lo + hi)
    t["glibc.logf_invc_logc"] = np.stack([1.0 / centre, np.log(centre)], 1)
    t["glibc.logf_ln2_poly"] = np.asarray([math.log(2.0), -0.25, 1.0 / 3.0, -0.5])
    powers = np.exp2(np.arange(32) / 32.0).view(np.uint64)
    t["glibc.expf_tab"] = powers - (np.arange(32, dtype=np.uint64) << np.uint64(47))
    step = math.log(2.0) / 32.0
    t["glibc.expf_invln2n_poly"] = np.asarray([1.0 / step, step ** 3 / 6.0, step ** 2 / 2.0, step])
    # binary32 sine and cosine: 1/pi, the rounding shift, pi in four parts of falling size, Taylor terms, the limit
    parts, rest = [], math.pi
    for _ in range(4):
        e = 2.0 ** (math.frexp(rest)[1] - 10)
        parts.append(math.trunc(rest / e) * e)
        rest -= parts[-1]
    shift, poly = 1.5 * 2.0 ** 23, [1.0 / 362880.0, -1.0 / 5040.0, 1.0 / 120.0, -1.0 / 6.0]
    t["svml.sinf"] = np.asarray([1.0 / math.pi, shift, shift, *parts, *poly, 1.0e4], np.float32)
    t["svml.cosf"] = np.asarray([math.pi / 2.0, 1.0 / math.pi, shift, shift, 0.5, *parts, *poly, 1.0e4], np.float32)
    return t


_KEPT = {}


def stand_in_blob():
    """Path of a table blob with the stand-in tables, written once per process."""
    if "blob" not in _KEPT:
        _package()
        from wrf_jax_b200 import tables
        fd, path = tempfile.mkstemp(suffix=".bin", prefix="rrtmg_tables_")
        os.close(fd)
        tables.write_blob(_tables(), path)
        _KEPT["blob"] = Path(path)
    return _KEPT["blob"]


def _context():
    """The process's radiation context (what a model keeps for its whole run), the default of every call."""
    if "ctx" not in _KEPT:
        path = stand_in_blob()
        from wrf_jax_b200 import prologue, rrtmg, synthetic, tables
        tables.DEFAULT_BLOB = path
        ctx = rrtmg.default_context()
        plev, lat, oz = synthetic.cam_ozone_climatology(seed=0)
        _KEPT["ozone"] = (np.asarray(plev, np.float32) * np.float32(100.0), lat, oz)
        prologue.set_ozone_climatology(*_KEPT["ozone"], context=ctx)
        os.unlink(path)
        del _KEPT["blob"]
        _KEPT["ctx"] = ctx
    return _KEPT["ctx"]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _Draws:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, device="cuda", generator=self.g) * (hi - lo) + lo

    def normal(self, sigma, *shape):
        return torch.randn(*shape, device="cuda", generator=self.g) * sigma


def _column_fields(case, seed):
    """Device fields of a domain, (nx, nk, ny) as the runtime holds them (the recipe of synthetic.make_columns)."""
    nx, ny, nk = case["nx"], case["ny"], case.get("nk", 50)
    p_top = case.get("p_top", 5000.0)
    r = _Draws(seed)
    s = torch.linspace(0.0, 1.0, nk + 1, device="cuda", dtype=torch.float64)
    eta = ((torch.exp(-3.0 * s) - math.exp(-3.0)) / (1.0 - math.exp(-3.0))).float().view(1, nk + 1, 1)
    psfc = r.uniform(95000.0, 103000.0, nx, 1, ny)
    p8w = p_top + eta * (psfc - p_top)
    p8w[:, nk] = p_top
    p3d = 0.5 * (p8w[:, :-1] + p8w[:, 1:])
    t3d = 288.0 * (p3d.clamp(min=20000.0) / 101325.0) ** 0.190263 + r.normal(2.0, nx, nk, ny)
    t8w = torch.empty(nx, nk + 1, ny, device="cuda")
    t8w[:, 1:nk] = 0.5 * (t3d[:, :-1] + t3d[:, 1:])
    t8w[:, 0] = 2.0 * t3d[:, 0] - t8w[:, 1]
    t8w[:, nk] = t3d[:, nk - 1]
    es = torch.minimum(610.78 * torch.exp(17.27 * (t3d - 273.16) / (t3d - 35.86)), 0.5 * p3d)
    qv = r.uniform(0.2, 1.0, nx, nk, ny) * (0.622 * es / (p3d - 0.378 * es))
    del es
    o3 = 8.0e-6 * torch.exp(-0.5 * (torch.log(p3d / 1000.0) / 1.1) ** 2) + 3.0e-8
    cloudy = ((r.uniform(0.0, 1.0, nx, nk, ny) < 0.3) & (p3d > 30000.0)).float()
    frac = cloudy * r.uniform(0.05, 1.0, nx, nk, ny) if case.get("fractional") else cloudy
    coszr = r.uniform(0.0, 1.0, nx, ny)
    coszr[r.uniform(0.0, 1.0, nx, ny) < case.get("night", 0.3)] = 0.0
    zero3, zero2 = torch.zeros_like(p3d), torch.zeros(nx, ny, device="cuda")
    radii = case.get("radii", False)
    f = dict(p3d=p3d, p8w=p8w, pi3d=(p3d / 1.0e5) ** (287.0 / 1004.5), t3d=t3d, t8w=t8w,
             tsk=t3d[:, 0] + r.uniform(-3.0, 3.0, nx, ny), dz8w=torch.full_like(p3d, 250.0), qv3d=qv,
             qc3d=cloudy * r.uniform(0.0, 5.0e-4, nx, nk, ny), qi3d=cloudy * r.uniform(0.0, 2.0e-4, nx, nk, ny),
             qs3d=cloudy * r.uniform(0.0, 1.0e-4, nx, nk, ny) if radii else zero3, cldfra3d=frac, o33d=o3,
             emiss=r.uniform(0.9, 1.0, nx, ny), albedo=r.uniform(0.05, 0.4, nx, ny), coszr=coszr,
             xland=1.0 + (r.uniform(0.0, 1.0, nx, ny) < 0.3).float() if radii else zero2 + 1.0, xice=zero2, snow=zero2,
             re_cloud=r.uniform(2.5e-6, 20.0e-6, nx, nk, ny) if radii else zero3,
             re_ice=r.uniform(5.0e-6, 100.0e-6, nx, nk, ny) if radii else zero3,
             re_snow=r.uniform(10.0e-6, 200.0e-6, nx, nk, ny) if radii else zero3)
    if case.get("noahmp"):
        for k in ("alswvisdir", "alswvisdif", "alswnirdir", "alswnirdif"):
            f[k] = r.uniform(0.05, 0.4, nx, ny)
    return {k: v.contiguous() for k, v in f.items()}


def _state_of(case, fields):
    from wrf_jax_b200 import synthetic
    h = 1 if case.get("radii") else 0
    scalars = dict(p_top=float(case.get("p_top", 5000.0)), yr=2024, julian=172.5, solcon=1326.5, has_reqc=h,
                   has_reqi=h, has_reqs=h, **synthetic.GASES)
    return synthetic.ColumnState(fields=fields, scalars=scalars, nx=case["nx"], ny=case["ny"], nk=case.get("nk", 50))


def _model():
    from wrf_jax_b200 import surrogate
    return surrogate.SurrogateModel.load(REPO / "wrf-jax_b200" / "weights" / "surrogate_nk50.npz")


_CALENDAR = dict(julian=172.5, xtime=720.0, gmt=6.0, yr=2024, radt=30.0)


def prepare(case, seed):
    _package()
    kind = case["kind"]
    ctx = _context()
    if kind in ("step", "lw", "sw"):
        fields = _column_fields(case, seed)
        st = _state_of(case, fields)
        albedos = {k: fields[k] for k in fields if k.startswith("alsw")}
        sw = st.sw_kwargs()
        if albedos:
            sw.update(sf_surface_physics=8, **albedos)
        return dict(kind=kind, ctx=ctx, lw=st.lw_kwargs(), sw=sw)
    if kind == "infer":
        fields = _column_fields(case, seed)
        if "model" not in _KEPT:
            _KEPT["model"] = _model()
        return dict(kind=kind, model=_KEPT["model"], st=_state_of(case, fields), d=fields, fallback=case["fallback"])
    if kind == "train":
        from wrf_jax_b200 import surrogate
        r = _Draws(seed)
        batch = case["batch"]
        rows = max(4096, 8 * batch)
        X = torch.zeros(rows, surrogate.K_IN, device="cuda", dtype=torch.bfloat16)
        X[:, :surrogate.N_FEATURES] = r.normal(1.0, rows, surrogate.N_FEATURES).bfloat16()
        mix = r.normal(surrogate.N_FEATURES ** -0.5, surrogate.N_FEATURES, surrogate.N_OUT)
        T = torch.tanh(X[:, :surrogate.N_FEATURES].float() @ mix) + r.normal(0.3, rows, surrogate.N_OUT)
        T[:, surrogate.N_TARGETS:] = 0.0
        model = _model()
        for w, m, v in list(zip(model.w, model.mw, model.vw)) + list(zip(model.b, model.mb, model.vb)):
            # moments of a run in progress: gradients of the batch's order of magnitude
            m.copy_(r.normal(3.0e-5, *w.shape))
            v.copy_(r.uniform(0.5e-8, 2.0e-8, *w.shape))
        idx = torch.randperm(rows, device="cuda", generator=r.g)[:batch].to(torch.int32).contiguous()
        return dict(kind=kind, model=model, X=X, T=T.contiguous(), idx=idx, weights=surrogate.target_weights())
    nx, nk, ny = case["nx"], case["nk"], case["ny"]
    r = _Draws(seed)
    if kind == "prologue":
        f = _column_fields(case, seed)
        # cloud water everywhere that it is cloudy, humidity near saturation there
        f = {k: f[k] for k in ("qv3d", "qc3d", "qi3d", "qs3d", "t3d", "p3d")}
        return dict(kind=kind, ctx=ctx, fields=f, xlat=r.uniform(-90.0, 90.0, nx, ny),
                    xlong=r.uniform(-180.0, 180.0, nx, ny))
    halo = case["halo"]
    mx, my = nx + 2 * halo, ny + 2 * halo
    bounds = dict(ids=1, ide=nx + 1, jds=1, jde=ny + 1, kds=1, kde=nk + 1, ims=1 - halo, ime=nx + halo, jms=1 - halo,
                  jme=ny + halo, kms=1, kme=nk + 1, its=1, ite=nx, jts=1, jte=ny, kts=1, kte=nk)
    return dict(kind=kind, bounds=bounds, flags=dict(specified=halo > 0),
                lw=r.normal(2.0e-5, mx, nk + 1, my), sw=r.normal(2.0e-5, mx, nk + 1, my),
                c1=r.uniform(0.0, 1.0, nk + 1), c2=r.uniform(0.0, 5000.0, nk + 1),
                mut=r.uniform(5.0e4, 9.0e4, mx, my), t=r.normal(1.0, mx, nk + 1, my))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind in ("step", "lw", "sw"):
        from wrf_jax_b200 import rrtmg
        out = ()
        if kind != "sw":
            out += (rrtmg.rrtmg_lwrad_wrf_columns(**state["lw"], context=state["ctx"]),)
        if kind != "lw":
            out += (rrtmg.rrtmg_swrad_wrf_columns(**state["sw"], context=state["ctx"]),)
        return out
    if kind == "infer":
        from wrf_jax_b200 import surrogate
        r = surrogate.infer(state["model"], state["st"], state["d"], fallback=state["fallback"])
        return dict(rthratenlw=r.rthratenlw, rthratensw=r.rthratensw, glw=r.glw, lwupb=r.lwupb, swdnb=r.swdnb,
                    swupb=r.swupb, flags=r.flags, n_fallback=r.n_fallback)
    if kind == "train":
        m = state["model"]
        m.train_step(state["X"], state["T"], state["idx"], state["weights"], lr=1.0e-4)
        return dict(w=m.w, b=m.b, mw=m.mw, mb=m.mb, vw=m.vw, vb=m.vb)
    if kind == "prologue":
        from wrf_jax_b200 import prologue
        f = state["fields"]
        r = prologue.radiation_prologue(qv=f["qv3d"], qc=f["qc3d"], qi=f["qi3d"], qs=f["qs3d"], t3d=f["t3d"],
                                        p3d=f["p3d"], xlat=state["xlat"], xlong=state["xlong"], case_dir=False,
                                        context=state["ctx"], **_CALENDAR)
        return dict(cldfra3d=r.cldfra3d, o33d=r.o33d, coszr=r.coszr, condensate=r.condensate_present)
    from wrf_jax_b200 import tendency
    return tendency.radiation_tendency(state["lw"], state["sw"], state["c1"], state["c2"], state["mut"], state["t"],
                                       state["flags"], **state["bounds"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("step", "lw", "sw"):
        ncol, nk = case["nx"] * case["ny"], case["nk"]
        layers = nk + int(case["p_top"] * 0.01 / 4.0 + 0.5)
        radii = 4 if case["radii"] else 0  # three radii and snow
        # LW: 10 profiles, 2 level fields, 4 surface fields in; 2 profiles and 17 2-D fields out.  SW likewise.
        lw_bytes = 4.0 * ncol * ((9 + radii) * nk + 2 * (nk + 1) + 4 + 2 * nk + 15)
        sw_bytes = 4.0 * ncol * ((9 + radii) * nk + 2 * (nk + 1) + 5 + 2 * nk + 21)
        # binary32 operations counted on the C restatement: 12.9e3 per LW layer, 35.6e3 per SW layer of a day column
        lw_flops, sw_flops = 12.9e3 * layers * ncol, 35.6e3 * (nk + 1) * ncol * (1.0 - case["night"])
        return dict(bytes=(kind != "sw") * lw_bytes + (kind != "lw") * sw_bytes,
                    flops=(kind != "sw") * lw_flops + (kind != "lw") * sw_flops)
    if kind == "infer":
        ncol = case["nx"] * case["ny"]
        return dict(bytes=ncol * 4.0 * (9 * 50 + 51 + 4 + 2 * 50 + 4 + 1) + 1.6e6,
                    flops=2.0 * ncol * (454 * 512 + 2 * 512 * 512 + 512 * 106))
    if kind == "train":
        params = 454 * 512 + 2 * 512 * 512 + 512 * 106
        return dict(bytes=case["batch"] * (2.0 * 454 + 4.0 * 106) + params * 24.0, flops=6.0 * params * case["batch"])
    n = float(case["nx"]) * case["nk"] * case["ny"]
    if kind == "prologue":
        return dict(bytes=32.0 * n + 12.0 * case["nx"] * case["ny"], flops=40.0 * n)
    return dict(bytes=20.0 * n, flops=6.0 * n)


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _exact_network(state):
    """The network's outputs from device fields, the BF16 weights and the FP32 normalization, in 64 bits."""
    d, m, nk = state["d"], state["model"], 50
    nx, ny = d["tsk"].shape
    dt = torch.float64
    n = m.norm
    mean, rstd = n.in_mean[:454].to(dt), n.in_rstd[:454].to(dt)
    rows = {k: torch.empty(nx, nk if k.startswith("rth") else 1, ny, device="cuda", dtype=dt)
            for k in ("rthratenlw", "rthratensw", "glw", "lwupb", "swdnb", "swupb")}
    for i in range(nx):
        col = lambda k: d[k][i].to(dt)  # noqa: E731  (levels, ny)
        p8w = col("p8w")
        x = torch.cat([col("t3d"), torch.log(col("p3d")), col("qv3d"), col("qc3d"), col("qi3d"), col("qs3d"),
                       col("cldfra3d"), col("o33d"), p8w[:-1] - p8w[1:],
                       torch.stack([col("tsk"), col("albedo"), col("coszr"), col("emiss")])]).t()
        h = torch.zeros(ny, 512, device="cuda", dtype=dt)
        h[:, :454] = (x - mean) * rstd
        for layer in range(4):
            h = h @ m.wb[layer].to(dt).t() + m.b[layer].to(dt)
            if layer < 3:
                h = torch.nn.functional.gelu(h, approximate="tanh")
        y = (h * n.out_std.to(dt) + n.out_mean.to(dt)).t()
        day = (d["coszr"][i] > 0.0).to(dt)
        pi = col("pi3d")
        rows["rthratenlw"][i] = y[:nk] / (86400.0 * pi)
        rows["rthratensw"][i] = y[nk:2 * nk] * day / (86400.0 * pi)
        rows["glw"][i, 0], rows["lwupb"][i, 0] = y[2 * nk], y[2 * nk + 1]
        rows["swdnb"][i, 0], rows["swupb"][i, 0] = y[2 * nk + 2] * day, y[2 * nk + 3] * day
    out = {k: v if k.startswith("rth") else v[:, 0] for k, v in rows.items()}
    return dict(out, flags=None, n_fallback=None)


def _exact_train(state):
    m, dt = state["model"], torch.float64
    idx = state["idx"].long()
    X, T, wt = state["X"][idx].to(dt), state["T"][idx].to(dt), state["weights"].to(dt)
    w = [q.to(dt).requires_grad_() for q in m.wb]
    b = [q.to(dt).requires_grad_() for q in m.b]
    h = X
    for layer in range(4):
        h = h @ w[layer].t() + b[layer]
        if layer < 3:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    (wt * (h - T) ** 2).sum().div(X.shape[0] * 106).backward()
    step = m.step + 1
    bc1, bc2 = 1.0 - 0.9 ** step, 1.0 - 0.999 ** step
    out = dict(w=[], b=[], mw=[], mb=[], vw=[], vb=[])
    for name, master, grads, ms, vs in (("w", m.w, w, m.mw, m.vw), ("b", m.b, b, m.mb, m.vb)):
        for p, g, m1, v1 in zip(master, grads, ms, vs):
            m2 = 0.9 * m1.to(dt) + 0.1 * g.grad
            v2 = 0.999 * v1.to(dt) + 0.001 * g.grad ** 2
            out["m" + name].append(m2)
            out["v" + name].append(v2)
            out[name].append(p.to(dt) - 1.0e-4 * (m2 / bc1) / (torch.sqrt(v2 / bc2) + 1.0e-8))
    return out


def _exact_prologue(state):
    dt = torch.float64
    f = {k: v.to(dt) for k, v in state["fields"].items()}
    t, p, qv = f["t3d"], f["p3d"], f["qv3d"]
    qcld = f["qi3d"] + f["qc3d"] + f["qs3d"]
    esw = 610.78 * torch.exp(17.2693882 * (t - 273.15) / (t - 35.86))
    esi = 610.78 * torch.exp(21.8745584 * (t - 273.15) / (t - 7.66))
    ep_2 = 287.0 / 461.6
    qvsw = torch.where(p - esw > 1.0, ep_2 * esw / (p - esw), torch.zeros_like(p))
    qvsi = torch.where(p - esi > 1.0, ep_2 * esi / (p - esi), torch.zeros_like(p))
    w = (f["qi3d"] + f["qs3d"]) / qcld.clamp(min=1.0e-300)
    qvs = (1.0 - w) * qvsw + w * qvsi
    del esw, esi, qvsw, qvsi, w
    rhum = qv / qvs
    arg = (-100.0 * qcld / (qvs - qv).clamp(min=1.0e-10) ** 0.49).clamp(min=-6.9)
    frac = rhum.clamp(min=1.0e-10) ** 0.25 * (1.0 - torch.exp(arg))
    frac = torch.where(frac < 0.01, torch.zeros_like(frac), frac)
    frac = torch.where(rhum >= 1.0, torch.ones_like(frac), frac)
    cld = torch.where((t > 100.0) & (p > 100.0) & (qcld >= 1.0e-12), frac, torch.zeros_like(frac))
    del frac, rhum, arg, qvs, qcld
    # cos zenith at the middle of the radiation interval
    julian, rad = _CALENDAR["julian"], math.pi / 180.0
    sxlong = 360.0 / 365.0 * (julian - 80.0) * rad
    declin = math.asin(math.sin(23.5 * rad) * math.sin(sxlong))
    da = 2.0 * math.pi * (julian - 1.0) / 365.0
    eot = 229.18 * (0.000075 + 0.001868 * math.cos(da) - 0.032077 * math.sin(da) - 0.014615 * math.cos(2 * da)
                    - 0.04089 * math.sin(2 * da))
    tloc = _CALENDAR["gmt"] + (math.fmod(_CALENDAR["xtime"] + 0.5 * _CALENDAR["radt"], 1440.0) + eot) / 60.0
    lat, lon = state["xlat"].to(dt), state["xlong"].to(dt)
    hour = 15.0 * (tloc + lon / 15.0 - 12.0) * rad
    cz = math.sin(declin) * torch.sin(lat * rad) + math.cos(declin) * torch.cos(lat * rad) * torch.cos(hour)
    # ozone: months (mid June 166, mid July 197), then latitude, then pressure
    plev, lats, oz = (torch.from_numpy(np.asarray(a)).to("cuda", dt) for a in _KEPT["ozone"])
    day = julian + 1.0
    table = (oz[5] * (197.0 - day) + oz[6] * (day - 166.0)) / 31.0
    li = (torch.searchsorted(lats, lat.contiguous()) - 1).clamp(0, len(lats) - 2)
    share = (lat - lats[li]) / (lats[li + 1] - lats[li])
    out = torch.empty_like(p)
    for k in range(p.shape[1]):
        pk = p[:, k].contiguous()
        kk = (torch.searchsorted(plev, pk) - 1).clamp(0, len(plev) - 2)
        at = lambda j: table[li, j] + share * (table[li + 1, j] - table[li, j])  # noqa: E731
        v = (at(kk) * (plev[kk + 1] - pk) + at(kk + 1) * (pk - plev[kk])) / (plev[kk + 1] - plev[kk])
        last = torch.full_like(kk, len(plev) - 1)
        v = torch.where(pk < plev[0], at(torch.zeros_like(kk)) * pk / plev[0], v)
        out[:, k] = torch.where(pk > plev[-1], at(last), v)
    return dict(cldfra3d=cld, o33d=out, coszr=cz.clamp(-1.0, 1.0), condensate=None)


def _exact_tendency(state):
    dt, b = torch.float64, state["bounds"]
    lw, sw, t = (state[k].to(dt) for k in ("lw", "sw", "t"))
    mass = state["c1"].to(dt).view(1, -1, 1) * state["mut"].to(dt).unsqueeze(1) + state["c2"].to(dt).view(1, -1, 1)
    heat = lw + sw
    i0, j0 = b["its"] - b["ims"], b["jts"] - b["jms"]
    i1, j1, k1 = b["ite"] - b["ims"] + 1, b["jte"] - b["jms"] + 1, b["kte"] - b["kms"] + 1
    heat[i0:i1, :k1, j0:j1] *= mass[i0:i1, :k1, j0:j1]
    edge = 1 if state["flags"]["specified"] else 0
    t = t.clone()
    t[i0 + edge:i1 - edge, :k1, j0 + edge:j1 - edge] += heat[i0 + edge:i1 - edge, :k1, j0 + edge:j1 - edge]
    return heat, t


def exact(case, seed):
    """Results in 64 bits.  The radiation calls have none here: a second restatement of RRTMG would be the size of
    the framework's own (they are held to the start's outputs), and the fallback's columns are such calls."""
    kind = case["kind"]
    if kind in ("step", "lw", "sw") or (kind == "infer" and case["fallback"]):
        return None
    state = prepare(case, seed)
    return dict(infer=_exact_network, train=_exact_train, prologue=_exact_prologue, tendency=_exact_tendency)[kind](state)
