"""The forms that the kernels take by size against each other and the oracles.

Radiation: a domain below the small-chunk limits, and the same columns repeated
until the domain is above them.  A column's result does not depend on its
neighbours, so every copy must have the bits of the small call; the general
form is what the parity tests hold against the oracle.  The tables are the
package's, or generated ones where no blob is built (the equality holds for
any).  The other paths compare with the oracles, with tolerances stated there.
"""

from __future__ import annotations

import importlib.util
import sys

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda(pkg):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.fixture(scope="module")
def ctx(torch_cuda):
    from wrf_jax_b200 import rrtmg, tables
    blob = tables.DEFAULT_BLOB
    if not blob.exists():
        spec = importlib.util.spec_from_file_location("perf_cases", REPO / "perf" / "cases.py")
        cases = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(cases)
        blob = cases.stand_in_blob()
    c = rrtmg.RrtmgContext(blob)
    yield c
    c.close()


def _repeat(kwargs, nx, times):
    return {k: np.concatenate([v] * times, axis=0) if isinstance(v, np.ndarray) and v.ndim >= 2 and v.shape[0] == nx
            else v for k, v in kwargs.items()}


def _assert_copies(small, big, nx, times, tag):
    for name, want in small._asdict().items():
        if want is None:
            continue
        got = np.asarray(getattr(big, name))
        want = np.asarray(want)
        for t in (0, times // 2, times - 1):
            part = got[t * nx:(t + 1) * nx]
            same = (part.view(np.uint32) == want.view(np.uint32)) | (np.isnan(part) & np.isnan(want))
            assert same.all(), f"{tag} {name}: copy {t}, {int((~same).sum())} of {same.size} differ"


# kSwSmallColumns = 320 day columns, kLwSmallColumns = 384 columns, kSmallColumns = 2,048 columns
@pytest.mark.parametrize("nx,ny,nk,more", [
    (1, 1, 17, {}),
    (3, 5, 44, dict(night_fraction=1.0)),
    (7, 9, 57, dict(p_top=2000.0, has_req=True, fractional_clouds=True)),
    (1, 319, 50, dict(night_fraction=0.0)),
    (1, 320, 50, dict(night_fraction=0.0, cloud_p=0.9)),
    (1, 321, 50, dict(night_fraction=0.0)),
    (1, 383, 31, dict(cloud_p=0.0)),
    (1, 384, 60, dict(p_top=1000.0)),
    (1, 385, 60, dict(p_top=1000.0, fractional_clouds=True)),
    (23, 89, 30, dict(night_fraction=0.9)),   # 2,047 columns, some 200 of them by day
    (32, 64, 30, dict(night_fraction=0.9)),   # 2,048
])
@pytest.mark.parametrize("options", [{}, dict(icloud=0), dict(fp64_steps=True)], ids=["plain", "clear", "fp64"])
def test_small_domains_equal_large_ones(ctx, nx, ny, nk, more, options):
    from wrf_jax_b200 import rrtmg, synthetic
    st = synthetic.make_columns(nx, ny, nk, seed=nx * 1000 + ny, **more)
    times = -(-2049 // (nx * ny))
    for call, kw in ((rrtmg.rrtmg_lwrad_wrf_columns, st.lw_kwargs()), (rrtmg.rrtmg_swrad_wrf_columns, st.sw_kwargs())):
        small = call(**{**kw, **options}, context=ctx)
        big = call(**{**_repeat(kw, nx, times), **options}, context=ctx)
        _assert_copies(small, big, nx, times, call.__name__)


def test_a_larger_domains_workspace_serves_a_smaller_one(ctx):
    """The workspace sizes do not fall as the domain grows, the end of the
    small-chunk forms (2,048 columns) included."""
    import ctypes
    from wrf_jax_b200 import rrtmg
    gases = dict(co2vmr=4.0e-4, n2ovmr=3.0e-7, ch4vmr=1.7e-6, yr=2024)
    for name, config in (("lw", lambda n: rrtmg.lw_config(1, n, 50, p_top=5000.0, **gases)),
                         ("sw", lambda n: rrtmg.sw_config(1, n, 50, solcon=1370.0, **gases))):
        query = getattr(ctx.lib, f"rrtmg_{name}_workspace_bytes")
        query.restype = ctypes.c_size_t
        sizes = [query(ctx.handle, ctypes.byref(config(n)))
                 for n in (1, 320, 384, 385, 2047, 2048, 2049, 2500, 3100, 5000, 16384, 16385, 32769, 100000)]
        assert sizes[0] > 0 and sizes == sorted(sizes), (name, sizes)


# kMaxBuf = 40 layers above the model top; a warp takes 30 of them (and two values of the top) at once
@pytest.mark.parametrize("p_top", [500.0, 11600.0, 12000.0, 12400.0, 15900.0])
def test_column_setup_by_warp_equals_by_thread(ctx, torch_cuda, p_top):
    """rrtmg_lwrad sets a column up with a warp, rrtmg_lwrad_static_scratch with a thread: the same bits."""
    from test_zz_no_alloc import _assert_same, _device_call
    from wrf_jax_b200 import _capi, synthetic
    st = synthetic.make_columns(5, 9, 20, seed=int(p_top), p_top=p_top)
    env = (ctx, _capi, torch_cuda)
    _assert_same(_device_call(env, st, "rrtmg_lwrad"), _device_call(env, st, "rrtmg_lwrad_static_scratch"), str(p_top))


@pytest.mark.parametrize("levsiz,latsiz", [(59, 64), (2, 2), (96, 65), (97, 65), (120, 90)])
def test_ozone_table_forms(ctx, torch_cuda, levsiz, latsiz):
    """The slopes formed once per block (up to 96 KB of rows: 96 x 64 levels and
    latitude gaps) and formed per column, with latitudes on, between and beyond
    the table's and pressures beyond its ends: the oracle's bits."""
    sys.path.insert(0, str(REPO / "oracle"))
    import prologue_oracle as po
    from wrf_jax_b200 import prologue
    rng = np.random.default_rng(levsiz)
    plev = np.sort(rng.uniform(30.0, 1.0e5, levsiz)).astype(np.float32)
    lat = np.linspace(-87.0, 88.0, latsiz).astype(np.float32)
    oz = rng.uniform(0.0, 1.0e-5, (12, latsiz, levsiz)).astype(np.float32)
    nx, nk, ny = 13, 9, 77
    xlat = rng.uniform(-90.0, 90.0, (nx, ny)).astype(np.float32)
    xlat[0, :2] = lat[0], lat[-1]
    p = np.sort(rng.uniform(10.0, 1.05e5, (nx, nk, ny)), axis=1)[:, ::-1].astype(np.float32)
    prologue.set_ozone_climatology(plev, lat, oz, context=ctx, key="table forms")
    got = prologue.cam_o3rad(xlat, np.ascontiguousarray(p), julian=170.0, case_dir=False, context=ctx)
    want = po.cam_o3rad(xlat, np.ascontiguousarray(p), julian=170.0, plev=plev, lat_oz=lat, ozone=oz)
    np.testing.assert_array_equal(np.asarray(got).view(np.uint32), np.asarray(want, np.float32).view(np.uint32))


@pytest.mark.parametrize("south_north,offset", [(4, 0), (5, 0), (6, 0), (7, 0), (9, 1), (33, 3), (258, 2), (1, 0)])
@pytest.mark.parametrize("couple", [True, False])
def test_tendency_ragged_rows(torch_cuda, south_north, offset, couple):
    """Rows of any length and arrays at any 4-byte offset, in place and into
    another array: the oracle's bits."""
    import ctypes
    torch = torch_cuda
    sys.path.insert(0, str(REPO / "oracle"))
    import tendency_oracle as to
    from wrf_jax_b200 import _capi, tendency
    rng = np.random.default_rng(south_north)
    nx, nk = 11, 5
    b = dict(ids=1, ide=nx - 2, jds=1, jde=south_north, kds=1, kde=nk, ims=0, ime=nx - 1, jms=1, jme=south_north, kms=1,
             kme=nk, its=1, ite=nx - 3, jts=1, jte=max(1, south_north - 1), kts=1, kte=nk - 1)
    shape = (nx, nk, south_north)
    lw, sw, t0 = (rng.normal(0.0, 1.0, shape).astype(np.float32) for _ in range(3))
    c1, c2 = rng.uniform(0, 1, nk).astype(np.float32), rng.uniform(0, 5000, nk).astype(np.float32)
    mut = rng.uniform(5e4, 9.5e4, (nx, south_north)).astype(np.float32)
    flags = dict(specified=False, nested=False, periodic_x=True)
    if couple:
        want_r, want_t = to.radiation_tendency(lw, sw, c1, c2, mut, t0, {**b, **flags})
        r, t = tendency.radiation_tendency(lw, sw, c1, c2, mut, t0, flags, **b)
        assert np.array_equal(r.view(np.uint32), want_r.view(np.uint32))
        assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))
    tb = tendency.bounds(flags, **b)

    def put(a):
        flat = torch.empty(a.size + 4, device="cuda")
        flat[offset:offset + a.size] = torch.from_numpy(a.ravel()).cuda()
        return flat, flat[offset:offset + a.size]
    keep = [put(a) for a in (lw, sw, c1, c2, mut, t0, np.zeros(shape, np.float32), np.full(shape, np.nan, np.float32))]
    d = [v.data_ptr() for _, v in keep]
    lib, s = _capi.load(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.rrtmg_radiation_tendency_into(ctypes.byref(tb), *d[:5], int(couple), d[6], d[5], d[7], s) == 0
    into_r, into_t = keep[6][1].clone(), keep[7][1].clone()
    assert lib.rrtmg_radiation_tendency(ctypes.byref(tb), *d[:5], int(couple), d[6], d[5], s) == 0
    assert torch.equal(into_r.view(torch.int32), keep[6][1].view(torch.int32))
    assert torch.equal(into_t.view(torch.int32), keep[5][1].view(torch.int32))
    if couple:
        assert np.array_equal(into_t.cpu().numpy().view(np.uint32), want_t.ravel().view(np.uint32))


# 2,304 columns are 72 tiles of 128 x 128 per layer (64-wide ones are taken up to 74), 2,432 are 76
@pytest.mark.parametrize("batch", [128, 384, 2304, 2432, 3712])
def test_training_step_batches(torch_cuda, batch):
    """Gradients against the CPU oracle with rows drawn in any order; tolerance
    as in test_surrogate_training: 2e-2 of each gradient's norm, for BF16
    activations that may round one unit apart."""
    torch = torch_cuda
    sys.path.insert(0, str(REPO / "oracle"))
    import surrogate_oracle as so
    from wrf_jax_b200 import surrogate as S
    model = S.SurrogateModel(seed=5)
    g = torch.Generator(device="cuda").manual_seed(batch)
    rows = batch + 37
    X = torch.randn(rows, S.K_IN, device="cuda", generator=g).bfloat16()
    X[:, S.N_FEATURES:] = 0
    Tn = torch.randn(rows, S.N_OUT, device="cuda", generator=g)
    idx = torch.randperm(rows, device="cuda", generator=g)[:batch].to(torch.int32)
    w = S.target_weights()
    wb, bs = [x.float().cpu().numpy() for x in model.wb], [x.cpu().numpy() for x in model.b]
    model.train_step(X, Tn, idx, w, lr=0.0)
    torch.cuda.synchronize()
    assert S.gemm_error() == 0
    at = idx.long()
    _, gw, gb = so.forward_backward(X[at].float().cpu().numpy(), Tn[at].cpu().numpy(), wb, bs, w.cpu().numpy(),
                                    1.0 / (batch * S.N_TARGETS))
    for layer in range(4):
        for got, want in ((model._buf["gw"][layer], gw[layer]), (model._buf["gb"][layer], gb[layer])):
            err = np.linalg.norm(got.cpu().numpy() - want) / max(np.linalg.norm(want), 1e-30)
            assert err < 2e-2, (layer, err)
    # the next step's weights: the master copies rounded, and their transposes
    for master, rounded, transposed in zip(model.w, model.wb, model.wbt):
        assert torch.equal(master.to(torch.bfloat16), rounded) and torch.equal(rounded.t(), transposed)


@pytest.mark.parametrize("batch", [1024, 6272, 16384])
def test_weight_gradients_of_large_batches(torch_cuda, batch):
    """The weight gradients against the same products in 64 bits.  A split of the
    batch sums at most 1,024 rows in the tensor cores, 64 instructions that may
    each lose a binary32 unit (2^-24) of the running sum, half of one on average:
    64 * 2^-25 = 1.9e-6 of the gradient's norm; 2e-6 with the splits' own sums."""
    torch = torch_cuda
    from wrf_jax_b200 import surrogate as S
    model = S.SurrogateModel(seed=6)
    g = torch.Generator(device="cuda").manual_seed(batch)
    X = torch.randn(batch, S.K_IN, device="cuda", generator=g).bfloat16()
    Tn = torch.randn(batch, S.N_OUT, device="cuda", generator=g)
    idx = torch.randperm(batch, device="cuda", generator=g).to(torch.int32)
    model.train_step(X, Tn, idx, S.target_weights(), lr=0.0)
    torch.cuda.synchronize()
    assert S.gemm_error() == 0
    b = model._buf
    for layer, (grad, inputs) in enumerate(zip([*b["dZt"], b["dYt"]], [b["Xbt"], *b["Ht"]])):
        want = grad.double() @ inputs.double().t()
        err = float((b["gw"][layer].double() - want).norm() / want.norm())
        assert err < 2e-6, (layer, err)


def test_training_step_with_weights_at_any_element(torch_cuda):
    """FP32 weights and moments that are views at odd elements of larger buffers:
    the same bits as with tensors of their own."""
    torch = torch_cuda
    from wrf_jax_b200 import surrogate as S
    g = torch.Generator(device="cuda").manual_seed(4)
    X = torch.randn(256, S.K_IN, device="cuda", generator=g).bfloat16()
    Tn = torch.randn(256, S.N_OUT, device="cuda", generator=g)
    idx = torch.arange(256, device="cuda", dtype=torch.int32)
    own, views = S.SurrogateModel(seed=9), S.SurrogateModel(seed=9)
    for name, shift in (("w", 1), ("mw", 2), ("vw", 3), ("b", 1), ("mb", 1), ("vb", 1)):
        tensors = getattr(views, name)
        for i, t in enumerate(tensors):
            tensors[i] = torch.cat([torch.zeros(shift, device="cuda"), t.flatten()])[shift:].view(t.shape)
            assert tensors[i].data_ptr() % 16
    for model in (own, views):
        model.train_step(X, Tn, idx, S.target_weights(), lr=1.0e-3, weight_decay=0.01)
    for name in ("w", "mw", "vw", "b", "mb", "vb", "wb", "wbt"):
        for a, b in zip(getattr(own, name), getattr(views, name)):
            assert torch.equal(a, b), name
