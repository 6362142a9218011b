"""Radiation tendency chain (LW + SW heating, mass coupling, accumulation into
the potential-temperature tendency): the oracle against the reference's golden
fixtures on the CPU, and the fused CUDA kernel bit for bit on the GPU."""

from __future__ import annotations

import ctypes
import sys

import numpy as np
import pytest

from conftest import GOLDEN, REPO


@pytest.fixture(scope="module")
def gold():
    with np.load(GOLDEN / "tendency_golden.npz") as d:
        data = {k: d[k] for k in d.files}
    cases = {}
    for key, v in data.items():
        name, field = key.split("/")
        cases.setdefault(name, {})[field] = v
    return cases


@pytest.fixture(scope="module")
def to():
    sys.path.insert(0, str(REPO / "oracle"))
    import tendency_oracle
    return tendency_oracle


def _bounds(c, to):
    bv = c["bounds"]
    b = dict(zip(to.BOUND_NAMES, map(int, bv[:18])))
    b.update(specified=bool(bv[18]), nested=bool(bv[19]), periodic_x=bool(bv[20]))
    return b


def test_oracle_matches_reference_golden(gold, to):
    for name, c in gold.items():
        r, t = to.radiation_tendency(c["lw"], c["sw"], c["c1"], c["c2"], c["mut"], c["rt_tendf"], _bounds(c, to))
        assert np.array_equal(r.view(np.uint32), c["rthraten"].view(np.uint32)), name
        assert np.array_equal(t.view(np.uint32), c["rt_tendf_out"].view(np.uint32)), name


def test_golden_cases_cover_the_regions(gold):
    # coupling and accumulation regions differ (boundary rows) and both leave
    # part of the memory array untouched
    for name, c in gold.items():
        coupled = c["rthraten"] != (c["lw"] + c["sw"])
        added = c["rt_tendf_out"] != c["rt_tendf"]
        assert coupled.any() and added.any() and not added.all(), name
    assert any((c["rthraten"] != c["lw"] + c["sw"]).sum() > (c["rt_tendf_out"] != c["rt_tendf"]).sum()
               for c in gold.values())


def test_c_abi_rejects_bad_arguments_without_gpu(pkg):
    from wrf_jax_b200 import _capi
    lib = _capi.load()
    tb = _capi.TendencyBounds(ids=1, ide=5, jds=1, jde=5, kds=1, kde=5, ims=3, ime=1, jms=1, jme=5, kms=1, kme=5,
                              its=1, ite=5, jts=1, jte=5, kts=1, kte=5)
    p = ctypes.c_void_p(16)
    # ime < ims, missing outputs, coupling without its arrays: rejected before any CUDA call
    assert lib.rrtmg_radiation_tendency(ctypes.byref(tb), p, p, p, p, p, 1, p, p, None) == 1
    tb.ime = 5
    assert lib.rrtmg_radiation_tendency(ctypes.byref(tb), p, p, p, p, p, 1, None, None, None) == 1
    assert lib.rrtmg_radiation_tendency(ctypes.byref(tb), p, p, None, p, p, 1, p, p, None) == 1
    assert lib.rrtmg_phy_ra_ten(ctypes.byref(tb), None, p, None) == 1


@pytest.mark.gpu
def test_gpu_matches_reference_golden(pkg, gold, to):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wrf_jax_b200 import tendency
    for name, c in gold.items():
        b = _bounds(c, to)
        flags = {k: b.pop(k) for k in ("specified", "nested", "periodic_x")}
        r, t = tendency.radiation_tendency(c["lw"], c["sw"], c["c1"], c["c2"], c["mut"], c["rt_tendf"], flags, **b)
        np.testing.assert_array_equal(r.view(np.uint32), c["rthraten"].view(np.uint32), err_msg=name)
        np.testing.assert_array_equal(t.view(np.uint32), c["rt_tendf_out"].view(np.uint32), err_msg=name)
        t2 = tendency.phy_ra_ten(flags, c["rt_tendf"], c["rthraten"], **b)
        np.testing.assert_array_equal(t2.view(np.uint32), c["rt_tendf_out"].view(np.uint32), err_msg=name)


@pytest.mark.gpu
@pytest.mark.parametrize("jme", [1205, 1207])  # 1,210 (scalar path) and 1,212 (four per thread) south-north
def test_gpu_matches_oracle_large(pkg, to, jme):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wrf_jax_b200 import tendency
    rng = np.random.default_rng(3)
    b = dict(ids=1, ide=301, jds=1, jde=1201, kds=1, kde=51, ims=-4, ime=305, jms=-4, jme=jme, kms=1, kme=51,
             its=1, ite=300, jts=1, jte=1200, kts=1, kte=50)
    shape = (b["ime"] - b["ims"] + 1, b["kme"] - b["kms"] + 1, b["jme"] - b["jms"] + 1)
    lw = rng.normal(-2e-5, 1e-5, shape).astype(np.float32)
    sw = rng.normal(1e-5, 1e-5, shape).astype(np.float32)
    c1 = rng.uniform(0, 1, shape[1]).astype(np.float32)
    c2 = rng.uniform(0, 5000, shape[1]).astype(np.float32)
    mut = rng.uniform(5e4, 9.5e4, (shape[0], shape[2])).astype(np.float32)
    t0 = rng.normal(0, 3, shape).astype(np.float32)
    for flags in (dict(specified=True, nested=False, periodic_x=False),
                  dict(specified=False, nested=False, periodic_x=True)):
        want_r, want_t = to.radiation_tendency(lw, sw, c1, c2, mut, t0, {**b, **flags})
        r, t = tendency.radiation_tendency(lw, sw, c1, c2, mut, t0, flags, **b)
        assert np.array_equal(r.view(np.uint32), want_r.view(np.uint32))
        assert np.array_equal(t.view(np.uint32), want_t.view(np.uint32))


# rows of a multiple of four elements, other rows, and arrays that are not 16-byte aligned
@pytest.mark.gpu
@pytest.mark.parametrize("south_north,offset", [(1000, 0), (1001, 0), (1000, 1)])
def test_gpu_in_place_tiles_on_two_streams(pkg, south_north, offset):
    """Two tiles of one array updated in place at the same time, on two streams:
    neither call writes outside its own tile, so no update of either is lost.
    Every pass adds 1 (small whole numbers, exact)."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wrf_jax_b200 import _capi, tendency
    lib = _capi.load()
    nx, nk, ny = 64, 21, south_north
    n, passes = nx * nk * ny, 200
    flat = torch.zeros(n + 4, device="cuda")
    t = flat[offset:offset + n]
    one = torch.ones(n + 4, device="cuda")[offset:offset + n]
    assert t.data_ptr() % 16 == 4 * offset
    dims = dict(ids=1, ide=nx + 1, jds=1, jde=ny + 1, kds=1, kde=nk, ims=1, ime=nx, jms=1, jme=ny, kms=1, kme=nk,
                kts=1, kte=nk - 1)
    # rows shared by both tiles, split where no 16-byte boundary lies; the second tile leaves out the last rows
    tiles = [dict(its=1, ite=nx, jts=3, jte=498), dict(its=2, ite=nx - 3, jts=499, jte=ny - 2)]
    streams = [torch.cuda.Stream() for _ in tiles]
    torch.cuda.synchronize()
    for _ in range(passes):
        for b, s in zip(tiles, streams):
            tb = tendency.bounds({}, **dims, **b)
            assert lib.rrtmg_phy_ra_ten(ctypes.byref(tb), t.data_ptr(), one.data_ptr(),
                                        ctypes.c_void_p(s.cuda_stream)) == 0
    torch.cuda.synchronize()
    want = torch.zeros(nx, nk, ny)
    for b in tiles:
        want[b["its"] - 1:b["ite"], :nk - 1, b["jts"] - 1:b["jte"]] += passes
    assert torch.equal(t.cpu().view(nx, nk, ny), want)
    assert not flat[:offset].any() and not flat[offset + n:].any()


@pytest.mark.gpu
def test_gpu_result_stays_tied_to_a_tracked_input(pkg):
    """rt_tendf with a gradient: the updated tendency is rt_tendf plus the heating,
    with the gradient of a copy, and rt_tendf itself is left as it was."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from wrf_jax_b200 import tendency
    b = dict(ids=1, ide=7, jds=1, jde=6, kds=1, kde=4, ims=1, ime=6, jms=1, jme=5, kms=1, kme=4, its=1, ite=6, jts=1,
             jte=5, kts=1, kte=3)
    lw, sw, t0 = (torch.randn(6, 4, 5, device="cuda") for _ in range(3))
    c1, c2, mut = torch.rand(4, device="cuda"), torch.rand(4, device="cuda"), torch.rand(6, 5, device="cuda")
    r, plain = tendency.radiation_tendency(lw, sw, c1, c2, mut, t0, {}, **b)
    tracked = t0.clone().requires_grad_()
    _, t = tendency.radiation_tendency(lw, sw, c1, c2, mut, tracked, {}, **b)
    assert torch.equal(t, plain) and torch.equal(tracked, t0)
    t.sum().backward()
    assert torch.equal(tracked.grad, torch.ones_like(t0))
