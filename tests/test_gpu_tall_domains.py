"""Domains of very many rows: the advection passes fold their rows into the grid's
65535 blocks."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _passes(nx, ny, nk, direction, form):
    """One pass over a tall domain and over its first 60 rows alone (what lies
    three rows from their end depends on nothing beyond)."""
    import ctypes

    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    cut, outs = 60, []
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda lo, hi, *k: lo + (hi - lo) * torch.rand((*k, ny, nx), dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    mask = torch.ones((ny, nx), dtype=torch.int32, device="cuda")
    metric = [r(0.5, 1.0) for _ in range(3)]
    u, h, hu, f = r(-0.1, 0.1, nk), r(1.0, 2.0, nk), r(1.0, 2.0, nk), r(5.0, 9.0, nk)
    if form != "fp64":
        u = u.float()
    for rows in (ny, cut):
        part = lambda a: a[..., :rows, :].contiguous()  # noqa: B023, E731
        m, d, inv, ia = part(mask), *[part(a) for a in metric]
        handles = []
        for _ in range(2):
            grid = ctypes.c_void_p()
            _lib.call("getm_create_grid", 1, nx - 4, 1, rows - 4, 1, nk, 2, 2, ctypes.byref(grid))
            for n, a in (("mask", m), ("dx", d), ("dy", d), ("idx", inv), ("idy", inv), ("iarea", ia)):
                _lib.call("getm_grid_set_array", grid, n.encode(), ctypes.c_void_p(a.data_ptr()))
            handles.append(grid)
        adv = ctypes.c_void_p()
        _lib.call("getm_advection_create", 5, handles[0], ctypes.byref(adv))
        uu, hh, hhu, ff = part(u), part(h), part(hu), part(f)
        ho, fo = torch.empty_like(hh), torch.empty_like(ff)
        _lib.call("getm_advection_uv_pass" + ("" if form == "fp64" else "_f64s"), direction, nk, adv, *handles, uu.data_ptr(), None,
                  0.3, hh.data_ptr(), ho.data_ptr(), hhu.data_ptr(), 1, _lib.ptr_array([ff.data_ptr()]),
                  _lib.ptr_array([fo.data_ptr()]), _s())
        torch.cuda.synchronize()
        outs.append((ho, fo))
        for n, hd in (("getm_advection_finalize", adv), *[("getm_grid_finalize", x) for x in handles]):
            _lib.call(n, hd)
    for a, b in zip(*outs):
        assert torch.equal(a[:, :cut - 5], b[:, :cut - 5])
    assert not torch.equal(outs[0][1][:, ny // 2:], f[:, ny // 2:])


@pytest.mark.parametrize("direction,nk,nx,ny", [(1, 2, 128, 140000), (2, 1, 8, 200000), (2, 2, 8, 200000)])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_rows(direction, nk, nx, ny, form):
    _passes(nx, ny, nk, direction, form)
