"""2D advection from the grid's column heights: the heights it starts from stay,
the split sequences end in the caller's arrays, and the tile heights of the y
pass give the same bits (a plane of many tiles against the same plane cut to
few columns)."""

import numpy as np
import pytest

from tests.test_gpu_operators import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [0, 1])
@pytest.mark.parametrize("split", [1, 2, 3])
@pytest.mark.parametrize("nx,ny", [(5, 3), (40, 30), (330, 400)])
def test_from_heights(nx, ny, split, mixed):
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _p, _s
    from getm_gb300.operators import Advection, AdvectionScheme, AdvectionSplit

    _, _, Td, rng = setup(seed=split, nx=nx, ny=ny, nz=1)
    up = lambda s: torch.from_numpy(rng.uniform(-s, s, (Td.ny_, Td.nx_))).cuda()  # noqa: E731
    u, v, f = up(0.4), up(0.4), 10.0 + up(5.0)
    adv = Advection(Td, AdvectionScheme.SUPERBEE, AdvectionSplit(split))
    D0 = Td.D.all_values.clone()
    a, Da = f.clone(), torch.full_like(f, 3.0)
    b, Db = f.clone(), D0.clone()
    tail = (_p(Td.ugrid.D), _p(Td.vgrid.D))
    head = (adv.p, Td.handle, Td.ugrid.handle, Td.vgrid.handle, 1, split, u.data_ptr(), v.data_ptr(), None, None, 20.0)
    _lib.call("getm_advection_2d_from", *head, _p(Td.D), Da.data_ptr(), *tail, a.data_ptr(), mixed, _s())
    _lib.call("getm_advection_2d_mixed" if mixed else "getm_advection_2d", *head, Db.data_ptr(), *tail, b.data_ptr(), _s())
    assert torch.equal(Td.D.all_values, D0)
    same = lambda x, y: bool(((x == y) | (x.isnan() & y.isnan())).all())  # noqa: E731
    assert same(a, b) and same(Da, Db)
    assert not torch.equal(a, f)


@pytest.mark.parametrize("nx,ny", [(33, 14), (64, 61), (97, 75)])
def test_tile_heights(nx, ny):
    """An FP64 batch of layers, whose many tiles are of 16 rows, and one layer
    of it alone, whose tiles are of 4."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300 import _lib
    from getm_gb300._pygetm import _p, _s

    nk = 152
    _, _, Td, rng = setup(seed=ny, nx=nx, ny=ny, nz=1)
    up = lambda lo, hi, k: torch.from_numpy(rng.uniform(lo, hi, (k, Td.ny_, Td.nx_))).cuda()  # noqa: E731
    v, h, hv, f = up(-0.4, 0.4, nk), up(1.0, 2.0, nk), up(1.0, 2.0, nk), up(0.0, 9.0, nk)
    outs = []
    from getm_gb300.operators import Advection, AdvectionScheme

    adv = Advection(Td, AdvectionScheme.MUSCL)
    for k0, n in ((0, nk), (7, 1)):
        hh, ff = h[k0:k0 + n].clone(), f[k0:k0 + n].clone()
        _lib.call("getm_advection_uv_calculate", 2, n, adv.p, Td.handle, Td.vgrid.handle, v[k0:k0 + n].data_ptr(), None,
                  20.0, hh.data_ptr(), hv[k0:k0 + n].data_ptr(), ff.data_ptr(), _s())
        outs.append((hh, ff))
    assert torch.equal(outs[0][0][7], outs[1][0][0]) and torch.equal(outs[0][1][7], outs[1][1][0])
