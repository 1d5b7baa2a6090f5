"""The squared shear frequency formed face by face along marching warps, against
plain torch in 64 bits: one row, rows that end a warp's march, rows and columns
one past it, masked columns untouched."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 2), (31, 8, 3), (32, 9, 2), (63, 33, 4), (390, 70, 40)])
def test_shear_frequency(nx, ny, nz, dtype):
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(nx + ny)
    h, NX, NY = 2, nx + 4, ny + 4
    t = getattr(torch, dtype)
    up = lambda a, d: torch.from_numpy(a).to("cuda", d)  # noqa: E731
    hu, hv = (up(rng.uniform(0.5, 2.0, (nz, NY, NX)), torch.float64) for _ in range(2))
    u, v = (up(rng.uniform(-1, 1, (nz, NY, NX)), t) for _ in range(2))
    mask = up((rng.uniform(size=(NY, NX)) > 0.2).astype(np.int32), torch.int32)
    SS = torch.full((nz + 1, NY, NX), -7.0, dtype=t, device="cuda")
    _lib.call("getm_shear_frequency" + ("_f32" if dtype == "float32" else ""), NX, NY, nz, h + 1, h + nx, h + 1, h + ny,
              mask.data_ptr(), hu.data_ptr(), hv.data_ptr(), u.data_ptr(), v.data_ptr(), SS.data_ptr(), _s())
    t1 = ((u[1:].double() - u[:-1].double()) / (0.5 * (hu[1:] + hu[:-1]))) ** 2
    t3 = ((v[1:].double() - v[:-1].double()) / (0.5 * (hv[1:] + hv[:-1]))) ** 2
    want = 0.5 * (t1[:, h:h + ny, h:h + nx] + t1[:, h:h + ny, h - 1:h + nx - 1] + t3[:, h:h + ny, h:h + nx]
                  + t3[:, h - 1:h + ny - 1, h:h + nx])
    wet = mask[h:h + ny, h:h + nx] > 0
    got = SS[1:nz, h:h + ny, h:h + nx].double()
    # per term a difference, a sum, a quotient and a square: twice some four
    # roundings (float thicknesses truncated to 2^-23), then three sums
    eps = 2.0 ** -53 if dtype == "float64" else 2.0 ** -22
    assert bool(((got - want).abs() <= 16 * eps * want + 8 * eps * (t1.max() + t3.max()) ** 0.5 * want ** 0.5)[:, wet].all())
    SS[1:nz, h:h + ny, h:h + nx][:, wet] = -7.0
    assert bool((SS == -7.0).all())
