"""The squared shear frequency on narrow domains, whose rows share a warp, and
around land without thickness, against plain torch in 64 bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("nx,ny,nz", [(2, 9, 3), (3, 40, 2), (4, 700, 9), (7, 33, 2), (14, 17, 4), (16, 5, 2), (33, 70, 60)])
def test_narrow_domains(nx, ny, nz, dtype):
    """Groups of four, eight, sixteen and 32 lanes, heights that leave groups and
    warps of the last rows idle, one row per group and several."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(nx + ny)
    h, NX, NY = 2, nx + 4, ny + 4
    t = getattr(torch, dtype)
    up = lambda a, d: torch.from_numpy(a).to("cuda", d)  # noqa: E731
    mask = up((rng.uniform(size=(NY, NX)) > 0.3).astype(np.int32), torch.int32)
    pad = torch.nn.functional.pad(mask, (0, 1, 0, 1))
    hu, hv = (up(rng.uniform(0.5, 2.0, (nz, NY, NX)), torch.float64) for _ in range(2))
    u, v = (up(rng.uniform(-1, 1, (nz, NY, NX)), t) for _ in range(2))
    # faces between two land points: no thickness, no velocity
    for f, w, other in ((hu, u, pad[:-1, 1:]), (hv, v, pad[1:, :-1])):
        dry = (mask == 0) & (other == 0)
        f[:, dry] = 0.0
        w[:, dry] = 0.0
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
    # roundings (float thicknesses truncated to 2^-23), then three sums; shears
    # are below 2 / 0.5
    eps = 2.0 ** -53 if dtype == "float64" else 2.0 ** -22
    assert bool(((got - want).abs() <= 16 * eps * want + 8 * eps * 8.0 * want ** 0.5)[:, wet].all())
    SS[1:nz, h:h + ny, h:h + nx][:, wet] = -7.0
    assert bool((SS == -7.0).all())
