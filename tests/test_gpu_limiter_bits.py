"""Float advection passes with every limiter: a field's bits depend neither on
the fields it is advected with nor on whether its column is shared by several
warps."""

import numpy as np
import pytest

from tests.test_gpu_field_batches import _fields
from tests.test_gpu_operators import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("form", ["mixed", "f32"])
def test_batch_partner(scheme, form):
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import Advection, AdvectionScheme

    nx, ny, nz, n = 60, 37, 9, 3
    _, _, Td, rng = setup(seed=scheme, nx=nx, ny=ny, nz=nz)
    vel = lambda g, z, k, s: Array(g, torch.from_numpy(rng.uniform(-s, s, (k, Td.ny_, Td.nx_))).to("cuda", torch.float32), z=z)  # noqa: E731
    u, v, w = vel(Td.ugrid, CENTERS, nz, 0.5), vel(Td.vgrid, CENTERS, nz, 0.5), vel(Td, INTERFACES, nz + 1, 2e-3)
    a = _fields(Td, rng, n, torch.float64 if form == "mixed" else torch.float32)
    b = [Array(Td, f.all_values.clone(), z=CENTERS) for f in a]
    adv = Advection(Td, AdvectionScheme(scheme))
    adv.apply_3d_batch(u, v, w, 100.0, a)
    for q in range(n):
        adv.apply_3d_batch(u, v, w, 100.0, b[q:q + 1])
    wet = Td.mask.all_values == 1
    assert all(torch.equal(x.all_values[:, wet], y.all_values[:, wet]) for x, y in zip(a, b))


@pytest.mark.parametrize("scheme", [1, 3, 5])
@pytest.mark.parametrize("form", ["mixed", "f32"])
def test_shared_columns(scheme, form):
    """Vertical motion alone: the columns of a small domain, whose levels several
    warps share, against the same columns repeated over one of 20 and more warps
    of columns per SM."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import Advection, AdvectionScheme

    nz, out = 17, []
    rng = np.random.default_rng(scheme)
    nx, ny = 28, 12
    w0 = rng.uniform(-4e-3, 4e-3, (nz + 1, ny, nx))
    w0[0] = w0[-1] = 0.0
    f0, h0 = rng.uniform(5.0, 15.0, (nz, ny, nx)), rng.uniform(0.3, 1.0, (nz, ny, nx))
    for reps in ((1, 1), (30, 11)):
        _, _, Td, _ = setup(seed=1, nx=nx * reps[1], ny=ny * reps[0], nz=nz)
        tile = lambda a: np.pad(np.tile(a, (1,) + reps), ((0, 0), (2, 2), (2, 2)), mode="edge")  # noqa: E731
        up = lambda a, t: torch.from_numpy(tile(a)).to("cuda", t)  # noqa: E731
        Td.mask.all_values.fill_(1)
        for g in (Td.ugrid, Td.vgrid):
            g.mask.all_values.zero_()  # no horizontal transports
        Td.ho.all_values.copy_(up(h0, torch.float64))
        zero = lambda g: Array(g, torch.zeros((nz, Td.ny_, Td.nx_), dtype=torch.float32, device="cuda"), z=CENTERS)  # noqa: E731
        f = Array(Td, up(f0, torch.float64 if form == "mixed" else torch.float32), z=CENTERS)
        Advection(Td, AdvectionScheme(scheme)).apply_3d(zero(Td.ugrid), zero(Td.vgrid), Array(Td, up(w0, torch.float32), z=INTERFACES),
                                                        100.0, f)
        out.append(f.all_values[:, 2:2 + ny, 2:2 + nx].clone())
    assert torch.equal(out[0], out[1])
    assert not torch.equal(out[0], torch.from_numpy(f0).to(out[0]))
