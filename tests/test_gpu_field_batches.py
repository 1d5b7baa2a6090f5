"""Fields of a batch swept side by side (column solve, x and y advection
passes): each field gets the bits it gets alone."""

import numpy as np
import pytest

from tests.test_gpu_operators import setup

pytestmark = pytest.mark.gpu


def _fields(Td, rng, n, dtype):
    import torch

    from getm_gb300.core import CENTERS, Array

    return [Array(Td, torch.from_numpy(rng.uniform(5.0, 15.0, (Td.nz, Td.ny_, Td.nx_))).to("cuda", dtype), z=CENTERS)
            for _ in range(n)]


@pytest.mark.parametrize("storage", ["float32", "float64"])
@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("nz", [1, 2, 20, 45, 46])
def test_column_solve(nz, sources, storage):
    """One layer, two, and both sides of the layer count up to which the
    coefficients stay in shared memory."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import VerticalDiffusion

    _, _, Td, rng = setup(seed=nz, nz=nz)
    n, dt = 3, getattr(torch, storage)
    nuh = Array(Td, torch.from_numpy(rng.uniform(1e-5, 1e-2, (nz + 1, Td.ny_, Td.nx_))).to("cuda", torch.float32),
                z=INTERFACES)
    src = lambda s: [Array(Td, torch.from_numpy(s * rng.uniform(0, 1e-2, (nz, Td.ny_, Td.nx_))).to("cuda", torch.float32),  # noqa: E731
                           z=CENTERS) for _ in range(n)] if sources else None
    ea2, ea4, mol = src(-1.0), src(1.0), [1e-7 * (q + 1) for q in range(n)]
    a = _fields(Td, rng, n, dt)
    b = [Array(Td, f.all_values.clone(), z=CENTERS) for f in a]
    vd = VerticalDiffusion(Td, cnpar=0.8)
    vd.batch(nuh, 300.0, a, mol, ea2, ea4)
    for q in range(n):
        vd.batch(nuh, 300.0, b[q:q + 1], mol[q:q + 1], ea2 and ea2[q:q + 1], ea4 and ea4[q:q + 1])
    assert all(torch.equal(x.all_values, y.all_values) for x, y in zip(a, b))


@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("nx,ny,nz", [(40, 30, 1), (40, 30, 2), (40, 30, 44), (40, 30, 45), (700, 300, 3)])
def test_column_solve_fp64(nx, ny, nz, sources):
    """FP64: few columns on both sides of the layer count up to which the
    coefficients stay in shared memory, and more columns than are resident."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import VerticalDiffusion

    _, _, Td, rng = setup(seed=nz, nx=nx, ny=ny, nz=nz)
    n = 3
    up = lambda lo, hi, k, z: Array(Td, torch.from_numpy(rng.uniform(lo, hi, (k, Td.ny_, Td.nx_))).cuda(), z=z)  # noqa: E731
    nuh = up(1e-5, 1e-2, nz + 1, INTERFACES)
    ea2 = [up(-1e-2, 0.0, nz, CENTERS) for _ in range(n)] if sources else None
    ea4 = [up(0.0, 1e-2, nz, CENTERS) for _ in range(n)] if sources else None
    mol = [1e-7 * (q + 1) for q in range(n)]
    a = _fields(Td, rng, n, torch.float64)
    b = [Array(Td, f.all_values.clone(), z=CENTERS) for f in a]
    vd = VerticalDiffusion(Td, cnpar=0.8)
    vd.batch(nuh, 300.0, a, mol, ea2, ea4)
    for q in range(n):
        vd.batch(nuh, 300.0, b[q:q + 1], mol[q:q + 1], ea2 and ea2[q:q + 1], ea4 and ea4[q:q + 1])
    assert all(torch.equal(x.all_values, y.all_values) for x, y in zip(a, b))


@pytest.mark.parametrize("nx,ny,nz,n", [(60, 9, 4, 3), (31, 70, 9, 5), (124, 33, 20, 2), (252, 40, 6, 9)])
@pytest.mark.parametrize("form", ["mixed", "f32"])
def test_advection(nx, ny, nz, n, form):
    """Rows that fill the four-cell chunks alone and in fours, rows of odd
    length, few and many rows per warp."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import Advection, AdvectionScheme

    _, _, Td, rng = setup(seed=n, nx=nx, ny=ny, nz=nz)
    vel = lambda g, z, k, s: Array(g, torch.from_numpy(rng.uniform(-s, s, (k, Td.ny_, Td.nx_))).to("cuda", torch.float32), z=z)  # noqa: E731
    u, v, w = vel(Td.ugrid, CENTERS, nz, 0.5), vel(Td.vgrid, CENTERS, nz, 0.5), vel(Td, INTERFACES, nz + 1, 1e-4)
    a = _fields(Td, rng, n, torch.float64 if form == "mixed" else torch.float32)
    b = [Array(Td, f.all_values.clone(), z=CENTERS) for f in a]
    adv = Advection(Td, AdvectionScheme.SUPERBEE)
    adv.apply_3d_batch(u, v, w, 10.0, a)
    for q in range(n):
        adv.apply_3d_batch(u, v, w, 10.0, b[q:q + 1])
    wet = Td.mask.all_values == 1
    assert all(torch.equal(x.all_values[:, wet], y.all_values[:, wet]) for x, y in zip(a, b))
