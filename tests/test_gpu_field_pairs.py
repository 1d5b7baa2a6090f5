"""Float column solves of several fields on either side of the rules that choose
between fields side by side (coefficients in shared memory, or in the workspace
with more layers) and pairs in turn: each field gets the bits it gets alone."""

import numpy as np
import pytest

from tests.test_gpu_field_batches import _fields
from tests.test_gpu_operators import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["float32", "float64"])
@pytest.mark.parametrize("sources", [False, True])
@pytest.mark.parametrize("nx,ny,nz,n", [(40, 30, 46, 2), (40, 30, 60, 5), (260, 170, 46, 3), (300, 200, 47, 3), (700, 300, 3, 3)])
def test_column_solve(nx, ny, nz, n, sources, storage):
    """Few columns, just below and above ten warps of them per SM, more than 20."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import VerticalDiffusion

    _, _, Td, rng = setup(seed=nz, nx=nx, ny=ny, nz=nz)
    up = lambda lo, hi, k, z: Array(Td, torch.from_numpy(rng.uniform(lo, hi, (k, Td.ny_, Td.nx_))).to("cuda", torch.float32), z=z)  # noqa: E731
    nuh = up(1e-5, 1e-2, nz + 1, INTERFACES)
    ea2 = [up(-1e-2, 0.0, nz, CENTERS) for _ in range(n)] if sources else None
    ea4 = [up(0.0, 1e-2, nz, CENTERS) for _ in range(n)] if sources else None
    mol = [1e-7 * (q + 1) for q in range(n)]
    a = _fields(Td, rng, n, getattr(torch, storage))
    b = [Array(Td, f.all_values.clone(), z=CENTERS) for f in a]
    vd = VerticalDiffusion(Td, cnpar=0.8)
    vd.batch(nuh, 300.0, a, mol, ea2, ea4)
    for q in range(n):
        vd.batch(nuh, 300.0, b[q:q + 1], mol[q:q + 1], ea2 and ea2[q:q + 1], ea4 and ea4[q:q + 1])
    assert all(torch.equal(x.all_values, y.all_values) for x, y in zip(a, b))
