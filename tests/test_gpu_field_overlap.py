"""Column solves of a batch whose fields share memory (one given twice, one that
is another's source) are swept in turn, not side by side."""

import numpy as np
import pytest

from tests.test_gpu_field_batches import _fields
from tests.test_gpu_operators import setup

pytestmark = pytest.mark.gpu


def _same(a, b):
    return bool(((a == b) | (a.isnan() & b.isnan())).all())


@pytest.mark.parametrize("nz", [2, 20])
@pytest.mark.parametrize("form", ["fp64", "mixed", "f32"])
def test_column_solve(form, nz):
    """FP64: the fields one after the other, the later ones seeing what the
    earlier ones left.  Float: in pairs, whose sweeps read both fields' old values."""
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import VerticalDiffusion

    _, _, Td, rng = setup(seed=nz, nz=nz)
    field = torch.float32 if form == "f32" else torch.float64
    other = torch.float64 if form == "fp64" else torch.float32
    nuh = Array(Td, torch.from_numpy(rng.uniform(1e-5, 1e-2, (nz + 1, Td.ny_, Td.nx_))).to("cuda", other), z=INTERFACES)
    vd = VerticalDiffusion(Td)
    copy = lambda f: Array(Td, f.all_values.clone(), z=CENTERS)  # noqa: E731
    (f, g) = _fields(Td, rng, 2, field)
    # twice: applied twice in turn, once where the pair's sweeps run together
    a, b = copy(f), copy(f)
    vd.batch(nuh, 300.0, [a, a], [0.0, 0.0])
    for _ in range(2 if form == "fp64" else 1):
        vd.batch(nuh, 300.0, [b], [0.0])
    assert _same(a.all_values, b.all_values) and not _same(a.all_values, f.all_values)
    if field != other:
        return
    # the second's source is the first: its new values in turn, its old ones in a pair
    a, b, c, d = copy(f), copy(g), copy(f), copy(g)
    vd.batch(nuh, 300.0, [a, b], [0.0, 0.0], ea4s=[None, a])
    old = copy(f)
    vd.batch(nuh, 300.0, [c], [0.0])
    vd.batch(nuh, 300.0, [d], [0.0], ea4s=[c if form == "fp64" else old])
    assert _same(a.all_values, c.all_values) and _same(b.all_values, d.all_values)
