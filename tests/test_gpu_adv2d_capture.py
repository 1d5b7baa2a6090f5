"""2D advection captured after 3D advection of one field has sized the handle's
buffers: it allocates nothing more."""

import numpy as np
import pytest

from tests.test_gpu_operators import setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [1, 2, 3])
@pytest.mark.parametrize("increments", ["float64", "float32"])
def test_captured_after_3d(split, increments):
    import torch

    from getm_gb300.core import CENTERS, INTERFACES, Array
    from getm_gb300.operators import Advection, AdvectionScheme, AdvectionSplit

    nz = 5
    _, _, Td, rng = setup(seed=split, nz=nz)
    for g in Td.all_grids():
        g.float_metrics()
    up = lambda g, s, k, z: Array(g, torch.from_numpy(rng.uniform(-s, s, (k, Td.ny_, Td.nx_))).cuda(), z=z)  # noqa: E731
    u3, v3, w3, t3 = up(Td.ugrid, 0.4, nz, CENTERS), up(Td.vgrid, 0.4, nz, CENTERS), up(Td, 1e-4, nz + 1, INTERFACES), up(Td, 9.0, nz, CENTERS)
    flat = lambda a: Array(a.grid, a.all_values[0].clone())  # noqa: E731
    u, v, f = flat(u3), flat(v3), flat(t3)
    want = Array(Td, f.all_values.clone())
    Advection(Td, AdvectionScheme.SUPERBEE, AdvectionSplit(split), increments)(u, v, 30.0, want)
    adv = Advection(Td, AdvectionScheme.SUPERBEE, AdvectionSplit(split), increments)
    adv.apply_3d(u3, v3, w3, 30.0, t3)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        adv(u, v, 30.0, f)
    graph.replay()
    torch.cuda.synchronize()
    assert bool(((f.all_values == want.all_values) | (f.all_values.isnan() & want.all_values.isnan())).all())
