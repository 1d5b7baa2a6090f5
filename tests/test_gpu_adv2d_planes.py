"""2D advection of planes large enough for the FP64 y pass's blocks of 16 rows
(more than 304 tiles of 32 x 15), against the oracle.

Tolerance as for the smaller planes: 1e-14 of the largest value."""

import pytest

from tests.gpu_helpers import host
from tests.test_gpu_operators import close, setup, velocity, wrap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(350, 420), (391, 500)])
@pytest.mark.parametrize("split", [1, 2, 3])
def test_against_oracle(nx, ny, split):
    import oracle.oracle as O
    from getm_gb300 import operators

    Th, To, Td, rng = setup(nz=1, seed=ny, nx=nx, ny=ny)
    assert -(-Td.nx_ // 32) * ((Td.ny_ + 15) // 15) > 304
    u, v = velocity(Th.ugrid, rng, 1, 0.3)[0], velocity(Th.vgrid, rng, 1, 0.3)[0]
    t = rng.uniform(5.0, 10.0, (Th.ny_, Th.nx_))
    ao = O.Advection(To, 5, O.AdvectionSplit(split))
    to = t.copy()
    ao(u, v, 600.0, to)
    ad = operators.Advection(Td, operators.AdvectionScheme(5), operators.AdvectionSplit(split))
    td = wrap(Td, t, False)
    ad(wrap(Td.ugrid, u, False), wrap(Td.vgrid, v, False), 600.0, td)
    close(host(td.all_values), to, rtol=1e-14)
    close(host(ad.D), ao.D, rtol=1e-14)
