"""The k-epsilon closure where interior turbulence has vanished: a zero kinetic
energy gives its interface an infinite sink, and only that interface."""

import numpy as np
import pytest

from tests.gpu_helpers import dev, host
from tests.test_gpu_operators import close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [2, 3, 12])
def test_zero_kinetic_energy(nz):
    """Single interfaces of every column, whole columns, and none.  One step;
    random columns of developed turbulence, so the tolerance is the one of the
    closure's own test: 100 times the oracle's response to a viscosity two units in
    the last place away, at least 1e-12."""
    import torch

    from getm_gb300.core import INTERFACES, Array, make_grids
    from getm_gb300.vertical_mixing import GOTM
    from oracle import turbulence as K
    from tests.helpers import full_grid

    Th, rng = full_grid(nx=24, ny=18, nz=nz, seed=nz)
    Td = make_grids(Th)
    shape = (nz + 1, Th.ny_, Th.nx_)
    plane = shape[1:]
    h = np.where(Th.mask[None] != 0, rng.uniform(0.5, 3.0, (nz,) + plane), 1.0)
    Td.hn.all_values.copy_(torch.from_numpy(h))
    NN, SS = rng.uniform(-1e-5, 1e-4, shape), rng.uniform(0.0, 1e-3, shape)
    us, ub = rng.uniform(0.0, 0.02, plane), rng.uniform(0.0, 0.02, plane)
    z0s, z0b = np.full(plane, 0.1), rng.uniform(0.001, 0.01, plane)
    vm = GOTM()
    vm.initialize(Td, dtype=torch.float64)
    k0, e0 = rng.uniform(1e-6, 1e-4, shape), rng.uniform(1e-9, 1e-7, shape)
    nu0 = vm.params.cm0 ** 4 * k0 * k0 / e0
    at = rng.integers(1, nz, plane)  # an interior interface of each column
    k0[at, np.arange(plane[0])[:, None], np.arange(plane[1])[None, :]] = 0.0
    k0[1:nz, :, 5] = 0.0
    k0[:, :, 9] = 1e-5
    o = dict(tke=k0, eps=e0, L=np.zeros(shape), num=nu0, nuh=nu0.copy())
    for n in ("tke", "eps", "num", "nuh"):
        getattr(vm, n).all_values.copy_(torch.from_numpy(o[n]))
    p = {n: x.copy() for n, x in o.items()}
    p["num"] = p["num"] * (1.0 + 4.4e-16)
    vm.advance(600.0, *[Array(Td, dev(a)) for a in (us, ub, z0s, z0b)], Array(Td, dev(NN), z=INTERFACES),
               Array(Td, dev(SS), z=INTERFACES))
    for st in (o, p):
        K.keps_advance(Th, 600.0, h, us, ub, z0s, z0b, NN, SS, st["tke"], st["eps"], st["L"], st["num"], st["nuh"])
    sel = np.zeros(plane, dtype=bool)
    sel[2:-2, 2:-2] = Th.mask[2:-2, 2:-2] == 1
    for n in ("tke", "eps", "L", "num", "nuh"):
        a, b = o[n][:, sel], p[n][:, sel]
        assert np.isfinite(a).all()
        spread = float(np.abs(a - b).max() / np.abs(a).max())
        close(host(getattr(vm, n).all_values), o[n], max(1e-12, 100.0 * spread), sel)
