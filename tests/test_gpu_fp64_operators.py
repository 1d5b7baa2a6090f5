"""FP64 operators at the sizes where their kernels can go wrong: rows and
columns around the 31-cell segments and 15-row tiles of the horizontal passes,
batches around the field groups, land that holds NaN.

Tolerance: a directional pass rounds at most about five times per cell in
either order of evaluation (u = 1.1e-16 each, weights at most one, h/hnew
below 1.2), five passes make some 30 u; 1e-14 is 90 u of the field's largest
value."""

import numpy as np
import pytest

from tests.gpu_helpers import host
from tests.test_gpu_operators import close, setup, velocity, wrap

pytestmark = pytest.mark.gpu
RTOL = 1e-14


@pytest.mark.parametrize("nx,ny,nz,nt,scheme", [(3, 3, 2, 1, 5), (26, 10, 3, 2, 1), (27, 11, 1, 3, 2), (28, 12, 4, 1, 3),
                                                (58, 26, 5, 5, 4), (59, 27, 2, 33, 5), (89, 41, 3, 2, 6)])
def test_split_at_tile_edges(nx, ny, nz, nt, scheme):
    import oracle.oracle as O
    from getm_gb300 import operators
    from getm_gb300.core import CENTERS, INTERFACES

    Th, To, Td, rng = setup(nz=nz, seed=nx, nx=nx, ny=ny)
    u, v = velocity(Th.ugrid, rng, nz, 0.3), velocity(Th.vgrid, rng, nz, 0.3)
    w = rng.uniform(-5e-4, 5e-4, (nz + 1, Th.ny_, Th.nx_))
    w[0] = w[-1] = 0.0
    tr = [rng.uniform(5.0, 10.0, (nz, Th.ny_, Th.nx_)) for _ in range(nt)]
    ah = [rng.uniform(0, 50.0, (Th.ny_, Th.nx_)) for _ in range(2)] if nt > 1 else [None, None]
    for t in tr:
        t[:, Th.mask == 0] = np.nan
    ao = O.Advection(To, scheme)
    tro = [t.copy() for t in tr]
    ao.apply_3d_batch(u, v, w, 600.0, tro, Ah_u=ah[0], Ah_v=ah[1])
    ad = operators.Advection(Td, operators.AdvectionScheme(scheme))
    trd = [wrap(Td, t, CENTERS) for t in tr]
    ad.apply_3d_batch(wrap(Td.ugrid, u, CENTERS), wrap(Td.vgrid, v, CENTERS), wrap(Td, w, INTERFACES), 600.0, trd,
                      Ah_u=None if ah[0] is None else wrap(Td.ugrid, ah[0], False),
                      Ah_v=None if ah[1] is None else wrap(Td.vgrid, ah[1], False))
    water = Th.mask != 0
    for a, b in zip(trd, tro):
        got = host(a.all_values)
        assert np.isnan(got[:, ~water]).all()
        close(got, b, rtol=RTOL, mask=water)
    close(host(ad.h), ao.h, rtol=RTOL)


@pytest.mark.parametrize("nx,ny", [(3, 3), (27, 11), (58, 26)])
@pytest.mark.parametrize("split", [1, 2, 3])
def test_plane_split_at_tile_edges(nx, ny, split):
    import oracle.oracle as O
    from getm_gb300 import operators

    Th, To, Td, rng = setup(nz=1, seed=ny, nx=nx, ny=ny)
    u, v = velocity(Th.ugrid, rng, 1, 0.3)[0], velocity(Th.vgrid, rng, 1, 0.3)[0]
    t = rng.uniform(5.0, 10.0, (Th.ny_, Th.nx_))
    ao = O.Advection(To, 5, O.AdvectionSplit(split))
    to = t.copy()
    ao(u, v, 600.0, to)
    ad = operators.Advection(Td, operators.AdvectionScheme(5), operators.AdvectionSplit(split))
    td = wrap(Td, t, False)
    ad(wrap(Td.ugrid, u, False), wrap(Td.vgrid, v, False), 600.0, td)
    close(host(td.all_values), to, rtol=RTOL)
    close(host(ad.D), ao.D, rtol=RTOL)


@pytest.mark.parametrize("nx,ny,nz,scheme,wmax", [(3, 3, 1, 5, 5e-4), (30, 12, 2, 1, 5e-4), (31, 13, 3, 3, 5e-3),
                                                  (60, 20, 9, 5, 2e-2), (29, 50, 40, 4, 2e-3)])
def test_vertical_pass_columns(nx, ny, nz, scheme, wmax):
    """Batches of one to three fields, the last with its own velocity, in
    columns of one to forty levels with Courant numbers from below one to
    several sub-steps.  A sub-step rounds some 15 u where the field's own
    velocity moves up to four layers' worth of it; six of them stay below
    1e-13."""
    import oracle.oracle as O
    from getm_gb300 import operators
    from getm_gb300.core import CENTERS, INTERFACES

    Th, To, Td, rng = setup(nz=nz, seed=nz, nx=nx, ny=ny)
    zero3 = lambda g: np.zeros((nz, g.ny_, g.nx_))  # noqa: E731
    w = rng.uniform(-2e-4, 2e-4, (nz + 1, Th.ny_, Th.nx_))
    own = rng.uniform(-wmax, wmax, w.shape)
    for a in (w, own):
        a[0] = a[-1] = 0.0
    for nt in (1, 2, 3):
        tr = [rng.uniform(5.0, 10.0, (nz, Th.ny_, Th.nx_)) for _ in range(nt)]
        ws = [own if q == 2 or nt == 1 else w for q in range(nt)]
        ao = O.Advection(To, scheme)
        tro = [t.copy() for t in tr]
        it = iter(ws)
        ao.apply_3d_batch(zero3(Th.ugrid), zero3(Th.vgrid), w, 300.0, tro, get_w=lambda _: next(it))
        ad = operators.Advection(Td, operators.AdvectionScheme(scheme))
        trd = [wrap(Td, t, CENTERS) for t in tr]
        wd, od = wrap(Td, w, INTERFACES), wrap(Td, own, INTERFACES)
        itd = iter([od if x is own else wd for x in ws])
        ad.apply_3d_batch(wrap(Td.ugrid, zero3(Th.ugrid), CENTERS), wrap(Td.vgrid, zero3(Th.vgrid), CENTERS), wd, 300.0,
                          trd, get_w=lambda _: next(itd))
        for a, b in zip(trd, tro):
            close(host(a.all_values), b, rtol=1e-13)
        close(host(ad.h), ao.h, rtol=RTOL)


def _diffuse_extended(x, nuh, ho, hn, dt, mol, cnpar, ea2, ea4):
    """diffusion.F90:135-314 of columns [k, n] in numpy's widest float."""
    x, nuh, ho, hn = (np.asarray(a, dtype=np.longdouble) for a in (x, nuh, ho, hn))
    nz, zero = x.shape[0], np.zeros_like(x[:1])
    c = 2 * np.longdouble(dt) * (nuh[1:-1] + np.longdouble(mol))
    ao, an = (1 - np.longdouble(cnpar)) * c / (ho[1:] + ho[:-1]), np.longdouble(cnpar) * c / (hn[1:] + hn[:-1])
    up, lo = np.concatenate([an, zero]), np.concatenate([zero, an])
    flux = ao * np.diff(x, axis=0)
    diag = hn + up + lo - (0 if ea2 is None else ea2)
    rhs = x * ho + np.concatenate([flux, zero]) - np.concatenate([zero, flux]) + (0 if ea4 is None else ea4)
    r, q = np.zeros_like(x), np.zeros_like(x)
    rk = qk = zero[0]
    for k in range(nz - 1, -1, -1):
        den = diag[k] - up[k] * rk
        r[k], q[k] = rk, qk = lo[k] / den, (rhs[k] + up[k] * qk) / den
    for k in range(1, nz):
        q[k] += r[k] * q[k - 1]
    return q.astype(np.float64)


@pytest.mark.parametrize("nx,ny,nz,cnpar,sources", [(3, 3, 1, 1.0, True), (29, 9, 2, 1.0, False), (28, 8, 3, 0.6, True),
                                                    (61, 20, 40, 1.0, True), (60, 5, 255, 0.6, False)])
def test_column_solve_levels(nx, ny, nz, cnpar, sources):
    """Fused, prepared and workspace-free solves of one to 255 levels, against
    the same system solved in extended precision (the oracle's own sweep loses
    digits to strong mixing).  A row of the elimination rounds about six times,
    and strong mixing carries a level's error to all: 6 nz u, and ten for the
    rest."""
    from getm_gb300 import operators
    from getm_gb300._lib import call
    from getm_gb300.core import CENTERS, INTERFACES

    Th, To, Td, rng = setup(nz=nz, seed=nz, nx=nx, ny=ny)
    rtol = (10 + 6 * nz) * 1.2e-16
    nuh = 10.0 ** rng.uniform(-6, -1, (nz + 1, Th.ny_, Th.nx_))
    t = rng.uniform(5.0, 10.0, (nz, Th.ny_, Th.nx_))
    t[:, Th.mask == 0] = np.nan
    ea2 = -rng.uniform(0, 0.1, t.shape) if sources else None
    ea4 = rng.uniform(0, 0.1, t.shape) if sources else None
    water = Th.mask != 0
    for use_ho in (False, True):
        to = _diffuse_extended(t[:, water], nuh[:, water], (To.ho if use_ho else To.hn)[:, water], To.hn[:, water], 600.0,
                               1e-6, cnpar, *[None if e is None else e[:, water] for e in (ea2, ea4)])
        vd = operators.VerticalDiffusion(Td, cnpar)
        nd = wrap(Td, nuh, INTERFACES)
        e2, e4 = [None if e is None else wrap(Td, e, CENTERS) for e in (ea2, ea4)]
        fused, other, prepared, bare = [wrap(Td, t, CENTERS) for _ in range(4)]
        vd.batch(nd, 600.0, [fused, other], [1e-6, 1e-6], [e2, e2], [e4, e4], use_ho)
        vd.prepare(nd, 600.0, 1e-6, use_ho)
        vd.apply(prepared, e2, e4, use_ho)
        arr = lambda *x: operators._lib.ptr_array([None if a is None else a.all_values.data_ptr() for a in x])  # noqa: E731
        mol = (operators.ctypes.c_double * 1)(1e-6)
        call("getm_vertical_diffusion_batch", Td.nx_, Td.ny_, nz, Td.mask.all_values.data_ptr(), nd.all_values.data_ptr(),
             600.0, cnpar, (Td.ho if use_ho else Td.hn).all_values.data_ptr(), Td.hn.all_values.data_ptr(), 1, mol,
             arr(bare), arr(e2), arr(e4), None, operators._s())
        for got in (fused, other, prepared, bare):
            close(host(got.all_values)[:, water], to, rtol=rtol)


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 1), (30, 8, 2), (31, 9, 4), (33, 16, 5), (64, 7, 13)])
def test_internal_pressure_tiles(nx, ny, nz):
    """Around the tiles of 32 columns, 8 rows and 4 levels.  The gradient is a
    difference of column integrals P of nz terms, each rounded some ten times;
    with the Jacobian's own ten that is 10 (nz + 2) u of the largest P, times the
    thickness and the inverse spacing."""
    import oracle.oracle as O
    import torch
    from getm_gb300 import _pygetm
    from getm_gb300.core import CENTERS, Array

    Th, To, Td, rng = setup(nz=nz, seed=nx + nz, nx=nx, ny=ny)
    for g, d in ((To, Td),):
        hn = np.where(Th.mask != 0, g.hn, 0.0)
        zf = np.concatenate([0 * hn[:1], hn.cumsum(axis=0)]) - np.where(Th.mask != 0, g.D, 0.0)
        g.zc[...] = 0.5 * (zf[1:] + zf[:-1])
        d.zc.all_values.copy_(torch.from_numpy(g.zc))
    z = rng.uniform(-0.3, 0.3, To.D.shape)
    b = np.sort(rng.uniform(-0.05, 0.0, (nz,) + z.shape), axis=0)
    b[:, Th.mask == 0] = np.nan
    ox, oy = np.zeros_like(b), np.zeros_like(b)
    O.shchepetkin_mcwilliams(To, b, ox, oy, z)
    Td.zin = Array(Td, torch.from_numpy(z).cuda())
    gx, gy = Td.ugrid.array(z=CENTERS, fill=0.0), Td.vgrid.array(z=CENTERS, fill=0.0)
    _pygetm.shchepetkin_mcwilliams(wrap(Td, b, CENTERS), gx, gy)
    hmax = hn.max()
    scale = 0.05 * hn.sum(axis=0).max() * hmax / 1000.0
    for got, want in ((gx, ox), (gy, oy)):
        err = np.abs(host(got.all_values) - want)
        assert np.isfinite(err).all()
        assert err.max() <= 10 * (nz + 2) * 1.2e-16 * scale
