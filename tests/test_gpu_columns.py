"""Thread-per-column kernels of the 3D momentum at the level counts and domain
sizes where they change the levels they load at once: the same recursions in
numpy."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (nx, ny, nz): parts of a chunk, one level more, whole chunks; few and many columns
SIZES = [(9, 7, 1), (9, 7, 2), (33, 8, 3), (33, 8, 4), (33, 8, 5), (40, 21, 9), (400, 300, 2), (400, 300, 5), (400, 300, 9)]


def _up(a, dtype=None):
    import torch

    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.to(dtype)


@pytest.mark.parametrize("form", ["fp64", "f32"])
@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_vertical_velocity(nx, ny, nz, form):
    """momentum.F90:191-216.  A level adds four products and a thickness change,
    eight roundings of terms below 8 (dy pk iarea and idt dh), nz levels of them;
    float: the same in float with its truncating conversions (2^-22)."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(nz)
    dt = torch.float64 if form == "fp64" else torch.float32
    plane, layers = (ny, nx), (nz, ny, nx)
    mask = (rng.random(plane) < 0.8).astype(np.int32)
    dyu, dxv, ia = (rng.uniform(1.0, 2.0, plane) for _ in range(3))
    ho, hn = rng.uniform(1.0, 2.0, layers), rng.uniform(1.0, 2.0, layers)
    pk, qk = (rng.uniform(-1.0, 1.0, layers).astype(np.float32).astype(float) for _ in range(2))
    w = rng.uniform(-1.0, 1.0, (nz + 1,) + plane).astype(np.float32).astype(float)
    want = w.copy()
    s = slice(2, -2)
    for k in range(1, nz):
        flux = pk[k - 1] * dyu - np.roll(pk[k - 1] * dyu, 1, 1) + qk[k - 1] * dxv - np.roll(qk[k - 1] * dxv, 1, 0)
        new = want[k - 1] - (hn[k - 1] - ho[k - 1]) / 2.0 - flux * ia
        want[k, s, s] = np.where(mask == 1, new, want[k])[s, s]
    got = _up(w, dt)
    up = [_up(a) for a in (mask, dyu, dxv, ia, ho, hn)] + [_up(pk, dt), _up(qk, dt)]
    _lib.call("getm_w_momentum_3d" + ("" if form == "fp64" else "_f32"), nx, ny, nz, 3, nx - 2, 3, ny - 2,
              *[t.data_ptr() for t in up], 2.0, got.data_ptr(), _s())
    err = np.abs(got.double().cpu().numpy() - want)
    assert err.max() <= nz * 8 * 8 * (1.2e-16 if form == "fp64" else 2.0 ** -22)
    land = np.broadcast_to(mask != 1, w.shape)
    assert (err[land] == 0.0).all()


@pytest.mark.parametrize("form", ["fp64", "f32"])
@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_transports_and_sums(nx, ny, nz, form):
    """tp3d = vel hn less the column's share of its excess over tp2d, and the
    column sums.  Products up to 4, sums of nz of them in FP64: 2 nz + 4 roundings
    of at most 4 nz, the share divided by depths above 1."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(nz)
    f64 = form == "fp64"
    dt, sfx, u = (torch.float64, "", 1.2e-16) if f64 else (torch.float32, "_f32", 2.0 ** -22)
    plane, layers = (ny, nx), (nz, ny, nx)
    vel = rng.uniform(-1.0, 1.0, layers).astype(np.float32).astype(float)
    hn, tp2, D = rng.uniform(1.0, 4.0, layers), rng.uniform(-1.0, 1.0, plane), rng.uniform(1.0, 4.0, plane)
    dev = ((vel * hn).sum(0) - tp2) / D
    want = vel * hn - dev * hn
    dv, dh, d2, dD = _up(vel, dt), _up(hn), _up(tp2), _up(D)
    tp3, ddev = torch.empty(layers, dtype=dt, device="cuda"), torch.empty(plane, dtype=torch.float64, device="cuda")
    _lib.call("getm_transport_3d_finish" + sfx, nx, ny, nz, dv.data_ptr(), dh.data_ptr(), d2.data_ptr(), dD.data_ptr(),
              tp3.data_ptr(), ddev.data_ptr(), _s())
    tol = (2 * nz + 4) * 4 * nz * u
    assert np.abs(ddev.cpu().numpy() - dev).max() <= tol
    assert np.abs(tp3.double().cpu().numpy() - want).max() <= 4 * tol
    # the sums themselves: FP64 sums of the stored values, bottom to top, exactly
    outs = [torch.full(plane, 3.0, dtype=torch.float64, device="cuda") for _ in range(2)]
    for subtract in (0, 1):
        _lib.call("getm_column_sums" + sfx, nx, ny, nz, subtract, dv.data_ptr(), outs[0].data_ptr(), None, None,
                  tp3.data_ptr(), outs[1].data_ptr(), None, None, _s())
        for src, got in ((dv, outs[0]), (tp3, outs[1])):
            ref = np.zeros(plane)
            for a in src.double().cpu().numpy():
                ref = ref + a
            assert np.array_equal(got.cpu().numpy(), ref if subtract == 0 else ref - ref)


@pytest.mark.parametrize("form", ["fp64", "f32"])
def test_vertical_velocity_of_any_domain(form):
    """Columns of a small domain, and the same columns repeated over one beyond the
    size up to which four levels are loaded at once: the same bits."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(1)
    dt = torch.float64 if form == "fp64" else torch.float32
    nx, ny, nz, outs = 40, 30, 11, []
    r = lambda lo, hi, *k: rng.uniform(lo, hi, (*k, ny, nx))  # noqa: E731
    fields = [np.ones((ny, nx), np.int32), r(1990, 2010), r(1990, 2010), r(2.4e-7, 2.6e-7), r(90, 110, nz), r(90, 110, nz),
              r(-10, 10, nz), r(-10, 10, nz), 0 * r(0, 1, nz + 1)]
    for reps in ((1, 1), (9, 8)):
        up = [_up(np.tile(a, (1,) * (a.ndim - 2) + reps)) for a in fields]
        up[6:] = [t.to(dt) for t in up[6:]]
        ny_, nx_ = up[0].shape
        _lib.call("getm_w_momentum_3d" + ("" if form == "fp64" else "_f32"), nx_, ny_, nz, 3, nx_ - 2, 3, ny_ - 2,
                  *[t.data_ptr() for t in up[:8]], 120.0, up[8].data_ptr(), _s())
        outs.append(up[8][:, 2:ny - 2, 2:nx - 2])
    assert torch.equal(*outs) and float(outs[0].abs().max()) > 0.0
