"""Open boundaries of any length in one call: points beyond one block's,
long ones between short ones, corners that two boundaries share."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables(lengths, nx):
    """Boundary b lies along row b + 1 from column 0, inward is the row below (the
    boundary before it), but for its point of column b, which it shares with the
    boundary before (a corner, in a column that its others do not read)."""
    i, j, start = [], [], [0]
    for b, n in enumerate(lengths):
        ii, jj = list(range(n)), [b + 1] * n
        if 0 < b < n:
            jj[b] = b
        i += ii
        j += jj
        start.append(len(i))
    ranges = [q for b in range(len(lengths)) for q in (start[b], start[b + 1])]
    return np.array(i, np.int32), np.array(j, np.int32), ranges


LENGTHS = [(1, 256, 257, 3), (255, 512, 513, 40), (2000, 5, 300, 2100)]


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_tracers(lengths, dtype):
    """Zero-gradient and clamped points alternately: exact copies, boundary after
    boundary."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    nb, nx, ny, nz, nt = len(lengths), max(lengths), len(lengths) + 1, 3, 2
    rng = np.random.default_rng(sum(lengths))
    i, j, ranges = _tables(lengths, nx)
    n = i.size
    type_ = np.where(np.arange(n) % 3 == 1, 3, 1).astype(np.int32)
    zero = np.zeros(n, np.int32)
    f = [rng.standard_normal((nz, ny, nx)).astype(dtype) for _ in range(nt)]
    bdy = [rng.standard_normal((nz, n)).astype(dtype) for _ in range(nt)]
    want = [a.copy() for a in f]
    for a, v in zip(want, bdy):
        for b in range(nb):
            for p in range(ranges[2 * b], ranges[2 * b + 1]):
                a[:, j[p], i[p]] = v[:, p] if type_[p] == 3 else a[:, j[p] - 1, i[p]]
    up = [torch.from_numpy(a).cuda() for a in (i, j, type_, zero, zero - 1, np.ones((ny, nx), np.int32))]
    fd, bd = [torch.from_numpy(a).cuda() for a in f], [torch.from_numpy(a).cuda() for a in bdy]
    _lib.call("getm_open_boundaries_tracers" + ("" if dtype == "float64" else "_f32"), nb, (ctypes.c_int * (2 * nb))(*ranges), n,
              nx, ny, nz, 0, *[t.data_ptr() for t in up], nt, _lib.ptr_array([t.data_ptr() for t in fd]),
              _lib.ptr_array([t.data_ptr() for t in bd]), _s())
    for a, b in zip(fd, want):
        assert np.array_equal(a.cpu().numpy(), b)


@pytest.mark.parametrize("lengths", LENGTHS)
def test_elevations(lengths):
    """Zero-gradient, clamped and Flather points in turn.  Copies are exact; a
    Flather value takes a square root, a quotient, a product and two differences:
    6 u of its terms (below 2)."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    nb, nx, ny = len(lengths), max(lengths), len(lengths) + 1
    rng = np.random.default_rng(sum(lengths))
    i, j, ranges = _tables(lengths, nx)
    n = i.size
    type_ = np.array([1, 3, 4, -4])[np.arange(n) % 4].astype(np.int32)
    zero = np.zeros(n, np.int32)
    plane = lambda lo, hi: rng.uniform(lo, hi, (ny, nx))  # noqa: E731
    H, D, U, V, z = plane(5, 50), plane(5, 50), plane(-1, 1), plane(-1, 1), plane(-0.5, 0.5)
    ze, fl, sign = rng.uniform(-0.5, 0.5, n), rng.uniform(-0.1, 0.1, n), np.where(rng.random(n) < 0.5, 1.0, -1.0)
    want = z.copy()
    for b in range(nb):
        for p in range(ranges[2 * b], ranges[2 * b + 1]):
            q = (j[p], i[p])
            if type_[p] == 1:
                v = want[j[p] - 1, i[p]]
            elif type_[p] == 3:
                v = ze[p]
            else:
                v = ze[p] - sign[p] * (V[q] - (fl[p] * D[q] if type_[p] == 4 else fl[p])) / np.sqrt(D[q] * 9.81)
            want[q] = max(0.02 - H[q], v)
    up = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
          (i, j, type_, zero, zero - 1, zero + 4, sign, H, D, U, V, ze, fl)]
    zd = torch.from_numpy(z).cuda()
    _lib.call("getm_open_boundary_elevations", nb, (ctypes.c_int * (2 * nb))(*ranges), n, nx, *[t.data_ptr() for t in up], 0.02,
              zd.data_ptr(), _s())
    assert np.abs(zd.cpu().numpy() - want).max() <= 6 * 1.2e-16 * 2.0


@pytest.mark.parametrize("n", [1536, 1537, 2500])
def test_mirror(n):
    """Pairs on both sides of the number that one block holds."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(n)
    f = torch.from_numpy(rng.standard_normal((2, 6000))).cuda()
    src = rng.permutation(6000)[:n].astype(np.int32)
    tgt = np.roll(src, 1)
    want = f.clone()
    want[:, torch.from_numpy(tgt).long()] = f[:, torch.from_numpy(src).long()]
    ds, dt, work = torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda(), torch.empty(2 * n, dtype=f.dtype, device="cuda")
    _lib.call("getm_mirror", n, ds.data_ptr(), dt.data_ptr(), 2, 6000, f.data_ptr(), work.data_ptr(), _s())
    assert torch.equal(f, want)
