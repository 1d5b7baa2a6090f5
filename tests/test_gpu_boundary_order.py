"""Boundary updates in one launch: the boundaries in turn, the mirrored points
and the tide, against plain numpy and torch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 513, 4096, 4097])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_mirror_reads_before_it_writes(n, dtype):
    """Chains of pairs (a target that is the source of another pair), within
    one block's registers and beyond them: exact copies."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(n)
    nlev, plane = 3, 5000
    f = torch.from_numpy(rng.standard_normal((nlev, plane))).to("cuda", getattr(torch, dtype))
    src = rng.permutation(plane)[:n].astype(np.int32)
    tgt = np.roll(src, 1)  # every source is another pair's target
    want = f.clone()
    want[:, torch.from_numpy(tgt).long()] = f[:, torch.from_numpy(src).long()]
    ds, dt = (torch.from_numpy(a).cuda() for a in (src, tgt))
    work = torch.empty(n * nlev, dtype=f.dtype, device="cuda")
    _lib.call("getm_mirror_f32" if dtype == "float32" else "getm_mirror", n, ds.data_ptr(), dt.data_ptr(), nlev, plane,
              f.data_ptr(), work.data_ptr(), _s())
    assert torch.equal(f, want)


@pytest.mark.parametrize("npts", [1, 255, 257, 700])
def test_boundaries_in_turn(npts):
    """Zero-gradient boundaries whose source points belong to the boundary
    before them: the values arrive through all of them, in order."""
    import ctypes

    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _p, _s  # noqa: F401

    nb, nx, nz, nt = 3, npts, 4, 2
    rng = np.random.default_rng(npts)
    j = np.repeat(np.arange(1, nb + 1), npts).astype(np.int32)
    i = np.tile(np.arange(npts), nb).astype(np.int32)
    z = np.zeros(nb * npts, np.int32)
    ranges = (ctypes.c_int * (2 * nb))(*[q for b in range(nb) for q in (b * npts, (b + 1) * npts)])
    up = {k: torch.from_numpy(a).cuda() for k, a in dict(i=i, j=j, type=z + 1, di=z, dj=z - 1, mask=np.ones((nb + 1, nx), np.int32)).items()}
    fs = [torch.from_numpy(rng.standard_normal((nz, nb + 1, nx))).cuda() for _ in range(nt)]
    first = [f[:, :1].clone() for f in fs]
    ptrs = _lib.ptr_array([f.data_ptr() for f in fs])
    _lib.call("getm_open_boundaries_tracers", nb, ranges, nb * npts, nx, nb + 1, nz, 0, up["i"].data_ptr(), up["j"].data_ptr(),
              up["type"].data_ptr(), up["di"].data_ptr(), up["dj"].data_ptr(), up["mask"].data_ptr(), nt, ptrs, ptrs, _s())
    for f, row in zip(fs, first):
        assert torch.equal(f, row.expand_as(f))


@pytest.mark.parametrize("nc", [1, 2, 17])
def test_tide_matches_torch(nc):
    """Sum of constituents, beyond one launch's number too: the torch
    expression's operations in its order, so the same bits."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s
    import ctypes

    rng = np.random.default_rng(nc)
    npts = 201
    cs = [(float(rng.uniform(1e-5, 2e-4)), torch.from_numpy(rng.uniform(0, 2, npts)).cuda(),
           torch.from_numpy(rng.uniform(-3, 3, npts)).cuda()) for _ in range(nc)]
    time = torch.tensor(123456.7, dtype=torch.float64, device="cuda")
    want = torch.zeros(npts, dtype=torch.float64, device="cuda")
    for om, a, p in cs:
        want.add_(a * (time * om + p).cos())
    z = torch.full((npts,), 7.0, dtype=torch.float64, device="cuda")
    _lib.call("getm_open_boundary_tide", npts, nc, (ctypes.c_double * nc)(*[c[0] for c in cs]),
              _lib.ptr_array([c[1].data_ptr() for c in cs]), _lib.ptr_array([c[2].data_ptr() for c in cs]),
              time.data_ptr(), z.data_ptr(), _s())
    assert torch.equal(z, want)
