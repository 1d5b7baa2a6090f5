"""The FP64 internal pressure gradient in whole tiles (8 rows, 4 levels), which
the domains of the other tests are too small for, against the same domain in
strips of few columns, whose tiles are half as high and of one level."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nz", [(37, 6), (64, 5), (61, 12)])
def test_strips_of_a_domain(ny, nz):
    """Copies of a strip side by side, land between them: every copy gets the
    bits the strip gets alone."""
    import torch

    from getm_gb300 import _lib
    from getm_gb300._pygetm import _s

    rng = np.random.default_rng(ny)
    w = 32  # columns of a strip, the outer two on either side land
    n = -(-6 * 152 * 32 // (w * -(-ny // 8) * -(-nz // 4))) + 1
    strip = lambda lo, hi, *k: rng.uniform(lo, hi, (*k, ny + 4, w))  # noqa: E731
    mask = np.zeros((ny + 4, w), np.int32)
    mask[2:-2, 2:-2] = rng.random((ny, w - 4)) < 0.85
    um, vm = np.zeros_like(mask), np.zeros_like(mask)
    um[:, :-1] = mask[:, :-1] * mask[:, 1:]
    vm[:-1] = mask[:-1] * mask[1:]
    h = strip(0.5, 1.5, nz)
    zc = h.cumsum(0) - 0.5 * h - h.sum(0)
    fields = [mask, um, vm, strip(0.1, 1.0), strip(0.1, 1.0), h, strip(-0.1, 0.1), zc, strip(0.0, 1e-3, nz).cumsum(0)]
    outs = []
    for reps in (1, n):
        up = [torch.from_numpy(np.ascontiguousarray(np.tile(a, (1,) * (a.ndim - 1) + (reps,)))).cuda() for a in fields]
        nx = w * reps
        gx, gy, work = (torch.zeros((k, ny + 4, nx), dtype=torch.float64, device="cuda") for k in (nz, nz, nz + 2))
        _lib.call("getm_shchepetkin_mcwilliams", nx, ny + 4, nz, 3, nx - 2, 3, ny + 2, *[t.data_ptr() for t in up],
                  gx.data_ptr(), gy.data_ptr(), work.data_ptr(), _s())
        outs.append((gx, gy))
    for one, many in zip(*outs):
        assert float(one.abs().max()) > 0.0
        got = many.view(nz, ny + 4, n, w)
        assert torch.equal(got, one[:, :, None, :].expand_as(got))
