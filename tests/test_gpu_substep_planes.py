"""The 2D substep's kernels on planes beyond one wave of small tiles: the same
state, bit for bit, as the operations launched one by one."""

import numpy as np
import pytest

from tests.test_gpu_substep_tiles import _assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [150, 180, 260])
def test_substep_on_larger_planes(precision, n):
    """150: depth tiles of six rows whose halves go to different warps, the mixed
    form without early launches, friction shared among the first pass's blocks;
    180: eight rows, one thread per point; 260: nine rows, the FP64 y passes in
    blocks of 16 rows."""
    import torch

    from getm_gb300 import workloads
    from getm_gb300.ensemble import make_member

    def member(fused):
        wl = workloads.ensemble_member(np.random.default_rng(n), nmin=n, nmax=n, nzmin=3, nzmax=3)
        wl.params["split_factor"] = 4
        s = make_member(wl, precision)
        if not fused:
            s._split2d_plan = lambda *w, **k: None
        for _ in range(10):
            s.advance()
        torch.cuda.synchronize()
        assert float(s.momentum.U.all_values[s.U.water].abs().max()) > 0.0
        return s

    _assert_same(member(True), member(False))
