"""Substeps that the fused 2D kernels must leave to the single operations: the
momentum advections' own split."""

import numpy as np
import pytest

from tests.test_gpu_substep_tiles import _assert_same

pytestmark = pytest.mark.gpu


def _member(precision="fp64", prepare=None, fused=True):
    from getm_gb300 import workloads
    from getm_gb300.ensemble import make_member

    wl = workloads.ensemble_member(np.random.default_rng(5), nmin=24, nmax=24, nzmin=4, nzmax=4)
    wl.params["split_factor"] = 4
    s = make_member(wl, precision)
    if prepare is not None:
        prepare(s)
    if not fused:
        s._split2d_plan = lambda *w, **k: None
    return s


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_split_of_the_advections(precision):
    """A split other than the momentum's, given to its advections, holds in
    every substep."""
    from getm_gb300.operators import AdvectionSplit

    def half(s):
        s.momentum.uadv.split_2d = s.momentum.vadv.split_2d = AdvectionSplit.HALF

    a, b = _member(precision, half), _member(precision, half, fused=False)
    for _ in range(9):
        a.advance()
        b.advance()
    _assert_same(a, b)
