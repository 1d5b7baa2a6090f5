"""Substeps that the fused 2D kernels must leave to the single operations: the
momentum advections' own split, operations that a subclass or a host program has
replaced."""

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


@pytest.mark.parametrize("owner,name,per_substep", [
    ("momentum", "advance_depth_integrated", 1), ("momentum", "update_depth_integrated_diagnostics", 1),
    ("momentum", "_transport_2d_momentum_fused", 1), ("sim", "advance_surface_elevation", 1),
    ("sim", "update_surface_pressure_gradient", 1)])
@pytest.mark.parametrize("by", ["instance", "class"])
def test_replaced_operations_run(owner, name, per_substep, by):
    """An operation replaced on the object or by a subclass runs in every substep
    of a simulation without the substep kernel, with and without a 3D step."""
    calls = []

    def replace(s):
        o = s if owner == "sim" else s.momentum
        own = getattr(type(o), name)

        def counted(self, *a, **k):
            calls.append(name)
            return own(self, *a, **k)

        if by == "instance":
            setattr(o, name, counted.__get__(o))
        else:
            o.__class__ = type("Counting", (type(o),), {name: counted})

    s = _member(prepare=replace)
    for _ in range(6):  # the fourth with a 3D step
        s.advance()
    assert len(calls) >= 6 * per_substep
