"""The 2D substep's four launches (getm_split2d_substep) and its phases
(getm_split2d_phases): the same state, bit for bit, as the operations launched
one by one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,mixed_orders,friction", [(8, False, True), (31, True, True), (61, False, False)])
def test_substep_matches_single_operations(precision, n, mixed_orders, friction):
    """Planes smaller than a block, one short of whole tiles and of several
    tiles; the two momentum advections in different orders; a wind field
    replaced after the start."""
    import torch

    from getm_gb300 import workloads
    from getm_gb300.core import Array
    from getm_gb300.ensemble import make_member

    def member(fused):
        wl = workloads.ensemble_member(np.random.default_rng(7), nmin=n, nmax=n, nzmin=4, nzmax=4)
        wl.params["split_factor"] = 5
        s = make_member(wl, precision)
        plans = []
        plan = s._split2d_plan
        s._split2d_plan = lambda *w, **k: plans.append(k) or plan(*w, **k) if fused else None
        s.momentum.apply_bottom_friction = friction
        if mixed_orders:
            s.momentum.vadv.ufirst = not s.momentum.uadv.ufirst
        for _ in range(7):
            s.advance()
        s.airsea.taux = Array(s.T, 1.5 * s.airsea.taux.all_values)
        for _ in range(6):
            s.advance()
        torch.cuda.synchronize()
        assert len(plans) == (13 if fused else 0)  # 11 whole substeps, 2 with a 3D step
        return s

    _assert_same(member(True), member(False))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ufirst", [True, False])
def test_phases_with_open_boundaries(precision, ufirst):
    """A shelf sea with tidal, clamped and sponge boundaries: mirrored
    transports between the phases, depths outside the boundaries, elevations
    before the surface pressure gradient."""
    import torch

    from getm_gb300 import workloads

    def shelf(fused):
        wl = workloads.shelf_sea(nx=45, ny=38, nz=5, ntracer=3, seed=2)
        wl.params.update(split_factor=3)
        s = workloads.start_shelf_sea(wl, precision)
        s.momentum._ufirst = ufirst
        if not fused:
            s._split2d_plan = lambda *w, **k: None
        for _ in range(10):
            s.advance()
        torch.cuda.synchronize()
        return s

    _assert_same(shelf(True), shelf(False))


def _assert_same(a, b):
    import torch

    from getm_gb300 import checkpoint

    sa, sb = checkpoint.state_tensors(a), checkpoint.state_tensors(b)
    bad = [k for k in sa if not bool(((sa[k] == sb[k]) | (torch.isnan(sa[k]) & torch.isnan(sb[k]))).all())]
    assert not bad, bad[:12]
    assert float(a._time) == float(b._time)
