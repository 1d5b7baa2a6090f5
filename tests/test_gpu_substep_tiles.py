"""The 2D substep's four launches (getm_split2d_substep): the same state, bit
for bit, as the operations launched one by one."""

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

    from getm_gb300 import checkpoint, workloads
    from getm_gb300.core import Array
    from getm_gb300.ensemble import make_member

    def member(fused):
        wl = workloads.ensemble_member(np.random.default_rng(7), nmin=n, nmax=n, nzmin=4, nzmax=4)
        wl.params["split_factor"] = 5
        s = make_member(wl, precision)
        plans = []
        plan = s._split2d_plan
        s._split2d_plan = (lambda w: plans.append(1) or plan(w)) if fused else (lambda w: None)
        s.momentum.apply_bottom_friction = friction
        if mixed_orders:
            s.momentum.vadv.ufirst = not s.momentum.uadv.ufirst
        for _ in range(7):
            s.advance()
        s.airsea.taux = Array(s.T, 1.5 * s.airsea.taux.all_values)
        for _ in range(6):
            s.advance()
        torch.cuda.synchronize()
        assert len(plans) == (11 if fused else 0)
        return s

    a, b = member(True), member(False)
    sa, sb = checkpoint.state_tensors(a), checkpoint.state_tensors(b)
    bad = [k for k in sa if not bool(((sa[k] == sb[k]) | (torch.isnan(sa[k]) & torch.isnan(sb[k]))).all())]
    assert not bad, bad[:12]
    assert float(a._time) == float(b._time)
