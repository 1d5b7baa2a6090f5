"""The 2D substep as one launch per phase (getm_split2d_substep_phases): the
same state, bit for bit, as the operations launched one by one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,mixed_orders,friction", [(8, False, True), (31, True, True), (61, False, False)])
def test_phases_match_single_operations(precision, n, mixed_orders, friction):
    """Planes smaller than a block, one short of whole tiles and of several
    tiles; the two momentum advections in different orders; a wind field
    replaced after the start."""
    import torch

    from getm_gb300 import checkpoint, workloads
    from getm_gb300.core import Array
    from getm_gb300.ensemble import make_member

    def member(phases):
        wl = workloads.ensemble_member(np.random.default_rng(7), nmin=n, nmax=n, nzmin=4, nzmax=4)
        wl.params["split_factor"] = 5
        s = make_member(wl, precision)
        plans = []
        plan = s._split2d_plan
        s._split2d_plan = (lambda **k: plans.append(1) or plan(**k)) if phases else (lambda **k: None)
        s.momentum.apply_bottom_friction = friction
        if mixed_orders:
            s.momentum.vadv.ufirst = not s.momentum.uadv.ufirst
        for _ in range(7):
            s.advance()
        s.airsea.taux = Array(s.T, 1.5 * s.airsea.taux.all_values)
        for _ in range(6):
            s.advance()
        torch.cuda.synchronize()
        assert len(plans) == (11 if phases else 0)
        return s

    a, b = member(True), member(False)
    sa, sb = checkpoint.state_tensors(a), checkpoint.state_tensors(b)
    bad = [k for k in sa if not bool(((sa[k] == sb[k]) | (torch.isnan(sa[k]) & torch.isnan(sb[k]))).all())]
    assert not bad, bad[:12]
    assert float(a._time) == float(b._time)
