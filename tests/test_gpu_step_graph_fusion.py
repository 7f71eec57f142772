"""The fusion switch takes effect on steps that are replayed from a recording, one
step a call (a call of several fused steps chains them and is never replayed)."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extra", [(32, {}), (64, dict(flow_type=1, kfmax=2)), (48, dict(n_scalars=1, sc=[0.7], scalar_type=[0])),
                                     (32, dict(precision=1))])
def test_fusion_switch_between_replayed_steps(n, extra):
    from hit3d_b200 import Context, Params
    a, b = (Context(Params(nx=n, nu=1.0 / 500.0, dt=0.1 / n, **extra)) for _ in range(2))
    for c in (a, b):
        c.init_velocity(RN1, 2, 4.0, 2.0)
        c.dealias_all()
    per_step = []
    for on in (False, True, False):
        for c in (a, b):
            c.set_update_fusion(on)
        for i in range(50):  # past the steps before a recording
            la, lb = a.launches, b.launches
            a.step(1)
            b.step_profile(1)
            assert a.launches - la == b.launches - lb, (on, i)
        per_step.append(a.launches - la)
        assert np.array_equal(a.download_fields(), b.download_fields())
        assert np.array_equal(a.download_rhs_old(), b.download_rhs_old())
    # one launch fewer, unless a scalar's products keep a z pass of their own
    assert per_step == [per_step[0], per_step[0] - (0 if extra.get("n_scalars") else 1), per_step[0]]
    a.close()
    b.close()
