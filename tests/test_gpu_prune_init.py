"""A Taylor-Green start is checked like any other change of the state: its transform
leaves rounding beyond N/3, so that what was known of the state before (here: all
zero, pruned) must not carry over."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(32, 0), (64, 0), (32, 1)])
def test_taylor_green_state_is_checked(n, precision):
    from hit3d_b200 import Context, Params
    out = []
    for look_first in (False, True):
        c = Context(Params(nx=n, nu=0.01, dt=0.01, precision=precision))
        if look_first:
            assert c.pruned
            c.stats()
        c.init_velocity(RN1, -1)
        pruned = c.pruned
        es = c.stats()[0]
        c.step(3)
        out.append([pruned, es, c.download_fields(), c.download_rhs_old()])
        c.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
