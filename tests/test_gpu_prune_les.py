"""The pruning switch never changes a result: the LES models whose clipped fields or
filtered products hold modes beyond N/3 stay unpruned with the switch on."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,nsc", [(3, 0), (3, 1), (4, 0), (5, 0), (6, 0), (7, 0), (10, 0), (10, 1)])
def test_switch_keeps_the_bits(model, nsc):
    from hit3d_b200 import Context, Params
    n, out = 32, []
    for prune in (True, False):
        c = Context(Params(nx=n, flow_type=1, kfmax=2, nu=1.0 / 2000.0, dt=0.128 / n, les_model=model, n_scalars=nsc,
                           sc=[0.7][:nsc], scalar_type=[0] * nsc, c_t=1.0, c_mixed=0.5))
        c.set_pruning(prune)
        c.init_velocity(RN1, 2, 4.0, 2.0)
        f = c.download_fields()
        f[3 + nsc, 0, 0, 2] = 0.15 * n ** 3  # negative on part of the domain
        c.upload_fields(f)
        c.dealias_all()
        assert not c.pruned
        c.step(6)
        out.append([c.download_fields(), c.download_rhs_old(), np.array(list(c.les_stats().values())), c.stats()[0]])
        c.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
