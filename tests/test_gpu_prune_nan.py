"""A state that is not finite beyond N/3 is not pruned: steps and statistics show the
NaN or infinity as the unpruned passes do, instead of skipping its mode."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, -np.nan, np.inf])
@pytest.mark.parametrize("field,history", [(0, False), (3, False), (1, True)])
def test_not_finite_beyond_the_cutoff(bad, field, history):
    from hit3d_b200 import Context, Params
    n = 32
    out = []
    for prune in (True, False):
        c = Context(Params(nx=n, nu=1.0 / 300.0, dt=0.002, n_scalars=1, sc=[0.7], scalar_type=[0]))
        c.set_pruning(prune)
        c.init_velocity(RN1, 2, 4.0, 2.0)
        c.init_scalar(0, 987654.0, 4.0)
        c.dealias_all()
        c.step(1)
        assert c.pruned == prune
        f = c.download_rhs_old() if history else c.download_fields()
        f[field, 0, 1, 2 * (n // 3 + 2)] = bad
        (c.upload_rhs_old if history else c.upload_fields)(f)
        assert not c.pruned
        es, st = c.stats()
        ss = c.scalar_stats(0)
        if not history:
            assert not np.isfinite(st["enstrophy"] if field < 3 else ss["diss"])
        c.step(1)
        out.append([es, np.array(list(st.values())), ss["spectrum"], ss["diss"], c.download_fields(), c.download_rhs_old()])
        c.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)
