"""Two scalars through one fused x pass against the same scalars one at a time, at
every tile shape, both dealias modes, with and without an unpaired third scalar.

Tolerance 1e-12 relative: the same operations, contracted otherwise, FP64, three
steps."""
import numpy as np
import pytest

from _cases import RN1, relerr

pytestmark = pytest.mark.gpu


def _run(n, which, dealias, prune):
    from hit3d_b200 import Context, Params
    sc, ty = [0.7, 1.0, 1.3], [0, 1, 0]
    c = Context(Params(nx=n, dealias=dealias, nu=1.0 / 300.0, dt=0.1 / n, n_scalars=len(which),
                       sc=[sc[s] for s in which], scalar_type=[ty[s] for s in which]))
    c.set_pruning(prune)
    c.init_velocity(RN1, 2, 4.0, 2.0)
    f = c.download_fields()
    for i, s in enumerate(which):
        f[3 + i] = np.roll(f[s], 1 + s, axis=0)  # not conjugate symmetric along the rolled axis
    c.upload_fields(f)
    c.dealias_all()
    c.step(3)
    out = c.download_fields()
    c.close()
    return out


@pytest.mark.parametrize("n,ns,dealias,prune", [(32, 2, 0, True), (48, 3, 0, True), (48, 2, 1, False), (64, 2, 0, False),
                                               (128, 3, 1, False), (256, 2, 0, True), (512, 2, 0, True)])
def test_paired_scalars_match_single_ones(n, ns, dealias, prune):
    both = _run(n, list(range(ns)), dealias, prune)
    for s in range(ns):
        one = _run(n, [s], dealias, prune)
        assert relerr(both[3 + s], one[3]) < 1e-12
        if s == 0:
            assert relerr(both[:3], one[:3]) < 1e-12
