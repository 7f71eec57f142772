"""2/3-rule pruning of the dynamic localization model: every field but k_sgs takes
the pruned passes, bit-identical with the unpruned step, also once clipping has
brought k_sgs modes beyond N/3 into the state."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


def _run(n, nsc, clip, prune):
    from hit3d_b200 import Context, Params
    c = Context(Params(nx=n, flow_type=1, kfmax=2, nu=1.0 / 2000.0, dt=0.128 / n, les_model=2, n_scalars=nsc,
                       sc=[0.7][:nsc], scalar_type=[0] * nsc))
    c.set_pruning(prune)
    c.init_velocity(RN1, 2, 4.0, 2.0)
    if nsc:
        c.init_scalar(0, 987654.0, 4.0)
    if clip:
        f = c.download_fields()
        f[3 + nsc, 0, 0, 2] = 0.15 * n ** 3  # + 0.3 cos(x) on a mean of 0.1: negative on part of the domain
        c.upload_fields(f)
    c.dealias_all()
    out = []
    for steps in (1, 1, 8):
        assert c.pruned == prune
        cour = c.step(steps)
        out += [c.download_fields(), c.download_rhs_old(), np.float64(cour)]
        out += [np.array(list(c.les_stats().values())), c.scalar_stats(nsc)["spectrum"], c.stats()[0]]
    c.close()
    return out


@pytest.mark.parametrize("n,nsc,clip", [(32, 0, False), (32, 0, True), (48, 1, True), (64, 0, True), (128, 0, True), (128, 1, False)])
def test_pruned_dlm_step_is_bit_identical(n, nsc, clip):
    a, b = _run(n, nsc, clip, True), _run(n, nsc, clip, False)
    kc = n // 3
    if clip:
        assert np.abs(a[0][3 + nsc][:, :, 2 * (kc + 1):]).max() > 0.0  # modes beyond N/3 did appear
    for i, (x, y) in enumerate(zip(a, b)):
        if i % 6 < 4:
            assert np.array_equal(x, y), i
        else:  # spectra: the kept modes are summed in another order
            assert np.all(np.abs(x - y) <= 1e-12 * np.abs(y).max()), i
