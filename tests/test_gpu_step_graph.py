"""Steps of small grids replayed from a recorded graph give the fields of steps
issued one by one (step_profile issues every launch), bit for bit, through every
change that drops the recording."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu

CASES = [(32, dict(flow_type=1, kfmax=2)), (48, dict(n_scalars=1, sc=[0.7], scalar_type=[0])), (32, dict(dealias=1)),
         (32, dict(les_model=2)), (32, dict(les_model=1, precision=1)), (128, dict(flow_type=1, kfmax=2))]


@pytest.mark.parametrize("n,extra", CASES)
def test_recorded_steps_are_the_issued_ones(n, extra):
    from hit3d_b200 import Context, Params
    a, b = (Context(Params(nx=n, nu=1.0 / 500.0, dt=0.1 / n, **extra)) for _ in range(2))
    for c in (a, b):
        c.init_velocity(RN1, 2, 4.0, 2.0)
        c.dealias_all()

    def go(steps):
        l0 = a.launches
        a.step(steps)
        la, l0 = a.launches - l0, b.launches
        b.step_profile(steps)
        assert la == b.launches - l0  # replayed kernels are counted
        assert np.array_equal(a.download_fields(), b.download_fields())
        assert np.array_equal(a.download_rhs_old(), b.download_rhs_old())

    go(12)
    go(1)
    for c in (a, b):
        c.set_dt(0.05 / n)
    go(12)
    for c in (a, b):
        c.set_variant(8)
        c.set_column_tile(1)
    go(7)
    if not extra.get("les_model"):
        for c in (a, b):
            c.set_pruning(False)
        go(7)
        x = np.random.default_rng(3).uniform(1.0, n + 1.0, (200, 3))
        for c in (a, b):
            c.particles_upload(x)
        go(7)
        for c in (a, b):
            c.particles_upload(x[:77])
        go(7)
        assert np.array_equal(a.particles_download()[0], b.particles_download()[0])
    if extra.get("n_scalars"):
        for c in (a, b):
            c.set_scalars_active(False)
        go(7)
    for c in (a, b):
        c.fov = 1
    go(6)  # a first-order step again, then recorded ones
    a.close()
    b.close()
