"""When a small grid's step is recorded: steps are replayed, not only issued, once
they have kept one key, and a key that keeps changing does not pay for recordings."""
import numpy as np
import pytest

from _cases import RN1
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _make(n, **extra):
    from hit3d_b200 import Context, Params
    c = Context(Params(nx=n, nu=1.0 / 500.0, dt=0.1 / n, **extra))
    if extra.get("les_model") == 20:
        delta = 4 * np.pi / n
        c.les_set_mlp(mo.bf16_bits(mo.smagorinsky_params(0.15, 2 * np.pi / n, delta)), delta, clip=True, kernel=1)
    c.init_velocity(RN1, 2, 4.0, 2.0)
    c.dealias_all()
    return c


@pytest.mark.parametrize("n,extra,filtered", [
    (32, {}, False), (48, dict(precision=1), False), (64, dict(les_model=20, flow_type=1, kfmax=2), False),
    (32, dict(les_model=20, precision=1), False), (32, {}, True), (32, dict(les_model=1, n_scalars=1, sc=[0.7], scalar_type=[0]), False),
    (32, dict(les_model=3), False), (32, dict(les_model=4), False), (32, dict(les_model=5, c_t=1.0), False),
    (32, dict(les_model=6, c_mixed=0.5), False), (32, dict(les_model=7, c_mixed=0.5), False),
    (32, dict(les_model=10, c_mixed=0.5, n_scalars=1, sc=[0.7], scalar_type=[0]), False), (128, {}, False)])
def test_recorded_and_replayed(n, extra, filtered):
    a, b = _make(n, **extra), _make(n, **extra)
    if filtered:
        x = np.random.default_rng(5).uniform(1.0, n + 1.0, (100, 3))
        for c in (a, b):
            c.particles_filter(8 * np.pi / n)
            c.particles_upload(x)
    for _ in range(9):  # a first-order step and eight with one key
        assert a.step_graph == (0, 0)
        a.step(1)
    assert a.step_graph == (1, 0)
    for k in range(6):
        a.step(1)
    assert a.step_graph == (1, 6)
    a.set_dt(0.05 / n)
    a.step(20)  # the second of twenty is recorded
    assert a.step_graph == (2, 25)
    b.step_profile(15)
    b.set_dt(0.05 / n)
    b.step_profile(20)
    assert np.array_equal(a.download_fields(), b.download_fields())
    assert np.array_equal(a.download_rhs_old(), b.download_rhs_old())
    if filtered:
        assert np.array_equal(a.particles_download()[0], b.particles_download()[0])
    a.close()
    b.close()


@pytest.mark.parametrize("every,most", [(5, 0), (9, 1), (12, 1), (17, 2)])
def test_changing_time_step_pays_for_few_recordings(every, most):
    c = _make(32)
    c.step(1)
    for i in range(40):
        c.set_dt(0.003 * (1.0 + 1e-6 * i))
        for _ in range(every):
            c.step(1)
    assert c.step_graph[0] <= most
    c.set_dt(0.002)  # a key that stays is recorded after all
    c.step(50)
    assert c.step_graph[1] >= 40
    c.close()


def test_calls_of_a_few_steps_and_large_grids():
    c = _make(32)
    c.step(1)
    for i in range(6):  # seven-step calls of one key each: no recording
        c.set_dt(0.003 * (1.0 + 1e-6 * i))
        c.step(7)
    assert c.step_graph == (0, 0)
    c.close()
    c = _make(256)
    c.step(20)
    assert c.step_graph == (0, 0)
    c.close()
