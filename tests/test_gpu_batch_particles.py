"""Particles of a batch's run uploaded again between calls: the recorded steps hold the
old arrays, which are gone, and must be recorded again."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


def test_particles_uploaded_between_calls():
    from hit3d_b200 import Context, Params
    from hit3d_b200.batch import Batch
    n = 32
    p = Params(nx=n, nu=1.0 / 500.0, dt=0.1 / n, n_scalars=1, sc=[0.7], scalar_type=[0])
    b = Batch([p])
    a, c = b.contexts[0], Context(p)
    x = np.random.default_rng(3).uniform(1.0, n + 1.0, (300, 3))
    for q in (a, c):
        q.init_velocity(RN1, 2, 4.0, 2.0)
        q.dealias_all()
    for m, delta, steps in ((200, None, 11), (300, None, 10), (77, 1.0, 10), (0, None, 10), (150, None, 10)):
        for q in (a, c):
            q.particles_upload(x[:m])
            if delta is not None:
                q.particles_filter(delta)
        b.step(steps, 5)
        c.step(steps)
        assert np.array_equal(a.download_fields(), c.download_fields())
        if m:
            for u, v in zip(a.particles_download(), c.particles_download()):
                assert np.array_equal(u, v)
    assert b.graph_launches == 10
    b.close()
    c.close()
