"""A batch replays its recorded steps only while every switch of every run is what it
was at the recording: a run of a batch, switched between calls, stays bit for bit
the run stepped on its own."""
import numpy as np
import pytest

from _cases import RN1
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu
N = 32


def _closure(c, seed, clip, delta):
    c.les_set_mlp(mo.bf16_bits(mo.smagorinsky_params(0.1 + 0.01 * seed, 2 * np.pi / N, delta)), delta, clip=clip, kernel=0)


def _idle(c):
    c.set_scalars_active(False)


def _active(c):
    c.set_scalars_active(True)


CASES = [
    # the idle passive scalars of a model with transported fields
    (dict(les_model=2, n_scalars=1, sc=[0.7], scalar_type=[0], flow_type=1, kfmax=2), None, [_idle, _active]),
    # the closure's clip switch and filter width (weights are read from the same place)
    (dict(les_model=20, flow_type=1, kfmax=2), lambda c: _closure(c, 0, False, 0.4),
     [lambda c: _closure(c, 0, False, 0.6), lambda c: _closure(c, 1, True, 0.6)]),
    # the fusion switch and launch shapes
    (dict(n_scalars=1, sc=[0.7], scalar_type=[0]), None,
     [lambda c: c.set_update_fusion(True), lambda c: (c.set_update_fusion(False), c.set_variant(8), c.set_column_tile(1))]),
]


def _run(extra, start, changes, batched):
    from hit3d_b200 import Context, Params
    from hit3d_b200.batch import Batch
    p = Params(nx=N, nu=1.0 / 500.0, dt=0.1 / N, **extra)
    b = Batch([p, Params(nx=N, nu=1.0 / 300.0, dt=0.1 / N)]) if batched else None
    c = b.contexts[0] if batched else Context(p)
    for q in b.contexts if batched else [c]:
        q.init_velocity(RN1, 2, 4.0, 2.0)
        q.dealias_all()
    if start:
        start(c)
    out = []
    for change in [None] + changes:
        if change:
            change(c)
        steps = 10 if change else 11  # the first step is first order, outside the recording
        if batched:
            b.step(steps, 5)
        else:
            for _ in range(steps):
                c.step(1)
        out += [c.download_fields(), c.download_rhs_old()]
    if batched:
        assert b.graph_launches == 6
    (b or c).close()
    return out


@pytest.mark.parametrize("case", range(len(CASES)))
def test_switch_between_calls(case):
    for x, y in zip(_run(*CASES[case], True), _run(*CASES[case], False)):
        assert np.array_equal(x, y)
