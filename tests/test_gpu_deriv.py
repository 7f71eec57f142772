"""The closures' strains and gradients from the velocity's own z inverse, on states
with energy in every mode (Nyquist planes, not solenoidal) and on the 2/3-rule band:
Smagorinsky and the dynamic localization model against the oracle, the learned
closure with Smagorinsky weights against Smagorinsky.

Tolerances are those of the step parity (1e-10) and of the learned closure's
equivalence with Smagorinsky (1e-6) on the same quantities."""
import numpy as np
import pytest

from _cases import make_pair, relerr
from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _state(o, nf, seed):
    n = o.n
    rng = np.random.default_rng(seed)
    out = np.zeros((nf, n, n, n + 2))
    for m in range(nf):
        out[m, :, :, :n] = rng.standard_normal((n, n, n)) if m < 3 else 1.0 + 0.3 * rng.random((n, n, n))
        o.fft3d(1, out[m])
    return out


@pytest.mark.parametrize("full", [True, False])
@pytest.mark.parametrize("n,model", [(32, 1), (48, 1), (64, 1), (32, 2), (48, 2)])
def test_strains_match_oracle(n, model, full):
    o, g = make_pair(n, flow_type=1, kfmax=2, nu=1.0 / 2000.0, dt=1e-3, les_model=model, c_smag=0.18)
    f = _state(o, o.fields.shape[0], n + model)
    o.fields[:] = f
    if not full:
        o.dealias_all()
    g.upload_fields(np.ascontiguousarray(o.fields))
    if model == 1:
        assert g.pruned == (not full)
    o.step(1)
    g.step(1)
    h = g.download_fields()
    # the strains' stress acts on the velocity; k_sgs of a state beyond N/3 in every
    # field, which no run holds, is not compared
    for m in range(h.shape[0] if not full else 3):
        assert relerr(h[m], o.fields[m]) < 1e-10, m
    g.close()


@pytest.mark.parametrize("n", [32, 48, 64, 128])
def test_gradients_match_smagorinsky(n):
    from hit3d_b200 import Context, Params
    dx, delta = 2 * np.pi / n, 4 * np.pi / n
    g1 = float(mo.bf16_round(np.float32(-2 * 0.18 ** 2 * dx * dx / delta ** 2)).item())
    cs = np.sqrt(-g1 * delta ** 2 / (2 * dx * dx))
    w = mo.smagorinsky_params(0.0, dx, delta)
    w[-5] = g1
    f = np.fft.rfft(np.random.default_rng(n).standard_normal((3, n, n, n)), axis=3)  # (f, z, y, kx)
    f = np.fft.fft(np.fft.fft(f, axis=2), axis=1).transpose(0, 2, 1, 3)               # (f, ky, kz, kx)
    f = np.ascontiguousarray(f).view(np.float64)
    out = []
    for model in (1, 20, 0):
        c = Context(Params(nx=n, flow_type=1, kfmax=2, nu=1.0 / 2000.0, dt=1e-3, les_model=model, c_smag=cs))
        if model == 20:
            c.les_set_mlp(mo.bf16_bits(w), delta, clip=False, kernel=1)
        c.upload_fields(f)
        c.step(1)
        out.append(c.download_fields())
        c.close()
    assert relerr(out[1], out[0]) < 1e-6
    assert relerr(out[2], out[0]) > 1e-4
