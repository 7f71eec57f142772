"""The two-at-a-time fused x passes (scalar fluxes, Smagorinsky stress) at every
tile shape: against the oracle up to 128^3 (1e-10, the step's own tolerance), and
the scalar pass at 512^3 against a torch FP64 transform of the same step."""
import numpy as np
import pytest

from _cases import make_pair, relerr, seed_scalars

pytestmark = pytest.mark.gpu


def _compare(o, g, nf):
    f = g.download_fields()
    for m in range(nf):
        assert relerr(f[m], o.fields[m]) < 1e-10, f"field {m}"


@pytest.mark.parametrize("prune", [True, False])
@pytest.mark.parametrize("n", [32, 48, 64, 128])
def test_scalar_fluxes_match_oracle(n, prune):
    o, g = make_pair(n, dealias=0, nu=1.0 / 300.0, dt=0.1 / n, nscal=2, sc=[0.7, 1.0], scalar_type=[0, 0], isp_type=2)
    seed_scalars(o, g, 2, np.random.default_rng(n))
    g.upload_fields(np.ascontiguousarray(o.fields))
    g.dealias_all()
    o.fields[:] = g.download_fields()
    g.set_pruning(prune)
    assert g.pruned == prune
    o.step(3)
    g.step(3)
    _compare(o, g, 5)


@pytest.mark.parametrize("prune", [True, False])
@pytest.mark.parametrize("n", [32, 48, 64, 128])
def test_smagorinsky_stress_matches_oracle(n, prune):
    o, g = make_pair(n, dealias=0, nu=1.0 / 2000.0, dt=0.1 / n, les_model=1, isp_type=2)
    g.set_pruning(prune)
    assert g.pruned == prune
    o.step(3)
    g.step(3)
    _compare(o, g, 3)


@pytest.mark.parametrize("n", [256, 512])
def test_scalar_fluxes_match_torch_at_large_grids(n):
    import torch
    from hit3d_b200 import Context, Params
    nu, dt = 1.0 / 300.0, 0.1 / n
    c = Context(Params(nx=n, nu=nu, dt=dt, n_scalars=1, sc=[0.7], scalar_type=[1]))
    c.init_velocity(1234567.0, 2, 4.0, 2.0)
    f = c.download_fields()
    f[3] = f[0][::-1]  # a field of the same spectrum; dealiased below
    c.upload_fields(f)
    c.dealias_all()
    f = torch.from_numpy(c.download_fields()).cuda()
    c.step(1)
    got = torch.from_numpy(c.download_fields()[3]).cuda()
    c.close()
    u = [torch.view_as_complex(q.reshape(n, n, n // 2 + 1, 2)).transpose(0, 1).contiguous() for q in f]
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    k = torch.where(2 * k > n, k - n, k)
    kk = (k[: n // 2 + 1].view(1, 1, -1), k.view(1, -1, 1), k.view(-1, 1, 1))
    keep = sum((q.abs() > n // 3).int() for q in kk) == 0
    # kx = 0 without conjugate symmetry: complex along z and y, real along x
    ph = [torch.fft.irfft(torch.fft.ifft(torch.fft.ifft(q, dim=0), dim=1), n=n, dim=2) for q in u]
    r = sum(-1j * kk[j] * torch.fft.rfftn(ph[3] * ph[j]) for j in range(3)) - nu / 0.7 * sum(q * q for q in kk) * u[3]
    ref = u[3] + dt * torch.where(keep, r, torch.zeros_like(r))
    ref = torch.view_as_real(ref.transpose(0, 1).contiguous()).reshape(n, n, n + 2)
    assert float((got - ref).abs().max() / ref.abs().max()) < 1e-12
