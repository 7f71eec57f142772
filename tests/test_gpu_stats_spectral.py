"""Statistics summed over the modes (spectrum, enstrophy, scalar dissipation)
against the same quantities from the physical fields, for states with energy in
every mode: the Nyquist planes, and kx = 0 without conjugate symmetry, where the
real transform keeps the symmetric part only.

Tolerance 1e-12 relative: sums of at most 2e6 terms of one sign, FP64, both
sides' rounding below 1e-13."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _waves(n):
    k = np.arange(n)
    k = np.where(2 * k > n, k - n, k).astype(float)
    return k[: n // 2 + 1].reshape(1, 1, -1), k.reshape(1, -1, 1), k.reshape(-1, 1, 1)


def _phys(f):
    """c2r of (kz, ky, kx) as the passes do it: complex along z and y, then real along x."""
    n = f.shape[0]
    return np.fft.irfft(np.fft.ifft(np.fft.ifft(f, axis=0), axis=1), n=n, axis=2)


def _context(n, seed, dealias=False):
    from hit3d_b200 import Context, Params
    c = Context(Params(nx=n, n_scalars=1, sc=[0.7], scalar_type=[0], nu=1.0 / 300.0))
    f = np.random.default_rng(seed).standard_normal((4, n, n, n + 2)) * n ** 1.5
    c.upload_fields(f)
    if dealias:
        c.dealias_all()
        f = c.download_fields()
        assert c.pruned
    u = (f[..., 0::2] + 1j * f[..., 1::2]).transpose(0, 2, 1, 3)  # (f, kz, ky, kx)
    return c, u


@pytest.mark.parametrize("n,dealias", [(32, False), (48, False), (64, False), (128, False), (32, True), (48, True), (128, True)])
def test_mode_sums_match_physical_fields(n, dealias):
    c, u = _context(n, n, dealias)
    kx, ky, kz = _waves(n)
    es, st = c.stats()
    w = [1j * (ky * u[2] - kz * u[1]), 1j * (kz * u[0] - kx * u[2]), 1j * (kx * u[1] - ky * u[0])]
    ens = sum((_phys(q) ** 2).mean() for q in w)
    assert abs(st["enstrophy"] - ens) <= 1e-12 * ens
    sh = np.rint(np.sqrt((kx * kx + ky * ky + kz * kz).astype(np.float32))).astype(int)[:, :, : n // 2]
    e = sum(q.real ** 2 + q.imag ** 2 for q in u[:3])[:, :, : n // 2] / float(n) ** 6
    e[:, :, 0] *= 0.5
    ref = np.bincount(sh.ravel(), e.ravel())[1: c.kmax + 1]
    assert np.all(np.abs(es - ref) <= 1e-12 * ref)
    sk = np.mean([(d ** 3).mean() / (d ** 2).mean() ** 1.5 for d in (_phys(1j * k * q) for k, q in zip((kx, ky, kz), u))])
    assert abs(st["skewness"] - sk) <= 1e-12
    ss = c.scalar_stats(0)
    diss = 2.0 * (1.0 / 300.0) / 0.7 * sum((_phys(1j * k * u[3]) ** 2).mean() for k in (kx, ky, kz))
    phi = _phys(u[3])
    assert abs(ss["diss"] - diss) <= 1e-12 * diss
    assert abs(ss["variance"] - phi.var()) <= 1e-12 * phi.var()
    assert abs(ss["min"] - phi.min()) <= 1e-12 * abs(phi.min()) and abs(ss["max"] - phi.max()) <= 1e-12 * abs(phi.max())
    c.close()
