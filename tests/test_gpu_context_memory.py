"""A context holds its state, AB2 history and work fields and one field to stage
transfers, whatever the number of fields; the work fields that small grids' transfers
pass through leave nothing behind for the next step."""
import numpy as np
import pytest

from _cases import RN1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nsc,precision", [(128, 4, 0), (128, 0, 0), (128, 2, 1)])
def test_device_memory_of_a_context(n, nsc, precision):
    import torch
    from hit3d_b200 import Context, Params
    Context(Params(nx=32)).close()  # what the library holds once
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    cs = [Context(Params(nx=n, n_scalars=nsc, sc=[1.0] * nsc, scalar_type=[0] * nsc, precision=precision)) for _ in range(4)]
    used = (free - torch.cuda.mem_get_info()[0]) / 4
    for c in cs:
        c.close()
    nh = n // 2 + 1
    f64, f32 = 16 * n * n * ((nh + 7) // 8 * 8), 8 * n * n * ((nh + 15) // 16 * 16)
    w = 6 + 3 * nsc
    expect = 2 * (3 + nsc) * f64 + (w * f64 if precision == 0 else w * f32 + 3 * f64) + 16 * n * n * nh
    # allocations round up to 2 MB; one field more is 17 MB
    assert used <= expect + 14e6, (used, expect)


@pytest.mark.parametrize("n,extra", [(32, {}), (48, dict(n_scalars=1, sc=[0.7], scalar_type=[1])), (64, dict(precision=1)),
                                     (128, dict(precision=1, les_model=1)), (32, dict(les_model=2)),
                                     (32, dict(dealias=1, n_scalars=2, sc=[0.7, 1.0], scalar_type=[1, 0]))])
@pytest.mark.parametrize("tile", [0, 3])
def test_transfers_leave_nothing_in_the_work_fields(n, extra, tile):
    from hit3d_b200 import Context, Params
    a, b = (Context(Params(nx=n, nu=1.0 / 500.0, dt=0.1 / n, **extra)) for _ in range(2))
    for c in (a, b):
        c.set_column_tile(tile)
        c.init_velocity(RN1, 2, 4.0, 2.0)
        if 1 in extra.get("scalar_type", []):
            c.init_scalar(0, 987654.0, 4.0)
        c.dealias_all()
    bad = np.full(a.field_shape(), np.nan)
    for steps in (1, 2, 1):
        f, r = a.download_fields(), a.download_rhs_old()
        a.upload_fields(bad)
        a.upload_rhs_old(bad)  # the work fields now hold NaN throughout
        assert np.isnan(a.download_rhs_old()).all()
        a.upload_rhs_old(r[:1])
        a.upload_fields(f[:1])  # the first field through a staging area that keeps NaN behind it
        a.upload_rhs_old(r)
        a.upload_fields(f)
        assert np.array_equal(a.download_fields(), f) and np.array_equal(a.download_rhs_old(), r)
        assert a.step(steps) == b.step(steps)
    assert np.array_equal(a.download_fields(), b.download_fields())
    assert np.array_equal(a.download_rhs_old(), b.download_rhs_old())
    a.close()
    b.close()
