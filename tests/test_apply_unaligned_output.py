"""Operator apply and lift into device memory that is not aligned for doubles (a field of a
packed record): copied there, not written by a kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 4])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_unaligned_output(orc, geo, precision, offset):
    import torch
    from geo_simulator_b200 import _native as N

    box = (1000.0, 1000.0, 600.0)
    xyz, conn = orc.generate_cube(5, 4, 3, *box)
    mask, vals = orc.thermal_bc(xyz, box[2])
    dm = geo.DofManager(xyz.shape[0], 1)
    idx = np.nonzero(mask)[0]
    dm.set_dirichlet(idx, vals[idx])
    op = geo.ThermalOperator(geo.Mesh(xyz, conn), dm, np.full(conn.shape[0], 3.0))
    x = np.random.default_rng(11).standard_normal(xyz.shape[0])
    prec = N.PRECISION_MIXED if precision == "mixed" else N.PRECISION_FP64
    dx = torch.from_numpy(x).cuda()
    for host, call in ((op.apply(x, precision), lambda a, b: N.lib().geo_op_apply(op.h, a, b, prec)),
                       (op.lift_rhs(x), lambda a, b: N.lib().geo_op_lift_rhs(op.h, a, b))):
        out = torch.zeros(8 * x.size + 16, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert call(dx.data_ptr(), out.data_ptr() + offset) == 0
        got = out.cpu().numpy()
        assert np.array_equal(got[offset:offset + 8 * x.size].view(np.uint8), host.view(np.uint8))
        assert not got[:offset].any() and not got[offset + 8 * x.size:].any()
