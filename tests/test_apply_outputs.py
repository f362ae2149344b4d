"""Operator apply and lift write the caller's vector where it is: host memory, device memory,
and device memory that holds the input as well. The results are the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dpn,shape", [(1, (1, 1, 1)), (1, (9, 8, 7)), (3, (2, 1, 1)), (3, (7, 5, 3))])
def test_outputs(orc, geo, dpn, shape, precision):
    import torch
    from geo_simulator_b200 import _native as N

    box = (1000.0, 1000.0, 600.0)
    xyz, conn = orc.generate_cube(*shape, *box)
    mask, vals = orc.thermal_bc(xyz, box[2])
    dm = geo.DofManager(xyz.shape[0], dpn)
    idx = np.nonzero(np.repeat(mask, dpn))[0]
    dm.set_dirichlet(idx, np.repeat(vals, dpn)[idx])
    mesh = geo.Mesh(xyz, conn)
    if dpn == 1:
        op = geo.ThermalOperator(mesh, dm, np.full(conn.shape[0], 3.0))
    else:
        op = geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1e11, 0.25), np.full(conn.shape[0], 1e11))
    x = np.random.default_rng(11).standard_normal(dpn * xyz.shape[0])
    prec = N.PRECISION_MIXED if precision == "mixed" else N.PRECISION_FP64
    for host, call in ((op.apply(x, precision), lambda a, b: N.lib().geo_op_apply(op.h, a, b, prec)),
                       (op.lift_rhs(x), lambda a, b: N.lib().geo_op_lift_rhs(op.h, a, b))):
        dx = torch.from_numpy(x).cuda()
        dy = torch.full_like(dx, float("nan"))
        torch.cuda.synchronize()
        assert call(dx.data_ptr(), dy.data_ptr()) == 0
        assert np.array_equal(dy.cpu().numpy(), host)
        assert call(dx.data_ptr(), dx.data_ptr()) == 0
        assert np.array_equal(dx.cpu().numpy(), host)
        hy = np.full_like(x, np.nan)
        dx = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        assert call(dx.data_ptr(), hy.ctypes.data) == 0
        assert np.array_equal(hy, host)
