"""Work pending on the default stream (a program's own kernels) does not get in the way of an
operator or a matrix made meanwhile: what their set-up writes is in place before their first
use, and a matrix made from device memory holds what that work leaves there."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def busy(torch, ms):
    """Queues about ms milliseconds on the default stream; returns the last result."""
    a = torch.full((4096, 4096), 1.0 / 4096, device="cuda")
    b = a
    for _ in range(max(1, int(ms / 2))):  # 2 ms each in FP32
        b = b @ a
    return b


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dpn", [1, 3])
def test_operator_made_and_used(orc, geo, dpn, precision):
    import torch
    shape = (9, 8, 7)
    xyz, conn = orc.generate_cube(*shape, 1000.0, 1000.0, 600.0)
    mask, vals = orc.thermal_bc(xyz, 600.0)
    dm = geo.DofManager(xyz.shape[0], dpn)
    idx = np.nonzero(np.repeat(mask, dpn))[0]
    dm.set_dirichlet(idx, np.repeat(vals, dpn)[idx])
    mesh = geo.Mesh(xyz, conn)
    f = np.random.default_rng(1).standard_normal(dpn * xyz.shape[0])
    solver = geo.ConjugateGradient().with_tolerance(1e-9).with_max_iterations(5000).with_precision(precision)

    def make_and_solve():
        op = (geo.ThermalOperator(mesh, dm, 3.0) if dpn == 1 else
              geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1.0, 0.25)))
        return op.forward(f, solver)

    quiet, st = make_and_solve()
    assert st.converged
    torch.cuda.synchronize()
    for _ in range(3):
        pending = busy(torch, 60)
        u, st2 = make_and_solve()
        assert st2.converged
        assert np.linalg.norm(u - quiet) <= 1e-6 * np.linalg.norm(quiet)
        del pending
    torch.cuda.synchronize()


def test_matrix_from_pending_device_data(geo):
    import torch
    from geo_simulator_b200 import _native as N
    n = 1000
    ip, ix = np.arange(n + 1), np.arange(n, dtype=np.int32)
    torch.cuda.synchronize()
    late = busy(torch, 60)
    data = late.flatten()[:n].double() + 1.0  # 1 + 1/4096 to FP32 rounding, when it is there
    h = ctypes.c_void_p()
    ctx = geo.Context.default()
    assert N.lib().geo_csr_create(ctx.h, n, n, n, ip.ctypes.data, ix.ctypes.data, data.data_ptr(), ctypes.byref(h)) == 0
    A = geo.CsrMatrix(h, ctx)
    b = np.ones(n)
    x, _ = geo.ConjugateGradient().solve(A, b)
    assert np.array_equal(A.to_host()[2], data.cpu().numpy())
    assert np.linalg.norm(A.to_host()[2] * x - b) <= 1e-8 * np.sqrt(n)
