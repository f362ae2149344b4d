"""CSR assembly at the sizes where its row kernels can go wrong: blocks of rows that end
inside the mesh, rows of more than 32 and of more than 256 entries (no places kept: the
searching form), blocks beyond shared memory, Dirichlet rows of every kind. Structure bit
for bit, values against the oracle at 1e-12 of the row scale."""
import numpy as np
import pytest

from test_golden import row_err

pytestmark = pytest.mark.gpu


def fan(n, rng):
    """n tetrahedra around one common vertex, all other nodes their own: a row of
    1 + 9 n entries."""
    conn, xyz = [], [np.zeros(3)]
    for _ in range(n):
        v = [xyz[0]] + [rng.standard_normal(3) for _ in range(3)]
        if np.linalg.det(np.array(v[1:]) - v[0]) < 0:
            v[2], v[3] = v[3], v[2]
        pts = v[1:] + [(v[a] + v[b]) / 2 for a, b in ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))]
        conn.append([0] + list(range(len(xyz), len(xyz) + 9)))
        xyz += pts
    return np.array(xyz), np.array(conn)


MESHES = ["1x1x1", "2x1x1", "5x3x2", "8x7x5", "fan3", "fan28", "fan29", "fan102"]


@pytest.mark.parametrize("name", MESHES)
def test_assembly_and_dirichlet(orc, geo, name):
    rng = np.random.default_rng(11)
    if name.startswith("fan"):
        xyz, conn = fan(int(name[3:]), rng)
    else:
        xyz, conn = orc.generate_cube(*map(int, name.split("x")), 1.0, 1.2, 0.8)
        nv = np.unique(conn[:, :4]).size
        xyz = xyz.copy()
        xyz[nv:] += rng.uniform(-0.004, 0.004, (xyz.shape[0] - nv, 3))
    N, E = xyz.shape[0], conn.shape[0]
    mesh = geo.Mesh(xyz, conn)
    k_e, E_e = rng.uniform(0.5, 4.0, E), rng.uniform(0.5e11, 2e11, E)
    for dpn in (1, 3):
        n = dpn * N
        mask = (rng.random(n) < 0.2).astype(np.uint8)
        mask[: dpn] = 0  # the fan's common row stays free
        vals = rng.standard_normal(n)
        dm = geo.DofManager(N, dpn)
        idx = np.nonzero(mask)[0]
        dm.set_dirichlet(idx, vals[idx])
        if dpn == 1:
            K = geo.Assembler.assemble_thermal_stiffness_parallel(mesh, dm, k_e)
            Ko = orc.assemble_thermal_stiffness(xyz, conn, k_e=k_e)
        else:
            K = geo.Assembler.assemble_elasticity_stiffness_parallel(mesh, dm, geo.IsotropicElasticity(1e11, 0.25), E_e)
            Ko = orc.assemble_elasticity_stiffness(xyz, conn, E_e=E_e, nu=0.25)
        f = rng.standard_normal(n)
        Kb, fb = geo.Assembler.apply_dirichlet_bcs(K, f, dm)
        Kbo, fbo = orc.apply_dirichlet_bcs(Ko, f, mask, np.where(mask, vals, 0.0))
        for A, B in ((K, Ko), (Kb, Kbo)):
            ip, ix, data = A.to_host()
            assert np.array_equal(ip, B.indptr) and np.array_equal(ix.astype(np.int64), B.indices), dpn
            assert row_err(data, B.data, ip) <= 1e-12, dpn
        assert np.abs(fb - fbo).max() <= 1e-12 * np.abs(fbo).max(), dpn
