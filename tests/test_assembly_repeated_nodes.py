"""CSR assembly of meshes with elements that list a node twice (an edge collapsed onto its
end, two midpoints in one): both contributions reach the entry that the two columns share,
with and without a row of more than 256 entries. Structure bit for bit, values against the
oracle's triplet merge at 1e-12 of the row scale."""
import numpy as np
import pytest

from test_assembly_rows import fan
from test_golden import row_err

pytestmark = pytest.mark.gpu

# element and the (local node, local node it repeats) pairs
REPEATS = {"vertex": {5: [(4, 0)]}, "midpoint": {7: [(6, 5)]}, "two": {3: [(4, 0), (8, 1)], 9: [(9, 3)]}}


@pytest.mark.parametrize("mesh", ["3x2x2", "fan12", "fan29"])  # fan29: a row of more than 256 entries
@pytest.mark.parametrize("kind", sorted(REPEATS))
def test_contributions_add_up(orc, geo, mesh, kind):
    if mesh.startswith("fan"):
        xyz, conn = fan(int(mesh[3:]), np.random.default_rng(11))
    else:
        xyz, conn = orc.generate_cube(*map(int, mesh.split("x")), 1.0, 1.2, 0.8)
    conn = np.array(conn)
    for e, pairs in REPEATS[kind].items():
        for a, b in pairs:
            conn[e, a] = conn[e, b]
    used = np.unique(conn)  # no node without an element
    new = np.full(xyz.shape[0], -1)
    new[used] = np.arange(used.size)
    xyz, conn = xyz[used], new[conn]
    coef = np.random.default_rng(2).uniform(0.5, 4.0, conn.shape[0])
    m = geo.Mesh(xyz, conn)
    for dpn in (1, 3):
        dm = geo.DofManager(xyz.shape[0], dpn)
        if dpn == 1:
            K = geo.Assembler.assemble_thermal_stiffness_parallel(m, dm, coef)
            Ko = orc.assemble_thermal_stiffness(xyz, conn, k_e=coef)
        else:
            K = geo.Assembler.assemble_elasticity_stiffness_parallel(m, dm, geo.IsotropicElasticity(1.0, 0.25), coef)
            Ko = orc.assemble_elasticity_stiffness(xyz, conn, E_e=coef, nu=0.25)
        ip, ix, data = K.to_host()
        assert np.array_equal(ip, Ko.indptr) and np.array_equal(ix.astype(np.int64), Ko.indices), dpn
        assert row_err(data, Ko.data, ip) <= 1e-12, dpn
