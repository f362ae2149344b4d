"""Several threads, each with a context of its own, make operators of different sizes, solve in
both precisions, assemble, and destroy, all at the same time: the results are those of one
thread alone. In a child process, so that a crash is this test's failure."""
import subprocess
import sys

import pytest

from conftest import ROOT

CHILD = """
import sys, threading
import numpy as np
sys.path.insert(0, sys.argv[1])
from oracle import oracle as orc
import geo_simulator_b200 as geo

SHAPES = [(1, (6, 5, 4)), (3, (4, 3, 3)), (1, (17, 13, 9))]
MESHES = {}
for _, shape in SHAPES:
    xyz, conn = orc.generate_cube(*shape, 1000.0, 1000.0, 600.0)
    MESHES[shape] = (xyz, conn) + orc.thermal_bc(xyz, 600.0)

def job(seed, ctx):
    rng, out = np.random.default_rng(seed), []
    for dpn, shape in SHAPES * 3:
        xyz, conn, mask, vals = MESHES[shape]
        dm = geo.DofManager(xyz.shape[0], dpn)
        idx = np.nonzero(np.repeat(mask, dpn))[0]
        dm.set_dirichlet(idx, np.repeat(vals, dpn)[idx])
        mesh, coef = geo.Mesh(xyz, conn), rng.uniform(1.0, 4.0, conn.shape[0])
        mat = geo.IsotropicElasticity(1.0, 0.25)
        if dpn == 1:
            op = geo.ThermalOperator(mesh, dm, coef, ctx=ctx)
            K = geo.Assembler.assemble_thermal_stiffness_parallel(mesh, dm, coef, ctx)
        else:
            op = geo.ElasticityOperator(mesh, dm, mat, coef, ctx=ctx)
            K = geo.Assembler.assemble_elasticity_stiffness_parallel(mesh, dm, mat, coef, ctx)
        f = rng.standard_normal(dpn * xyz.shape[0])
        cg = lambda p: geo.ConjugateGradient().with_tolerance(1e-10).with_max_iterations(5000).with_precision(p)
        out += [op.forward(f, cg(p))[0] for p in ("mixed", "fp64", "mixed")]
        Kb, fb = geo.Assembler.apply_dirichlet_bcs(K, f, dm, ctx)
        out += [op.apply(f), Kb.to_host()[2], cg("fp64").solve(Kb, fb)[0]]
        if f.size < 2500:
            out.append(geo.DirectSolver().solve(Kb, fb)[0])
    return out

n = 4
ctxs = [geo.Context() for _ in range(n)]
alone = [job(s, ctxs[s]) for s in range(n)]
for _ in range(6):
    got, errors = [None] * n, []
    def run(s):
        try:
            got[s] = job(s, ctxs[s])
        except Exception as e:
            errors.append(repr(e))
    threads = [threading.Thread(target=run, args=(s,)) for s in range(n)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
    for a, b in zip(alone, got):
        for x, y in zip(a, b):
            # the patch layout may differ from one operator to the next: rounding, within the tolerance
            assert np.linalg.norm(x - y) <= 1e-7 * np.linalg.norm(x)
print("as alone")
"""


@pytest.mark.gpu
def test_threads_with_contexts_of_their_own():
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "as alone" in r.stdout, (r.returncode, r.stdout[-2000:], r.stderr[-2000:])
