"""A process that destroys its objects and contexts, resets the device and starts again finds
everything working as the first time. In a child process: the reset ends its CUDA context."""
import subprocess
import sys

import pytest

from conftest import ROOT

CHILD = """
import ctypes, gc, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from oracle import oracle as orc
import geo_simulator_b200 as geo
from geo_simulator_b200 import _native as N

def run():
    xyz, conn = orc.generate_cube(9, 8, 7, 1000.0, 1000.0, 600.0)
    mesh = geo.Mesh(xyz, conn)
    out = []
    for dpn in (1, 3):
        dm = geo.DofManager(xyz.shape[0], dpn)
        op = (geo.ThermalOperator(mesh, dm, 3.0) if dpn == 1 else
              geo.ElasticityOperator(mesh, dm, geo.IsotropicElasticity(1e11, 0.25)))
        x = np.random.default_rng(0).standard_normal(dpn * xyz.shape[0])
        few = geo.ConjugateGradient().with_tolerance(0.0).with_max_iterations(20)
        out += [op.apply(x, "fp64"), op.apply(x, "mixed"), op.solve(x, few)[0]]
    return out

first = run()
gc.collect()
geo.Context._default.clear()
gc.collect()
live, cached, mallocs = (ctypes.c_int64() for _ in range(3))
N.lib().geo_device_memory_stats(ctypes.byref(live), ctypes.byref(cached), ctypes.byref(mallocs))
assert live.value == 0 and cached.value == 0
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
for a, b in zip(first, run()):
    assert np.array_equal(a, b)
print("ran again")
"""


@pytest.mark.gpu
def test_reset_and_again():
    import os

    import nvidia.cuda_runtime
    libs = [os.path.join(p, "lib") for p in nvidia.cuda_runtime.__path__] + ["/usr/local/cuda/lib64"]
    env = dict(os.environ, LD_LIBRARY_PATH=":".join(libs + [os.environ.get("LD_LIBRARY_PATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ran again" in r.stdout, r.stdout + r.stderr
