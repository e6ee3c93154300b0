"""A long Lanczos step is waited for as the caller set its device to wait:
with blocking waits the host core is free meanwhile."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, os, sys, time
cuda = ctypes.CDLL("libcuda.so.1")
assert cuda.cuInit(0) == 0
assert cuda.cuDevicePrimaryCtxSetFlags_v2(0, 4) == 0  # this process's own context: blocking waits
sys.path[:0] = [%r, os.path.join(%r, "tests", "golden")]
import models
import pyqcm_gb300 as pg
params = {"t": 1.0, "U": 8.0, "mu": 4.0}
ns, nb, ops = models.hubbard_cluster(4, 4)
m = pg.ClusterModel(ns, nb)
for name, (typ, els) in ops.items():
    if name in params:
        m.new_operator(name, typ, els)
H = pg.Hamiltonian(m, params, "R0:N12:S0")  # 64,128,064 states: more than a millisecond a step
assert H.fx_available()
def steps(n):
    try:
        H.lanczos(tol=1e-300, max_iter=n, reorth=0, want_psi=False)
    except pg.QcmgError as e:
        assert e.code == -4, e
steps(3)  # the seeded start vector, the tables
wall, cpu = time.perf_counter(), time.process_time()
steps(200)
print(time.process_time() - cpu, time.perf_counter() - wall)
"""


def test_blocking_waits_leave_the_core_free():
    out = subprocess.run([sys.executable, "-c", CHILD % (ROOT, ROOT)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    cpu, wall = map(float, out.stdout.split()[-2:])
    # 200 us of polling in a step of more than 1 ms, and the host's share of a
    # step (launches, the convergence test: tens of microseconds)
    assert cpu < 0.5 * wall, (cpu, wall)
