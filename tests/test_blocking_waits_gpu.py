"""A process that asks CUDA for blocking waits has the defect solve's wait block
too: the Krylov iteration's running norm, which the host reads after every
iteration, is not spun for.  The host's work is some 30 us of 400 per iteration at
401 x 401; a spinning wait takes all of it."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CHILD = """
import ctypes, json, sys, time
sys.path[:0] = [%r, %r, %r]
cuda = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cuda.cuInit(0) == 0 and cuda.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cuda.cuDevicePrimaryCtxSetFlags_v2(dev, ctypes.c_uint(4)) == 0   # CU_CTX_SCHED_BLOCKING_SYNC
import numpy as np
import mdz
from test_multigrid_odd_gpu import _case
g, f = _case(401, 401)
rng = np.random.default_rng(3)
F = [rng.standard_normal(g.size(c)) * (t == -1) for c, t in ((-1, g.BCu), (-2, g.BCv))]
Fp = rng.standard_normal(g.size(1))
ctx = mdz.Context(g, 1, 1)
for _ in range(2):
    w, c = time.perf_counter(), time.process_time()
    its = ctx.SolveStokesDefect(f, 0, 64, 1e-10, 3000, F[0], F[1], Fp - Fp.mean())[3]
    w, c = time.perf_counter() - w, time.process_time() - c
ctx.close()
print(json.dumps([w, c, its]))
"""


def test_blocking_wait():
    root = os.path.dirname(HERE)
    r = subprocess.run([sys.executable, "-c", CHILD % (os.path.join(root, "mdoodz6.0_gb300"), os.path.join(root, "oracle"), HERE)],
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    wall, cpu, its = json.loads(r.stdout.strip().splitlines()[-1])
    assert its > 40 and cpu < 0.5 * wall, (wall, cpu, its)
