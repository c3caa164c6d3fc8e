"""A program that asks for blocking waits (cudaDeviceScheduleBlockingSync)
keeps its cores during a stage: 30 stages of about 0.6 ms use less than half
of their wall time on the CPU (a polling wait uses all of it), and return the
polling program's bits."""
import json
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r'''
import ctypes, json, sys, time
cu = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuDevicePrimaryCtxSetFlags(dev, int(sys.argv[2])) == 0
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/oracle"]
import numpy as np
import greenstein2002_gb300 as G
import oracle as O
n = 12500
s = O.rest_set(n, "base", 5489)
s["frus"][:, 1:] = 10 ** np.random.default_rng(5).uniform(-4.0, -2.0, (n, 4))
cell = G.Cell(n)
cell.upload(s)
cell.save()
d0, df = [5.0, 3e-4, 0.5], [5.4, 3e-4, 0.49]
cell.flux(d0)
for warm in (True, False):
    wall, cpu = time.perf_counter(), time.thread_time()
    for i in range(30):
        cell.resume()
        out, num = cell.stage(0.0, 0.05, d0, df)
    wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
print(json.dumps({"wall": wall, "cpu": cpu, "sums": [x.hex() for x in num.tolist() + out.tolist()]}))
'''


def _run(flags):
    out = subprocess.run([sys.executable, "-c", PROGRAM, ROOT, str(flags)], capture_output=True, text=True, timeout=300,
                         check=True).stdout
    return json.loads(out.splitlines()[-1])


def test_blocking_waits_keep_the_core(gw):
    polling, blocking = _run(0), _run(4)  # CU_CTX_SCHED_AUTO, CU_CTX_SCHED_BLOCKING_SYNC
    print(polling["wall"], polling["cpu"], blocking["wall"], blocking["cpu"])
    assert blocking["cpu"] < 0.5 * blocking["wall"]
    assert blocking["sums"] == polling["sums"]
