"""The first call of the allocation-free entry leaves no kernel for later calls to load, whatever their size, query
lengths and scoring: in a fresh process a call of another size returns as fast the first time as later (loading its
kernels takes several times as long)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import statistics, sys, time
import torch
from bsbolt_gb300 import _lib, extend, synth
from test_zz_no_alloc import _buffers, _call
L, st = _lib.load(), torch.cuda.current_stream().cuda_stream
sets = [(a, *synth.ksw_jobs(n, seed=n, qmin=1, qmax=400)) for a, n in ((1, 64), (1, 12000), (16, 30000), (1, 100000), (1, 250000))]
sets = [(extend.make_param(synth.fill_scmat(a, 4), 6, 1, 6, 1, 100), len(j), len(s), _buffers(j, s)) for a, j, s in sets]
free = None
for k, (p, n, size, (dj, ds, do, dc)) in enumerate(sets):
    t = []
    for _ in range(8):
        t0 = time.perf_counter()
        _call(L, p, dj, n, ds, size, do, None, st)
        t.append((time.perf_counter() - t0) * 1e3)
        torch.cuda.synchronize()
    print(n, *("%.3f" % x for x in t))
    if k == 0:
        free = torch.cuda.mem_get_info()[0]
    else:
        assert t[0] < 2.5 * statistics.median(t[1:]) + 0.1, (n, t)
assert torch.cuda.mem_get_info()[0] == free
"""


def test_no_kernel_is_loaded_after_the_first_call():
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests")]))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
