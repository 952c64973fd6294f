"""GPU: launches that are the first CUDA call of their thread, and first launches of a process from several threads at once.  The driver's tensor-map encoder
needs the device's context on the calling thread, and is looked up once for all threads; run in a process of its own, where nothing has happened yet."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu
CODE = r"""
import sys, threading
import numpy as np, torch
from fovi_b200 import ops
rs = np.random.RandomState(0)
n_in, n_out, K, V, threads = 40, 30, 9, 9, 24
idx = rs.randint(0, n_in, (K, n_out)).astype(np.int32)
plan = ops.KnnConvPlan(idx, rs.randint(0, V, (n_out, K)).astype(np.uint16), n_in, V, 64, 64)
wt = plan.pack_weights(torch.randn(64, 64 * V, device="cuda"))
xs = [torch.randn(4, n_in, 64, device="cuda").to(torch.bfloat16) for _ in range(threads)]
outs = [torch.empty(4, n_out, 64, device="cuda", dtype=torch.float32) for _ in range(threads)]
errors = []
def run(i, gate=None):
    if gate: gate.wait()
    try:
        plan.forward(xs[i], wt, out=outs[i])
    except Exception as e:
        errors.append(str(e))
if sys.argv[1] == "after":                      # one thread after the other, the main thread first
    run(0)
    torch.cuda.synchronize()
    for i in range(1, 4):
        t = threading.Thread(target=run, args=(i,)); t.start(); t.join()
else:                                           # the process's first launches, all at once
    torch.cuda.synchronize()
    gate = threading.Barrier(threads)
    ts = [threading.Thread(target=run, args=(i, gate)) for i in range(threads)]
    [t.start() for t in ts]; [t.join() for t in ts]
assert not errors, errors
plan.check()
for x, y in list(zip(xs, outs))[:4]:
    assert torch.equal(plan.forward(x, wt, out_dtype=torch.float32), y)
"""


@pytest.mark.parametrize("order", ["after", "at once"])
def test_first_launches_of_threads(order):
    r = subprocess.run([sys.executable, "-c", CODE, order], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
