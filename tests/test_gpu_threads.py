"""Contexts on several threads whose first calls come at the same time (what a device can do is found out once per process)."""
import os
import subprocess
import sys

import pytest

import helpers

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes as C, sys, threading
sys.path.insert(0, %r)
import numpy as np
from helpers import Native, load_package
N = load_package().native
rng = np.random.default_rng(0)
x, w = rng.standard_normal((300, 256)).astype(np.float32), rng.standard_normal((512, 256)).astype(np.float16)
k = rng.standard_normal((600, 2, 64)).astype(np.float16)
q = rng.standard_normal((500, 8, 64)).astype(np.float32)
nats = [Native(N.lib()) for _ in range(8)]
start, results = threading.Barrier(len(nats)), [None] * len(nats)

def work(i, nat):
    out, att = nat.buf(300 * 512 * 4), nat.buf(q.nbytes)
    kv = nat.kv_dense(600, 1, 2, 64)
    nat.kv_fill(kv, 0, k, k)
    call = N.Linear(nat.buf(x).ptr, nat.buf(w).ptr, None, out.ptr, None, None, N.Norm(), N.Norm(), 300, 256, 512, 0, N.DT_F16, 0, 0, 0.0)
    rows = N.StepRows(rows=500, segments=1, max_segment_rows=500, max_len=600, slot_mul=1, slot_add=0, seg=nat.buf(np.array([0, 500, 0, 100], np.uint32)).ptr)
    qd = nat.buf(q)
    start.wait()
    codes = [nat.lib.m40llm_linear_async(nat.ctx, C.byref(call), 1), nat.lib.m40llm_attention_step_rows_async(nat.ctx, kv, qd.ptr, 8, C.byref(rows), att.ptr)]
    nat.sync(1)
    results[i] = codes, out.download(np.float32, (300, 512)), att.download(np.float32, q.shape)

threads = [threading.Thread(target=work, args=a) for a in enumerate(nats)]
[t.start() for t in threads]
[t.join() for t in threads]
for r in results:
    assert r is not None and r[0] == [0, 0], r and r[0]
    assert np.array_equal(r[1], results[0][1]) and np.array_equal(r[2], results[0][2])
assert np.abs(results[0][1] - x.astype(np.float64) @ w.astype(np.float64).T).max() < 1e-4 * 16
print("same")
"""


def test_first_calls_from_several_threads():
    run = subprocess.run([sys.executable, "-c", PROGRAM % os.path.join(helpers.ROOT, "tests")], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip().endswith("same"), run.stdout + run.stderr
