"""The grid barriers of the cooperative launches (ch64_steps, cs_solve) when
their wait runs out, and the handle after it.

MMSP_GPU_TEST_STALL_LAUNCHES=1 makes the next such launch wait for a count that
never comes: every block gives up after 2 s, the host reports ETIMEDOUT once,
and the words are cleared on the handle's own stream, so that the next steps are
right however much work the program has queued on its default stream.  Run in a
child process so the variable does not reach other tests.
"""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys
import time
import numpy as np
import torch
sys.path.insert(0, %r)
from mmsp_gb300 import inputs, native
from oracle import pf_oracle
L = native.load()
model = sys.argv[1]
if model == "ch":
    x = inputs.noisy_composition((70, 90), 0.45, 0.05, 5)
    d, n = native.make_desc(x.shape, 1, np.float64, "ch", dt=0.004), 40
    want = pf_oracle.ch_baseline(x, n, 1.0, 1.0, 0.004)
else:
    x = inputs.convex_start((40, 24), 17)
    d, n = native.make_desc(x.shape[:2], 2, np.float64, "ch_convex"), 2
    want = pf_oracle.ch_convex(x, n)
torch.zeros(1, device="cuda")
with native.Stepper(d) as s:
    s.upload(x)
    s.step(1 if model == "ch_convex" else 7)    # the stalled launch
    time.sleep(2.5)                             # the waits are over, ...
    torch.cuda._sleep(2 * 10 ** 9)              # ... the default stream has about a second of work
    done = torch.cuda.Event()
    done.record()
    print("first", L.mmsp_gpu_synchronize(s.h), flush=True)
    s.upload(x)
    s.step(n)
    print("again", L.mmsp_gpu_synchronize(s.h), flush=True)
    print("busy", int(not done.query()), flush=True)
    print("err", float(np.abs(s.download() - want).max()), flush=True)
"""


@pytest.mark.parametrize("model,bound", [("ch", 0.0), ("ch_convex", 1e-10)])
def test_barrier_runs_out_and_the_handle_stays_usable(gpu, model, bound):
    env = dict(os.environ, MMSP_GPU_TEST_STALL_LAUNCHES="1")
    r = subprocess.run([sys.executable, "-c", CHILD % ROOT, model], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    lines = dict(line.split(None, 1) for line in r.stdout.splitlines() if line.strip())
    assert int(lines["first"]) == gpu.ETIMEDOUT
    assert int(lines["again"]) == gpu.OK
    assert float(lines["err"]) <= bound
    assert int(lines["busy"])                   # or it has shown nothing about the default stream
