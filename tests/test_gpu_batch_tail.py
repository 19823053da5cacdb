"""Batches whose blocked kernel is followed by the per-step kernel: step counts
that are no multiple of the depth, in one call and over several, through the
graph and the step that aligns it, with work counters at zero and as other
kernels have left them.

Strips against tiles of the same depth bit for bit (the same operations per
cell, the same split of the steps over the kernels); a batch tuned in the
process against the FP64 oracle within 1e-5, the bound of the other FP32
Cahn-Hilliard tests, after few enough steps that each moves the state by more.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 32), (64, 64), (130, 512), (77, 224)]
# (kernel that runs before, its steps), then the calls
RUNS = [((None, 0), [n]) for n in (1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 101, 131, 333)] + \
       [((None, 0), [5, 5]), ((None, 0), [4, 1, 8, 3, 12, 2]), ((None, 0), [5, 130, 7, 131, 1, 133])] + \
       [((k, n), [m, 6]) for k in ("0,0", "4,0") for n in (1, 2, 12) for m in (5, 6, 7, 9, 131)]

CHILD = """
import json, os, sys
import numpy as np
sys.path[:0] = [%r, %r]
import test_gpu_batch_tail as t
from mmsp_gb300 import native as gpu
from mmsp_gb300 import inputs

form = os.environ.get("MMSP_GPU_BATCH_TILE")
descs = [gpu.make_desc(s, 1, np.float32, "ch", kappa=0.8, dt=0.004) for s in t.SHAPES]
x = [inputs.noisy_composition(s, 0.45, 0.03, 9 + s[0]).astype(np.float32) for s in t.SHAPES]
out = {}
for k, ((before, n), calls) in enumerate(t.RUNS):
    with gpu.Batch(descs) as b:
        b.upload_all(x)
        if before:
            os.environ["MMSP_GPU_BATCH_TILE"] = before
            b.tune()
            b.step(n)
            del os.environ["MMSP_GPU_BATCH_TILE"]
            if form:
                os.environ["MMSP_GPU_BATCH_TILE"] = form
        b.tune()
        for m in calls:
            b.step(m)
        rows = b.info().tile_rows
        for i, v in enumerate(b.download_all()):
            out["%%d_%%d" %% (k, i)] = v
print(rows)
np.savez(sys.argv[1], **out)
"""


def run_child(out, env):
    here = os.path.dirname(os.path.abspath(__file__))
    base = {k: v for k, v in os.environ.items() if not k.startswith(("MMSP_GPU_BATCH", "MMSP_GPU_TUNE"))}
    r = subprocess.run([sys.executable, "-c", CHILD % (os.path.dirname(here), here), str(out)], env={**base, **env},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    with np.load(out) as f:
        return int(r.stdout), {k: f[k] for k in f.files}


def test_strips_and_single_steps_in_any_order(gpu, tmp_path):
    cache = tmp_path / "tune.json"
    run_child(tmp_path / "tuned.npz", {"MMSP_GPU_TUNE_CACHE": str(cache)})
    (key,) = json.loads(cache.read_text())
    cache.write_text('{\n  "%s": [16, 128, 4, 11]\n}\n' % key)       # strips of 72 rows
    rows, got = run_child(tmp_path / "strips.npz", {"MMSP_GPU_TUNE_CACHE": str(cache)})
    assert rows == 72 + 16
    rows, want = run_child(tmp_path / "tiles.npz", {"MMSP_GPU_BATCH_TILE": "4,0"})
    assert rows == 64
    wrong = sorted({int(k.split("_")[0]) for k in want if not np.array_equal(got[k], want[k])})
    assert not wrong, [RUNS[k] for k in wrong]


@pytest.mark.parametrize("steps", [[5], [6], [7], [5, 5], [9, 3]], ids=str)
def test_single_steps_after_tuning_in_the_process(gpu, oracle, monkeypatch, steps):
    from mmsp_gb300 import inputs

    monkeypatch.delenv("MMSP_GPU_TUNE_CACHE", raising=False)
    monkeypatch.delenv("MMSP_GPU_BATCH_TILE", raising=False)
    work = inputs.batched_cahn_hilliard(count=48, seed=11)
    with gpu.Batch([gpu.make_desc(c0.shape, 1, np.float32, "ch", kappa=k, dt=0.005) for c0, k in work]) as b:
        b.upload_all([c0.astype(np.float32) for c0, _ in work])
        b.tune(force=True)
        for n in steps:
            b.step(n)
        got = b.download_all()
    for (c0, k), v in zip(work, got):
        x = c0.astype(np.float32).astype(np.float64)
        want, before = [oracle.ch_baseline(x, n, k, 1.0, 0.005) for n in (sum(steps), sum(steps) - 1)]
        assert np.abs(v - want).max() <= 1e-5 < np.abs(want - before).max()
