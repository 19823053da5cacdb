"""The strip kernel of 2D FP32 Cahn-Hilliard (ch2_strip_kernel in pf_batch.cu)
where its windows and strips can go wrong: the fewest rows that it takes and
one less (the tile kernel's), rows of one cell, fewer than a group of four and
fewer than the halo, rows that are no multiple of four cells, strips that do
not divide the rows (the last one overlaps), windows over several strips and
several windows a strip, both models, spacings of one and other.

Single grids and batches against the tile kernel bit for bit where it takes
them (the same operations per cell), and against the FP64 oracle within 1e-5,
the bound of the other FP32 Cahn-Hilliard tests.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(23, 40), (24, 1), (24, 3), (25, 13), (29, 96), (31, 32), (60, 113), (64, 64), (101, 7), (113, 512), (157, 1030),
          (700, 511)]
BATCH = [((3, 32), "ch"), ((64, 64), "ch"), ((130, 512), "ch"), ((77, 224), "ch")]


def grid(shape, model):
    from mmsp_gb300 import inputs

    return inputs.noisy_composition(shape, 0.45 if model == "ch" else 0.0, 0.03, 40 + shape[0])


def desc(gpu, shape, model, dx=None):
    p = dict(kappa=0.8) if model == "ch" else dict(kappa=0.8, r=1.0, u=1.0)
    return gpu.make_desc(shape, 1, np.float32, model, mobility=1.0, dt=0.004, dx=dx, **p)


@pytest.mark.parametrize("dx", [None, [1.1, 0.9]], ids=["unit", "spaced"])
@pytest.mark.parametrize("model", ["ch", "ch_poly"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_strips_of_a_grid(gpu, oracle, monkeypatch, shape, model, dx):
    x = grid(shape, model)
    d = desc(gpu, shape, model, dx)
    with gpu.Stepper(d) as s:
        s.upload(x.astype(np.float32))
        s.step(24)
        got = s.download()
    want = (oracle.ch_baseline(x, 24, 0.8, 1.0, 0.004, dx=dx) if model == "ch"
            else oracle.ch_shipped(x, 24, 1.0, 1.0, 0.8, 1.0, 0.004, dx=dx))
    assert np.abs(got.astype(np.float64) - want).max() <= 1e-5
    if shape[1] % 32 == 0 and shape[1] <= 512:
        monkeypatch.setenv("MMSP_GPU_BATCH_TILE", "4,0")
        with gpu.Batch([d]) as b:
            b.upload(0, x.astype(np.float32))
            b.step(24)
            assert b.info().tile_rows == 64
            assert np.array_equal(b.download(0), got)


CHILD = """
import sys
import numpy as np
sys.path[:0] = [%r, %r]
import test_gpu_ch2_strips as t
from mmsp_gb300 import native as gpu
with gpu.Batch([t.desc(gpu, s, m) for s, m in t.BATCH]) as b:
    for i, (s, m) in enumerate(t.BATCH):
        b.upload(i, t.grid(s, m).astype(np.float32))
    b.step(152)      # graph replays, then launches
    info = b.info()
    print(info.tuned_from_cache, info.temporal_depth, info.tile_rows)
    np.savez(sys.argv[1], *[b.download(i) for i in range(len(t.BATCH))])
"""


def run_child(out, env):
    here = os.path.dirname(os.path.abspath(__file__))
    base = {k: v for k, v in os.environ.items() if not k.startswith("MMSP_GPU_BATCH")}
    r = subprocess.run([sys.executable, "-c", CHILD % (os.path.dirname(here), here), str(out)], env={**base, **env},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    with np.load(out) as f:
        return [int(v) for v in r.stdout.split()], [f[k] for k in f.files]


def test_strips_of_a_batch_from_a_saved_tuning(gpu, tmp_path):
    """Batches take the strips that a saved tuning names (shape 4 and up, depth
    4); an entry that names no kernel is tuned anew."""
    cache = tmp_path / "tune.json"
    _, tiles = run_child(tmp_path / "tiles.npz", {"MMSP_GPU_BATCH_TILE": "4,0"})
    run_child(tmp_path / "tuned.npz", {"MMSP_GPU_TUNE_CACHE": str(cache)})
    (key,) = json.loads(cache.read_text())
    for entry, rows in (([16, 128, 4, 4], 20), ([16, 128, 4, 11], 72 + 16), ([16, 128, 8, 11], None),
                        ([16, 128, 4, 99], None)):
        cache.write_text('{\n  "%s": %s\n}\n' % (key, json.dumps(entry)))
        (cached, depth, tile_rows), got = run_child(tmp_path / "strips.npz", {"MMSP_GPU_TUNE_CACHE": str(cache)})
        assert cached == (rows is not None)
        if rows is not None:
            assert (depth, tile_rows) == (4, rows)
            assert all(np.array_equal(a, b) for a, b in zip(got, tiles))
