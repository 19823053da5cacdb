"""The FP32 3D Cahn-Hilliard kernel on warp windows (pf_ch3_flat.cu) at the
sizes where its index arithmetic and rules change: strips of 2, 4 and 6 rows
with a last strip that overlaps the one before, rows of 4 and 5 cells (several
rows per window), odd rows (single-cell loads), windows that end at a row's
last cell, one and two planes, runs of planes that end short, states above the
L2 bound (prefetch), and the walk's two directions (every second step).

Against the FP64 oracle within 1e-5 (the precision form's bound).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-5

SMALL = [(1, 2, 4), (2, 3, 5), (5, 4, 6), (3, 5, 7), (9, 7, 56), (4, 6, 57), (6, 2, 61), (2, 9, 60), (17, 11, 31),
         (30, 60, 58), (70, 45, 47)]
LARGE = [(86, 207, 207), (90, 208, 206), (700, 6, 900), (51, 497, 505), (50, 505, 502)]


@pytest.mark.parametrize("model", ["ch", "ch_poly"])
@pytest.mark.parametrize("shape", SMALL + LARGE, ids=["x".join(map(str, s)) for s in SMALL + LARGE])
def test_windows_kernel_against_oracle(gpu, oracle, shape, model):
    from mmsp_gb300 import inputs

    steps = 21 if shape in SMALL else 3
    if model == "ch":
        c0 = inputs.noisy_composition(shape, 0.4, 0.05, 300 + shape[0])
        d = gpu.make_desc(shape, 1, np.float32, "ch", kappa=0.9, mobility=1.1, dt=0.002, dx=[1.0, 0.9, 1.1])
        want = oracle.ch_baseline(c0, steps, 0.9, 1.1, 0.002, dx=[1.0, 0.9, 1.1])
    else:
        c0 = inputs.noisy_composition(shape, 0.0, 0.5, 301 + shape[0])
        d = gpu.make_desc(shape, 1, np.float32, "ch_poly", r=1.0, u=1.0, kappa=1.0, mobility=1.0, dt=0.002)
        want = oracle.ch_shipped(c0, steps, 1.0, 1.0, 1.0, 1.0, 0.002)
    with gpu.Stepper(d) as s:
        s.upload(c0.astype(np.float32))
        s.step(steps)
        got = s.download().astype(np.float64)
    assert np.abs(got - want).max() <= TOL_F32
