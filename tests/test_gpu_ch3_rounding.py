"""Rounding errors of the FP32 3D Cahn-Hilliard step on rows above 512 cells
(pf_ch3_flat.cu) against those of the reference's own expressions, every
operation rounded to FP32 (numpy).  The kernel's expressions are the same but
for fused products, so the RMS errors after 40 steps agree within sampling: 3%.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((11, 11, 513), "ch", None), ((2, 60, 700), "ch", None), ((20, 6, 1500), "ch", None), ((5, 70, 514), "ch", [1.1, 1.0, 1.2]),
         ((90, 90, 514), "ch", None), ((20, 6, 1501), "ch_poly", None), ((11, 11, 514), "ch_poly", [1.0, 1.1, 1.2])]


def reference(c, model, steps, dt, dx, T):
    c, two, one = c.astype(T), T(2), T(1)
    w = [T(1.0 / (h * h)) for h in (dx or [1.0, 1.0, 1.0])]

    def lap(f):
        out = np.zeros_like(f)
        for a in range(3):
            out = out + w[a] * ((np.roll(f, -1, a) - two * f) + np.roll(f, 1, a))
        return out

    for _ in range(steps):
        fp = two * c * (one - c) * (one - two * c) if model == "ch" else -c + c * c * c
        c = c + T(dt) * lap(fp - lap(c))
    return c


@pytest.mark.parametrize("shape,model,dx", CASES, ids=["%s-%s" % ("x".join(map(str, s)), m) for s, m, _ in CASES])
def test_error_against_the_reference_expressions(gpu, shape, model, dx):
    from mmsp_gb300 import inputs

    x = inputs.noisy_composition(shape, 0.425 if model == "ch" else 0.0, 0.025 if model == "ch" else 0.2, 3)
    x = x.astype(np.float32)
    p = {} if model == "ch" else dict(r=1.0, u=1.0)
    with gpu.Stepper(gpu.make_desc(shape, 1, np.float32, model, kappa=1.0, mobility=1.0, dt=0.01, dx=dx, **p)) as s:
        s.upload(x)
        s.step(40)
        got = s.download()
    want = reference(x, model, 40, 0.01, dx, np.float64)

    def rms(y):
        return np.sqrt(np.mean((y.astype(np.float64) - want) ** 2))

    assert rms(got) <= 1.03 * rms(reference(x, model, 40, 0.01, dx, np.float32))
