"""Rounding errors of the FP32 Allen-Cahn steps (pf_ac_cols.cu) against those of
the reference's own expressions, every operation rounded to FP32 (numpy): a
kernel that regroups terms or fuses operations must not lose accuracy by it.

The bound on the ratio of the relative RMS errors after 40 steps.  Differences
along each axis (1D, 2D, 3D rows above 256 cells, many fields on long rows): the
same roundings but for fused products and the order of additions, 1.15.  Sums of
neighbours (other 3D grids): those round at the size of several cells, and with
them a share of the error that grows with the Laplacian's coefficient: 1.5 for
kappa dt = 0.1, 1.25 for grain growth's 2 dt = 0.02.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((1000,), 3, "ac", 1.15), ((1000,), 3, "gg", 1.15), ((64, 64), 3, "ac", 1.15), ((64, 64), 3, "gg", 1.15),
         ((100, 99), 5, "gg", 1.15), ((130, 66), 6, "zener", 1.15), ((300, 37), 20, "gg", 1.15), ((256, 256), 1, "ac_poly", 1.15),
         ((12, 20, 300), 4, "ac", 1.15), ((12, 20, 257), 6, "gg", 1.15), ((8, 6, 200), 32, "ac", 1.15), ((80, 2, 96), 4, "ac", 1.15),
         ((20, 24, 28), 3, "ac", 1.5), ((20, 24, 28), 3, "gg", 1.25), ((32, 32, 32), 8, "gg", 1.25), ((18, 21, 27), 5, "zener", 1.25)]


def reference(x, model, steps, dt, T):
    """The examples' updates in type T, operation by operation."""
    x, two = x.astype(T), T(2)
    for _ in range(steps):
        lap = np.zeros_like(x)
        for a in range(x.ndim - 1):
            lap = lap + ((np.roll(x, -1, a) - two * x) + np.roll(x, 1, a))
        sq = np.zeros(x.shape[:-1], T)
        for f in range(x.shape[-1]):
            sq = sq + x[..., f] * x[..., f]
        sq = sq[..., None]
        if model == "ac":
            e = -x + x * x * x + T(3) * x * (sq - x * x) - two * lap
        elif model == "ac_poly":
            e = -x + x * x * x - lap
        else:
            e = -x - x * x * x + two * (x * sq - lap)
        new = x - T(dt) * e
        if model == "zener":
            new[..., 0] = x[..., 0]
        x = new
    return x


@pytest.mark.parametrize("shape,fields,model,bound", CASES,
                         ids=["%s-%d-%s" % ("x".join(map(str, s)), f, m) for s, f, m, _ in CASES])
def test_error_against_the_reference_expressions(gpu, shape, fields, model, bound):
    from mmsp_gb300 import inputs

    steps, dt = 40, 0.05 if model == "ac" else 0.01
    if fields > 1:
        x = inputs.voronoi_grains(shape, 60, fields, 90 + shape[0])
        d = gpu.make_desc(shape, fields, np.float32, model, dt=dt, **(dict(gamma=1.5, kappa=2.0) if model == "ac" else {}))
    else:
        x = inputs.noisy_composition(shape, 0.0, 0.8, 90)[..., None].astype(np.float32).astype(np.float64)
        d = gpu.make_desc(shape, 1, np.float32, model, dt=dt, r=1.0, u=1.0, kappa=1.0)
    with gpu.Stepper(d) as s:
        s.upload(x.astype(np.float32) if fields > 1 else x[..., 0].astype(np.float32))
        s.step(steps)
        got = s.download().astype(np.float64).reshape(x.shape)
    want = reference(x, model, steps, dt, np.float64)

    def rms(y):
        return np.sqrt(np.mean((y - want) ** 2))

    assert rms(got) <= bound * rms(reference(x, model, steps, dt, np.float32).astype(np.float64))
