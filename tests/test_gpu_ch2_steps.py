"""The many-steps launch of small 2D FP64 Cahn-Hilliard grids (ch64_steps in
pf_ch64.cu) where its tiles and buffers can go wrong: tiles of one, two and
more cells a side (no inner part, a rim that is the whole tile), grids smaller
than a tile's halo (several wraps), ragged last tiles, the largest grid it
takes and the first it does not, odd and even step counts, calls longer than
one launch, a second call from the other buffer.

The reference's order bit for bit against the oracle; the contracted form and
the pow(x,3) model within 1e-12 relative, the bound of their other tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((1, 1), 3), ((1, 40), 5), ((2, 3), 4), ((3, 5), 7), ((5, 1), 2), ((7, 300), 3), ((31, 29), 513), ((64, 64), 257),
         ((153, 153), 4), ((90, 457), 3), ((640, 640), 3), ((641, 640), 2)]


@pytest.mark.parametrize("form", ["exact", "contract", "poly"])
@pytest.mark.parametrize("shape,steps", CASES, ids=["%s-%d" % ("x".join(map(str, s)), n) for s, n in CASES])
def test_many_steps_launch_against_oracle(gpu, oracle, shape, steps, form):
    from mmsp_gb300 import inputs

    dx = [1.0, 1.1] if steps % 2 else None
    if form == "poly":
        x = inputs.noisy_composition(shape, 0.0, 0.5, 70 + shape[1])
        d = gpu.make_desc(shape, 1, np.float64, "ch_poly", r=1.0, u=1.0, kappa=1.0, mobility=1.0, dt=0.004, dx=dx)
        want = oracle.ch_shipped(x, steps, 1.0, 1.0, 1.0, 1.0, 0.004, dx=dx)
    else:
        kappa = 1.0 if shape[0] % 2 else 0.8
        x = inputs.noisy_composition(shape, 0.45, 0.05, 71 + shape[1])
        d = gpu.make_desc(shape, 1, np.float64, "ch", kappa=kappa, mobility=1.1, dt=0.004, dx=dx, contract=form == "contract")
        want = oracle.ch_baseline(x, steps, kappa, 1.1, 0.004, dx=dx)
    with gpu.Stepper(d) as s:
        s.upload(x)
        s.step(steps)
        got = s.download()
        s.upload(x)
        s.step(1)
        if steps > 1:
            s.step(steps - 1)
        again = s.download()
    assert np.array_equal(got, again)
    if form == "exact":
        assert np.array_equal(got, want)
    else:
        assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(want).max())
