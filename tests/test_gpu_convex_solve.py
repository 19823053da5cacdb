"""The one-launch convex-splitting solve (pf_convex.cu) at the ends of its
ranges: axes of two cells (both neighbours are the same cell), a block of one
warp, shares of a color that fill two rounds of a block, non-unit spacing.

Iterations within one residual period (5) of the oracle's and values within
1e-10, the bounds of the model's other tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((2,), None, 3), ((2, 2), None, 3), ((2, 2, 2), None, 2), ((6, 2, 4), None, 3), ((20, 14), [1.0, 1.1], 3),
         ((10, 6, 8), [1.1, 1.0, 1.05], 2), ((640, 250), None, 1)]


@pytest.mark.parametrize("shape,dx,steps", CASES, ids=["x".join(map(str, s)) for s, _, _ in CASES])
def test_convex_solve_sizes(gpu, oracle, shape, dx, steps):
    from mmsp_gb300 import inputs

    x = inputs.convex_start(shape, 17)
    want, iters = oracle.ch_convex(x, steps, dx=dx, return_iters=True)
    d = gpu.make_desc(shape, 2, np.float64, "ch_convex", dx=dx)
    with gpu.Stepper(d) as s:
        s.upload(x)
        s.step(steps)
        got = s.download()
        st = s.reduce()
    assert abs(st.solver_iterations - iters) <= 5
    assert np.abs(got - want).max() <= 1e-10 * max(1.0, np.abs(want).max())
