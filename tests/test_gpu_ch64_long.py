"""FP64 3D Cahn-Hilliard on grids of very many planes: the two passes, and with
them the contracted form, up to 16 * 65535 planes.

A grid that repeats along X evolves as its period does: the contracted form bit
for bit as on a short grid that takes the same kernels, the form with shared pair
sums (4 M cells and more) within 1e-12 relative, its bound of other tests.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,period,contract,same", [(131076, 12, True, True), (131076, 12, False, True),
                                                         (196680, 22, True, True), (400008, 24, True, False),
                                                         (1048536, 24, True, False)])
def test_many_planes(gpu, oracle, planes, period, contract, same):
    from mmsp_gb300 import inputs

    assert planes % period == 0
    x = inputs.noisy_composition((period, 2, 8), 0.45, 0.1, 7)
    p = dict(kappa=1.0, mobility=1.0, dt=0.004, contract=contract)

    def run(shape, v):
        with gpu.Stepper(gpu.make_desc(shape, 1, np.float64, "ch", **p)) as s:
            s.upload(v)
            s.step(5)
            return s.download()

    got = run((planes, 2, 8), np.tile(x, (planes // period, 1, 1))).reshape(planes // period, period, 2, 8)
    want = run((period, 2, 8), x)
    exact = oracle.ch_baseline(x, 5, 1.0, 1.0, 0.004)
    assert np.abs(want - exact).max() <= 1e-12 * np.abs(exact).max()
    assert np.array_equal(want, exact) == (not contract)      # or the forms cannot be told apart
    if same:
        assert (got == want).all()
    else:
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
