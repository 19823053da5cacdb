"""The stochastic FP32 3D Cahn-Hilliard kernels (pf_ch64.cu) around the size at
which their runs of planes get longer: the last grid below and grids from it on,
a last run that is short or a single plane.

Against the FP64 form with the same deviates within 1e-5, the bound of the FP32
form's other tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(99, 100, 101), (100, 100, 100), (103, 99, 101), (9, 340, 341), (65, 124, 125)],
                         ids=lambda s: "x".join(map(str, s)))
def test_runs_of_planes(gpu, shape):
    from mmsp_gb300 import inputs

    x = inputs.noisy_composition(shape, 0.0, 0.4, 21).astype(np.float32)
    got = {}
    for dtype in (np.float32, np.float64):
        with gpu.Stepper(gpu.make_desc(shape, 1, dtype, "ch_poly", r=1.0, u=1.0, kappa=1.0, mobility=1.0, dt=0.002,
                                       noise=0.05, seed=11)) as s:
            s.upload(x.astype(dtype))
            s.step(7)
            got[dtype] = s.download().astype(np.float64)
    assert np.abs(got[np.float32] - got[np.float64]).max() <= 1e-5
    assert np.abs(got[np.float64] - x).max() > 1e-2       # the steps and their noise move the state by much more
