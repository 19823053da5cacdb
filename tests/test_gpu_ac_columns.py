"""The column kernels of the Allen-Cahn models (pf_ac_cols.cu) at the sizes
where their rules and index arithmetic change: 4, 2 and 1 cells per thread
(row length against field count), more than 16 fields, last partial blocks,
rows, planes and axes of one or two cells, the step direction and the plane
runs of states above the L2 bound, 32-thread blocks and 128-thread blocks of
the FP64 form, gradient coefficients of 1, 2 and any other value.

FP32 against the FP64 oracle within 1e-5 (the precision form's bound); FP64
bit for bit where the oracle has no pow(x,3), else within 1e-12 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL_SHIPPED = 1e-12
TOL_F32 = 1e-5

CASES = [((1, 7, 4), 7, "ac", 2.0), ((3, 1, 8), 8, "ac", 1.0), ((5, 6, 2), 16, "gg", 2.0), ((2, 3, 1), 3, "ac", 0.7),
         ((4, 9, 33), 17, "ac", 2.0), ((3, 5, 36), 32, "gg", 2.0), ((2, 40, 100), 1, "ac_poly", 1.0),
         ((3, 21, 50), 1, "ac_poly", 0.6), ((37, 64), 7, "ac", 2.0), ((9, 130), 8, "zener", 2.0), ((300,), 5, "gg", 2.0),
         ((2, 1), 4, "ac", 2.0), ((6, 43, 128), 6, "zener", 2.0), ((16, 80, 111), 2, "ac", 0.7),
         ((20, 65, 128), 4, "ac", 1.0)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,fields,model,kappa", CASES,
                         ids=["%s-%d-%s" % ("x".join(map(str, s)), f, m) for s, f, m, _ in CASES])
def test_column_kernels_against_oracle(gpu, oracle, shape, fields, model, kappa, dtype):
    from mmsp_gb300 import inputs

    steps = 12
    dx = [1.0, 1.1, 0.9][: len(shape)] if fields % 2 else None
    if model == "ac_poly":
        x = inputs.noisy_composition(shape, 0.0, 0.8, 40 + shape[0])
        d = gpu.make_desc(shape, 1, dtype, model, r=1.0, u=1.0, kappa=kappa, mobility=1.0, dt=0.01, dx=dx)
        want = oracle.ac_scalar_shipped(x, steps, 1.0, 1.0, kappa, 1.0, 0.01, dx=dx)
    else:
        x = inputs.voronoi_grains(shape, 7, fields, 41 + shape[0]) * 0.8 + 0.05
        if model == "ac":
            d = gpu.make_desc(shape, fields, dtype, model, gamma=1.5, kappa=kappa, mobility=1.0, dt=0.02, dx=dx)
            want = oracle.ac_baseline(x, steps, 1.5, kappa, 1.0, 0.02, dx=dx)
        else:
            d = gpu.make_desc(shape, fields, dtype, model, dt=0.01, dx=dx)
            want = (oracle.ac_graingrowth if model == "gg" else oracle.ac_zener)(x, steps, 0.01, dx=dx)
    with gpu.Stepper(d) as s:
        s.upload(x.astype(dtype))
        s.step(steps)
        got = s.download().astype(np.float64)
    if dtype == np.float32:
        assert np.abs(got - want).max() <= TOL_F32
    elif model == "ac":
        assert np.array_equal(got, want)
    else:
        assert np.abs(got - want).max() <= TOL_SHIPPED * max(1.0, np.abs(want).max())


# two states above 96 MB: plane runs of 3 (up to 8 fields) and 2, with a last
# run that is shorter, stepping in both directions
@pytest.mark.parametrize("shape,fields", [((64, 128, 200), 8), ((51, 130, 125), 16)])
def test_column_kernel_above_l2(gpu, oracle, shape, fields):
    from mmsp_gb300 import inputs

    x = inputs.voronoi_grains(shape, 5, fields, 77) * 0.8 + 0.05
    d = gpu.make_desc(shape, fields, np.float32, "ac", gamma=1.5, kappa=2.0, mobility=1.0, dt=0.05)
    with gpu.Stepper(d) as s:
        s.upload(x.astype(np.float32))
        s.step(3)
        got = s.download().astype(np.float64)
    assert np.abs(got - oracle.ac_baseline(x, 3, 1.5, 2.0, 1.0, 0.05)).max() <= TOL_F32


# the form that prefetches a plane ahead: odd rows, 5 to 9 fields, above 96 MB;
# fewer planes than a run, a run and one plane, several runs
@pytest.mark.parametrize("shape,fields,model", [((2, 2521, 501), 5, "ac"), ((4, 1181, 333), 9, "gg"),
                                                ((19, 250, 333), 8, "zener")])
def test_prefetching_column_kernel(gpu, oracle, shape, fields, model):
    from mmsp_gb300 import inputs

    x = inputs.voronoi_grains(shape, 5, fields, 78) * 0.8 + 0.05
    if model == "ac":
        d = gpu.make_desc(shape, fields, np.float32, "ac", gamma=1.5, kappa=2.0, mobility=1.0, dt=0.05)
        want = oracle.ac_baseline(x, 3, 1.5, 2.0, 1.0, 0.05)
    else:
        d = gpu.make_desc(shape, fields, np.float32, model, dt=0.01)
        want = (oracle.ac_graingrowth if model == "gg" else oracle.ac_zener)(x, 3, 0.01)
    with gpu.Stepper(d) as s:
        s.upload(x.astype(np.float32))
        s.step(3)
        got = s.download().astype(np.float64)
    assert np.abs(got - want).max() <= TOL_F32
