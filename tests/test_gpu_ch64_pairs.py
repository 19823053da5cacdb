"""The contracted FP64 3D Cahn-Hilliard kernels that share pair sums
(ch64_mu_pairs, ch64_update_pairs in pf_ch64.cu) where their walk can go wrong:
the first size they take and one below, odd and even rows (the last strip
repeats one), rows that leave part of a warp idle, a last run of planes that is
short or single, two planes, both models, kappa of one and other.

Within 1e-12 relative of the oracle, the bound of the contracted form's other
tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((2, 1024, 2048), "ch", 1.0), ((2, 1023, 2050), "ch", 0.8), ((7, 1025, 600), "ch", 0.8),
         ((13, 300, 1090), "ch_poly", 1.0), ((163, 161, 161), "ch", 1.0), ((1500, 2, 1400), "ch_poly", 0.7),
         ((1400, 3, 1000), "ch", 1.0), ((2, 1024, 2047), "ch", 1.0)]


@pytest.mark.parametrize("shape,model,kappa", CASES, ids=["x".join(map(str, c[0])) for c in CASES])
def test_pair_sums_against_oracle(gpu, oracle, shape, model, kappa):
    from mmsp_gb300 import inputs

    x = inputs.noisy_composition(shape, 0.45 if model == "ch" else 0.0, 0.05, 60 + shape[0])
    p = dict(r=1.0, u=1.0) if model == "ch_poly" else {}
    d = gpu.make_desc(shape, 1, np.float64, model, kappa=kappa, mobility=1.1, dt=0.004, contract=True, **p)
    with gpu.Stepper(d) as s:
        s.upload(x)
        s.step(3)
        got = s.download()
    want = (oracle.ch_shipped(x, 3, 1.0, 1.0, kappa, 1.1, 0.004) if model == "ch_poly"
            else oracle.ch_baseline(x, 3, kappa, 1.1, 0.004))
    assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(want).max())
