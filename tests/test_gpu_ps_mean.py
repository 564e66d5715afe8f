"""Compute_PS of a box whose mean delta_T is 0: the reference divides by the mean
(ComputePowerSpectrum.c:94-110), so that every bin of the power and of its error is
NaN, and the bins' mean |k| is what it is for any box.  A mean that is not 0, of
either sign and however small, gives finite powers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [16, 26])
def test_power_spectrum_of_a_zero_mean_box(D):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("plain_64", D)
    step = ReionGridStep(w.params, w.redshifts)
    ones = torch.ones((D, D, D), device="cuda")
    ones[::2] = 2.0
    k = step.Compute_PS(ones)[0]
    signs = torch.ones((D, D, D), device="cuda")
    signs[1::2] = -1.0  # the cells cancel exactly
    for box in (torch.zeros((D, D, D), device="cuda"), signs):
        k0, power, error = step.Compute_PS(box)
        assert np.array_equal(k0, k)
        assert np.isnan(power).all() and np.isnan(error).all()
    for mean in (1e-30, -1e-30, -3.0):
        box = signs * abs(mean) * 0.5 + mean
        k0, power, error = step.Compute_PS(box)
        assert np.array_equal(k0, k)
        assert np.isfinite(power).all() and np.isfinite(error).all()
