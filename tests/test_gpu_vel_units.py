"""The in-place unit conversion of the velocities (BrightnessTemperature.c:158-217)
over the whole range of floats: each factor in FP64, rounded to float after each, in
numpy.  The library holds a factor in 48 bits, so a product may be rounded the other
way where it lies within 2^-48 of a tie: about 2^-24 of the cells per factor, below one
of these 6000 x 3.  At most two cells may differ, by an ulp, results below the normal
floats and products that overflow included."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trees,z", [(0, 7.3), (1, 9.0), (2, 14.7), (3, 6.2)])
def test_velocity_units(trees, z):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    D = 18
    p = dataclasses.replace(workload("full_256", D).params, flag_pecvel=1, trees_id=trees)
    rng = np.random.default_rng(trees)
    vel = np.zeros((D, D, D + 2), np.float32)
    vel[:, :, :D] = rng.choice([-1.0, 1.0], (D, D, D)) * 10.0 ** rng.uniform(-38.0, 38.5, (D, D, D))
    g = {"deltax": np.zeros((D, D, D + 2), np.float32), "xH": np.ones((D, D, D), np.float32),
         "TS_box": np.full((D, D, D), 20.0, np.float32), "vel": vel, "delta_T": np.zeros((D, D, D), np.float32)}
    g = {k: torch.from_numpy(a.copy()).cuda() for k, a in g.items()}
    ReionGridStep(p, [z + 1.0, z]).ComputeBrightnessTemperatureBox(1, g)
    got = g["vel"].cpu().numpy()[:, :, :D]
    zf = float(np.float32(z))
    with np.errstate(over="ignore", under="ignore"):
        want = vel[:, :, :D].astype(np.float64)
        if trees == 1:
            want = np.float32(np.sqrt(1.0 / (1.0 + zf)) * want / 1000.0)
        elif trees in (0, 2):
            want = np.float32((1.0 + zf) * want)
        want = np.float32(want.astype(np.float64) * (1000.0 * 100.0 / 3.086e24))
        want = np.float32(want.astype(np.float64) / (1.0 / (1.0 + zf)))
    assert np.isinf(want).any() == (trees in (0, 2)) and (np.abs(want) < 1e-38).any()
    assert (got != want).sum() <= 2
    assert np.isfinite(want[got != want]).all()
    step = np.spacing(np.abs(want[got != want])).astype(np.float64)
    assert (np.abs(got.astype(np.float64) - want)[got != want] <= step).all()
