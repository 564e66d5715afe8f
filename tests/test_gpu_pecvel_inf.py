"""Infinite and NaN velocities through the in-place unit conversion of the
peculiar-velocity modes (BrightnessTemperature.c:158-217): each factor is a positive
double, so an infinity stays one of the same sign and a NaN stays NaN.  Every other
velocity is what it is without them: it is converted by itself.

Snapshots: the factors' low parts take either sign and, at a redshift whose 1 + z is
a power of two, are 0."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trees,z", [(0, 7.0), (1, 7.0), (2, 9.3), (1, 11.1), (3, 6.2)])
def test_infinite_velocities_stay_infinite(trees, z):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    D = 24
    w = workload("full_256", D)
    p = dataclasses.replace(w.params, flag_pecvel=1, trees_id=trees)
    rng = np.random.default_rng(trees)
    vel = np.zeros((D, D, D + 2), np.float32)
    vel[:, :, :D] = rng.normal(0.0, 200.0, (D, D, D))
    special = vel.copy()
    special[1, 2, 3], special[4, 5, 6], special[7, 8, 9] = np.inf, -np.inf, np.nan
    out = []
    for v in (vel, special):
        g = {"deltax": np.zeros((D, D, D + 2), np.float32), "xH": np.ones((D, D, D), np.float32),
             "TS_box": np.full((D, D, D), 20.0, np.float32), "vel": v, "delta_T": np.zeros((D, D, D), np.float32)}
        g = {k: torch.from_numpy(a.copy()).cuda() for k, a in g.items()}
        ReionGridStep(p, [z + 1.0, z]).ComputeBrightnessTemperatureBox(1, g)
        out.append(g["vel"].cpu().numpy()[:, :, :D])
    plain, got = out
    assert got[1, 2, 3] == np.inf and got[4, 5, 6] == -np.inf and np.isnan(got[7, 8, 9])
    same = np.isfinite(special[:, :, :D])
    assert np.array_equal(got[same], plain[same])
