"""The line-of-sight remap where neighbouring velocities differ by up to thousands
of cells, so that a cell's sub-cells land far apart and its halves cross thousands
of cell boundaries: against the fifty sub-cells in numpy FP64.

Tolerance 1e-6 of the box's largest |delta_T|.  H(z) and the displacement (a float
quotient) are formed here by the library's operations; positions agree to 2^-40
cells and FP64 rounding (1e-12 of 4096 cells), the shares and their sums to 1e-8 of
a source, and the result is a float (6e-8).  A count of sub-cells below a boundary
that is off by one would move up to 1e-2 / 50 of a source.
"""
import dataclasses

import numpy as np
import pytest

from test_gpu_pecvel import _remap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,cells", [(10, 4000.0), (34, 4000.0), (34, 300.0), (24, 3.0), (24, 0.9)])
def test_remap_of_far_subcells(D, cells):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("full_256", D)
    p = w.params
    z = np.float32(w.redshifts[1])
    opz = float(np.float32(1) + z)
    H = np.float32(3.2407789e-18 * p.hubble_h * np.sqrt(p.omega_m * opz ** 3 + p.omega_r * opz ** 4 + p.omega_lambda))
    inv_cell = float(D) / (p.box_size / p.hubble_h)
    rng = np.random.default_rng(D)
    shape = (D, D, 2 * (D // 2 + 1))
    vel, deltax = np.zeros(shape, np.float32), np.zeros(shape, np.float32)
    vel[:, :, :D] = rng.uniform(-cells, cells, (D, D, D)) / inv_cell * float(H) / (opz ** 2 * (1e5 / 3.086e24))
    deltax[:, :, :D] = rng.uniform(-0.5, 2.0, (D, D, D))
    xH = np.where(rng.random((D, D, D)) < 0.2, 0.0, rng.random((D, D, D))).astype(np.float32)
    TS = rng.uniform(5.0, 60.0, (D, D, D)).astype(np.float32)

    def run(mode):
        step = ReionGridStep(dataclasses.replace(p, flag_pecvel=mode), w.redshifts)
        g = {"deltax": deltax, "xH": xH, "TS_box": TS, "vel": vel.copy(), "delta_T": np.zeros((D, D, D), np.float32)}
        g = {k: torch.from_numpy(v).cuda() for k, v in g.items()}
        step.ComputeBrightnessTemperatureBox(1, g)
        return g["delta_T"].cpu().numpy(), g["vel"].cpu().numpy()[:, :, :D]

    dT2, _ = run(2)
    dT3, v = run(3)
    moved = (v / H).astype(np.float64) * inv_cell
    assert np.abs(moved).max() < 4096.0 and np.abs(moved).max() > 0.9 * cells
    want = _remap(dT2, xH, moved)
    assert np.abs(dT3 - want).max() <= 1e-6 * np.abs(want).max()
